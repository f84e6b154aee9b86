"""The SBVR encoder on B200: dense fp16 tensor -> bit-planes + codebook (reference `_encode_to_sbvr`, sbvr/core.py:655-805).

The reference walks the groups of 256 values one by one in Python and, for each, materialises the squared differences
to every candidate coefficient line as tensors.  What it decides per group is kept here exactly:

  * after a warm-up of `cache_warmup_num` codebook lines, a group first looks for the best line already in the codebook
    and takes it if its MSE is below 0.99 x the mean MSE of the last `mse_window_size` accepted searches
    (sbvr/core.py:555-577);
  * otherwise (and while the codebook has room) it builds the group's own search space from the group's statistics
    (:400-483, :368-386), takes the best candidate, and if that beats the codebook's best, stores it as a new line
    (or reuses a line within 0.01 % of it) (:605-653).

How it is computed is different.  A step of the walk (`sbvr_encode_advance`) compares the line the last step added with
every undecided group, finds the first group whose best stored line is not good enough, and generates and evaluates that
group's own candidates in one kernel; what becomes of the winner is decided from it alone, on the device for many steps in a row
(`sbvr_encode_run`) and here for what that leaves over.  Nothing of size candidates x 256 x 2^S is ever stored, and every
group meets every line exactly once, so the result is that of the sequential walk.

The search space of a group is generated with the same tensor operations and the same fp16 roundings as the
reference's; `space_device` says where: "cpu" runs the tensor operations on the CPU and reproduces a reference run there
bit for bit; "cuda" is what the reference does when a GPU is present, with the roundings of the CUDA tensor operations
restated in the search kernel (groups it does not cover take the operations themselves).
"""
from __future__ import annotations

import ctypes
import itertools
import math
import sys
from dataclasses import dataclass, field
from typing import List, Optional, Tuple

import numpy as np
import torch

from . import _lib

GROUP = 256


@dataclass
class EncoderConfig:
    """The knobs of the reference's `_sbvr_enc_conf` (sbvr/core.py:19-37) that the data-difference error function uses."""
    num_sums: int = 4
    r_search_num: int = 64
    b_search_num: int = 40
    s_search_num: int = 40
    error_function: str = "data_diff_mse"
    mse_window_size: int = 20
    search_extend_ratio: float = 1.2
    cache_warmup_num: int = 10
    acceptable_mse: float = 10 ** -12
    extend_ratio: float = 1.2
    max_cache_lines: int = 2 ** 16
    batch_groups: int = 256            # accepted; the look-up covers all undecided groups at once
    space_device: str = "cuda"
    mse_history: List[float] = field(default_factory=list)

    @classmethod
    def from_dict(cls, d: Optional[dict]) -> "EncoderConfig":
        d = dict(d or {})
        known = {k: d[k] for k in list(d) if k in cls.__dataclass_fields__}
        conf = cls(**known)
        if conf.error_function != "data_diff_mse":
            raise ValueError("only the data_diff_mse error function is implemented (the reference's other one is unfinished)")
        if not 1 <= conf.num_sums <= 4:
            raise ValueError("the GPU encoder covers num_sums 1..4")
        return conf


def _bin_combs(S: int, device, dtype=torch.float16) -> torch.Tensor:
    """[2^S, S] rows of 0/1, first column = most significant selector bit (sbvr/core.py:345-351)."""
    return torch.tensor(list(itertools.product([0, 1], repeat=S)), dtype=dtype, device=device)


# ---------------------------------------------------------------------------------------------------------------
# the candidate lines of one group
# ---------------------------------------------------------------------------------------------------------------
def _ratio_bias_scale_lines(r_list, b_list, s_list, S: int) -> torch.Tensor:
    """Lines b + s * (1, r, r^2, ..) / span(r) for every (b, s, r), b outermost, r innermost
    (`_get_coeff_search_space_from_lists`, sbvr/core.py:388-398); span = max - min over the 2^S sums of the powers."""
    powers = r_list.unsqueeze(1) ** torch.arange(S, device=r_list.device).unsqueeze(0)         # [R, S]
    sums = powers @ _bin_combs(S, r_list.device, r_list.dtype).T                               # [R, 2^S]
    unit = powers / (sums.max(dim=1)[0] - sums.min(dim=1)[0]).unsqueeze(1)
    scaled = s_list.view(-1, 1, 1) * unit.unsqueeze(0)                                         # [Sn, R, S]
    return (b_list.view(-1, 1, 1, 1) + scaled.unsqueeze(0)).view(-1, S)


def _grid_intervals(conf: EncoderConfig, S: int, extended: bool) -> int:
    budget = conf.r_search_num * conf.b_search_num * conf.s_search_num * 1.4
    if extended:
        budget *= conf.search_extend_ratio ** 3
    return int(budget ** (1 / S))


def _grid_lines(data: torch.Tensor, conf: EncoderConfig, S: int, extended: bool) -> torch.Tensor:
    """A plain grid over the data range, one axis per coefficient (`_get_additional_search_space`, sbvr/core.py:368-386)."""
    per_dim = _grid_intervals(conf, S, extended)
    lo, hi = torch.min(data), torch.max(data)
    edges = torch.linspace(lo, hi, S + 1, device=data.device, dtype=data.dtype)
    axes = []
    for i in range(S):
        slack = abs(edges[i]) * 0.8
        axes.append(torch.linspace(edges[i] - slack, edges[i + 1] + slack, per_dim + 1, device=data.device,
                                   dtype=data.dtype))
    return torch.cartesian_prod(*axes).view(-1, S)


def _ratio_list(conf: EncoderConfig, extended: bool, device, dtype=torch.float16) -> torch.Tensor:
    """The ratios of neighbouring coefficients: below one, then above (sbvr/core.py:404-430)."""
    r_lo = (math.pi / 6, 0.94)
    r_hi = (1.06, math.pi * 2 / 3)
    r_lo_step = (r_lo[1] - r_lo[0]) / (conf.r_search_num / 2)
    r_hi_step = (r_hi[1] - r_hi[0]) / (conf.r_search_num / 2)
    if extended:
        r_lo_step /= conf.extend_ratio
        r_hi_step /= conf.extend_ratio
    kw = dict(device=device, dtype=dtype)
    return torch.cat((-torch.arange(r_lo[0] + r_lo_step, r_lo[1] + r_lo_step, r_lo_step, **kw),
                      -torch.arange(r_hi[0] + r_hi_step, r_hi[1] + r_hi_step, r_hi_step, **kw)))


def _bias_list(conf: EncoderConfig, b_hi, extended: bool, device, dtype=torch.float16) -> torch.Tensor:
    b_lo = -b_hi
    b_step = (b_hi - b_lo) / conf.b_search_num
    if extended:
        b_step /= conf.extend_ratio
    kw = dict(device=device, dtype=dtype)
    return torch.arange(b_lo, b_hi, b_step, **kw) if b_step != 0 else torch.tensor([b_lo], **kw)


def group_search_space(data: torch.Tensor, conf: EncoderConfig, extended: bool) -> torch.Tensor:
    """Candidate lines [n, S] (fp16, each sorted by magnitude) for one group of values `data` (fp16, on the device the
    space is to be generated on): `_get_coeff_search_space`, sbvr/core.py:400-483.  Every quantity has the type it has
    there (fp16 tensors for the data statistics, an fp32 tensor for the 95 % quantile, Python floats for the ratio
    ranges), because the fp16 roundings decide the candidates."""
    S = conf.num_sums
    d_max, d_avg, d_min = torch.max(data), torch.mean(data), torch.min(data)
    d_95 = torch.quantile(data.to(torch.float), 0.95)

    b_hi = abs(d_avg) * 2.0 / S
    if b_hi < 0.3:
        b_hi = 0.3
    s_hi = (d_max - d_min) * 1.1
    s_lo = 2 * d_95
    s_step = (s_hi - s_lo) / conf.s_search_num
    if extended:
        s_step /= conf.extend_ratio

    kw = dict(device=data.device, dtype=data.dtype)
    r_list = _ratio_list(conf, extended, data.device, data.dtype)
    s_list = torch.arange(s_lo + s_step, s_hi + s_step, s_step, **kw) if s_step != 0 else torch.tensor([s_lo], **kw)
    b_list = _bias_list(conf, b_hi, extended, data.device, data.dtype)

    space = _ratio_bias_scale_lines(r_list, b_list, s_list, S)
    if S <= 6:
        space = torch.cat((space, _grid_lines(data, conf, S, extended)), dim=0)
    order = torch.sort(space.abs(), dim=1)[1]
    return torch.gather(space, dim=1, index=order).contiguous()


# ---------------------------------------------------------------------------------------------------------------
# device helpers (thin wrappers of the C ABI)
# ---------------------------------------------------------------------------------------------------------------
def _mse(data: torch.Tensor, lines: torch.Tensor, S: int) -> torch.Tensor:
    """fp32 [groups, L]: MSE of every group of `data` [groups, 256] against every line of `lines` [L, S]."""
    groups, L = data.shape[0], lines.shape[0]
    out = torch.empty((groups, L), dtype=torch.float32, device=data.device)
    st = torch.cuda.current_stream(data.device).cuda_stream
    for g0 in range(0, groups, 32768):                      # grid.y limit
        g1 = min(groups, g0 + 32768)
        _lib.check(_lib.lib.sbvr_encode_mse_f16(data[g0:g1].data_ptr(), g1 - g0, lines.data_ptr(), L, S,
                                                out[g0:g1].data_ptr(), st), "sbvr_encode_mse_f16")
    return out


def _select(data: torch.Tensor, lines: torch.Tensor, which: torch.Tensor, S: int, sel_out: torch.Tensor) -> None:
    """sel_out[b] (uint8 [groups, 256]) = nearest-sum selectors of group b for line which[b] of `lines`."""
    st = torch.cuda.current_stream(data.device).cuda_stream
    _lib.check(_lib.lib.sbvr_encode_select_f16(data.data_ptr(), data.shape[0], lines.data_ptr(), which.data_ptr(), S,
                                               sel_out.data_ptr(), st), "sbvr_encode_select_f16")


def pack_selectors(sel: torch.Tensor, S: int) -> torch.Tensor:
    """Selectors uint8 [N, Kp] (device) -> bvr uint32 [Kp/32, N, S]."""
    N, Kp = sel.shape
    bvr = torch.empty((Kp // 32, N, S), dtype=torch.int32, device=sel.device)
    st = torch.cuda.current_stream(sel.device).cuda_stream
    _lib.check(_lib.lib.sbvr_encode_pack(sel.data_ptr(), N, Kp, S, bvr.data_ptr(), st), "sbvr_encode_pack")
    return bvr.view(torch.uint32)


# ---------------------------------------------------------------------------------------------------------------
# the walk over the groups
# ---------------------------------------------------------------------------------------------------------------
def _compensated_sum(values) -> float:
    """A sum of floats with Neumaier's compensation (Z. angew. Math. Mech. 54, 1974): what the walk kernel forms, and `sum` from Python
    3.12 on."""
    total = lost = 0.0
    for x in values:
        t = total + x
        lost += (total - t) + x if abs(total) >= abs(x) else (x - t) + total
        total = t
    return total + lost if lost and math.isfinite(lost) else total


_sum = sum if sys.version_info >= (3, 12) else _compensated_sum


class _Codebook:
    """The growing coefficient cache and the running statistics that steer the search (the mutable part of the
    reference's `_sbvr_enc_conf`: coeff_cache, num_coeff_cache_lines, mse_history, cache_hits, group_idx).  The lines are
    kept on the device and mirrored here, so that a step needs no copy back."""

    def __init__(self, conf: EncoderConfig, device):
        self.conf = conf
        self.lines = torch.zeros((conf.max_cache_lines, conf.num_sums), dtype=torch.float16, device=device)
        self.host = np.zeros((256, conf.num_sums), dtype=np.float16)
        self.n = 0
        self.history: List[float] = list(conf.mse_history)
        self._cutoff: Optional[float] = None

    def accept(self, mse: float) -> None:
        self.history.append(mse)
        self._cutoff = None

    def cutoff(self) -> float:
        """0.99 x the mean MSE of the most recent accepted searches, not below `acceptable_mse` (sbvr/core.py:563-568)."""
        if self._cutoff is None:
            window = self.history[-min(len(self.history), self.conf.mse_window_size):]
            self._cutoff = max((_sum(window) / len(window)) * 0.99, self.conf.acceptable_mse)
        return self._cutoff

    def find_or_add(self, line: np.ndarray) -> Tuple[int, bool]:
        """Index of a stored line within 0.01 % (summed magnitude, fp16 arithmetic) of `line`, else the index it is
        appended at (sbvr/core.py:634-646).  Returns (index, appended); the caller stores an appended line on the device."""
        if self.n:
            def mag(v):                            # |v| summed over the last dimension, fp32 sum rounded to fp16
                return np.abs(v).astype(np.float32).sum(-1).astype(np.float16)
            near = (mag(line).astype(np.float32) * np.float32(0.0001)).astype(np.float16)
            stored = self.host[:self.n]
            # fp32 first: the fp16 arithmetic of numpy is slow, and almost no line is anywhere near
            rough = np.abs(stored.astype(np.float32) - line.astype(np.float32)).sum(-1) <= 2 * float(near) + 1e-4
            for i in np.nonzero(rough)[0]:
                if mag(stored[i] - line) < near:
                    return int(i), False
        if self.n >= len(self.lines):              # (a warm-up longer than the codebook)
            raise IndexError(f"the codebook has {len(self.lines)} lines")
        self.mirror(line)
        return self.n - 1, True

    def mirror(self, line: np.ndarray) -> None:
        if self.n == len(self.host):
            self.host = np.concatenate((self.host, np.zeros_like(self.host)))
        self.host[self.n] = line
        self.n += 1


def _full_search(group: torch.Tensor, conf: EncoderConfig, extended: bool) -> Tuple[float, np.ndarray]:
    """Best candidate of the group's own search space by tensor operations: (mse, line)."""
    src = group if conf.space_device == "cuda" else group.to(conf.space_device)
    space = group_search_space(src, conf, extended).to(group.device)
    mse = _mse(group.view(1, GROUP), space, conf.num_sums)[0]
    at = torch.argmin(mse)                                   # the first of equal minima, like the reference's argmin
    return float(mse[at]), space[at].cpu().numpy()


class _SearchTables:
    """What the candidates of all groups have in common, plain and extended: the power lines over the span of their sums and
    the biases, made by the tensor operations of `group_search_space` (fp16 on the device), and the grid's intervals."""

    def __init__(self, conf: EncoderConfig, device):
        S = conf.num_sums
        self.unit, self.bias, self.per_dim = [], [], []
        for extended in (False, True):
            r_list, b_list = _ratio_list(conf, extended, device), _bias_list(conf, 0.3, extended, device)
            powers = r_list.unsqueeze(1) ** torch.arange(S, device=device).unsqueeze(0)
            sums = powers @ _bin_combs(S, device, torch.float16).T
            self.unit.append((powers / (sums.max(dim=1)[0] - sums.min(dim=1)[0]).unsqueeze(1)).contiguous())
            self.bias.append(b_list)
            self.per_dim.append(_grid_intervals(conf, S, extended))
        # what the kernel's candidate numbers (31 bits) and fp16 grid positions can count; the limits of sbvr_encode_advance
        self.covered = conf.s_search_num >= 1 and conf.extend_ratio > 0 and all(
            len(u) >= 1 and len(b) >= 1 and 1 <= d <= 2000 and len(u) * len(b) * 1024 + (d + 1) ** S < 2.0e9
            for u, b, d in zip(self.unit, self.bias, self.per_dim))


class _ManySteps:
    """`sbvr_encode_run`: steps of the walk on the device until the host has to look at a group."""
    LIMIT, WINDOW = 1024, 64

    def __init__(self, conf: EncoderConfig, device):
        self.conf = conf
        self.ctl = torch.empty(8, dtype=torch.int64, device=device)
        size = ctypes.sizeof(_lib.EncodeRecord)
        self.pinned = torch.empty(32 + self.LIMIT * size, dtype=torch.uint8, pin_memory=True)
        at = self.pinned.data_ptr()
        self.outcome = (ctypes.c_int * 6).from_address(at)
        self.records = np.frombuffer((ctypes.c_ubyte * (self.LIMIT * size)).from_address(at + 32), dtype=np.dtype(
            {"names": ["group", "at", "mse", "line"], "formats": [np.int32, np.int32, np.float32, (np.uint16, 4)], "offsets": [0, 4, 8, 12],
             "itemsize": size}))
        self.args = _lib.EncodeRun(ctl=self.ctl.data_ptr(), records=at + 32, outcome=at, capacity=conf.max_cache_lines,
                                   warmup=conf.cache_warmup_num, window=conf.mse_window_size, limit=self.LIMIT,
                                   acceptable=conf.acceptable_mse)

    def run(self, walk, book: "_Codebook", stream: int, own_groups: list, own_lines: list, own_index: list) -> Tuple[int, int]:
        """Walks on from `walk.from_`; returns the first group that is not decided, and why it stopped."""
        a, S = self.args, self.conf.num_sums
        tail = book.history[-self.conf.mse_window_size:]
        a.n, a.hist_n = book.n, len(tail)
        a.hist[:len(tail)] = tail
        _lib.check(_lib.lib.sbvr_encode_run(ctypes.byref(walk), ctypes.byref(a), stream), "sbvr_encode_run")
        why, gi, n, walk.line0, walk.misses, accepted = self.outcome
        rec = self.records[:accepted].copy()
        lines = rec["line"][:, :S].copy().view(np.float16)
        own_groups += rec["group"].tolist()
        own_lines += list(lines)
        own_index += rec["at"].tolist()
        for at, line in zip(rec["at"].tolist(), lines):
            if at == book.n:
                book.mirror(line)
        assert book.n == n
        for mse in rec["mse"].tolist():
            book.accept(mse)
        return walk.groups if why == _lib.ENCODE_DONE else gi, why


def _sorted_line(bits, S: int, device) -> np.ndarray:
    """A candidate's coefficients in ascending magnitude; equal magnitudes in the order the device's sort leaves them in."""
    line = np.array(bits[:S], dtype=np.uint16).view(np.float16)
    mag = np.abs(line)
    if len(set(mag.tolist())) == S:
        return line[np.argsort(mag)]
    t = torch.from_numpy(line).to(device).view(1, S)
    return torch.gather(t, 1, torch.sort(t.abs(), dim=1)[1])[0].cpu().numpy()


@torch.inference_mode()
def encode(data: torch.Tensor, conf: EncoderConfig, device: Optional[torch.device] = None, progress=None):
    """Dense tensor [..., K] -> (bvr uint32 [Kp/32, N, S], coeff_idx uint8|uint16 [Kp/256, N], coeff_cache fp16 [C, S],
    stats) in the reference's GPU layout, N = product of the leading dimensions, Kp = K rounded up to 256 (zero padded,
    sbvr/core.py:667-676)."""
    dev = torch.device(device) if device is not None else torch.device("cuda")
    if dev.type != "cuda":
        raise RuntimeError("the encoder runs on a CUDA device (there is no CPU implementation)")
    S = conf.num_sums
    K = int(data.shape[-1])
    Kp = (K + GROUP - 1) // GROUP * GROUP
    flat = data.reshape(-1, K).to(dev).to(torch.float16)
    N = flat.shape[0]
    if Kp != K:
        flat = torch.nn.functional.pad(flat, (0, Kp - K))
    flat = flat.contiguous()
    if flat.data_ptr() % 16:
        flat = flat.clone()
    groups = flat.view(-1, GROUP)                            # group i = (row i // (Kp/256), block i % (Kp/256))
    NG = groups.shape[0]
    with torch.cuda.device(dev):
        st = torch.cuda.current_stream().cuda_stream
        book = _Codebook(conf, dev)
        best_mse = torch.full((NG,), float("inf"), dtype=torch.float32, device=dev)
        line_of = torch.zeros(NG, dtype=torch.int32, device=dev)            # of undecided groups: the best stored line so far
        scratch = torch.empty(2, dtype=torch.int64, device=dev)
        pinned = torch.empty(ctypes.sizeof(_lib.EncodeResult), dtype=torch.uint8, pin_memory=True)
        res = _lib.EncodeResult.from_address(pinned.data_ptr())
        walk = _lib.EncodeWalk(data=groups.data_ptr(), lines=book.lines.data_ptr(), best_mse=best_mse.data_ptr(),
                               best_at=line_of.data_ptr(), scratch=scratch.data_ptr(), result=pinned.data_ptr(), S=S, groups=NG,
                               s_search_num=conf.s_search_num, extend_ratio=conf.extend_ratio, append_at=-1)
        # one coefficient has a grid axis of 10^5 points, beyond what fp16 steps can count: tensor operations
        tables = _SearchTables(conf, dev) if conf.space_device == "cuda" and S > 1 else None
        kernel_search = tables is not None and tables.covered
        if kernel_search:
            group_stats = torch.empty((NG, 4), dtype=torch.float32, device=dev)
            _lib.check(_lib.lib.sbvr_encode_stats_f16(groups.data_ptr(), NG, group_stats.data_ptr(), st), "sbvr_encode_stats_f16")
            walk.stats = group_stats.data_ptr()
            for e in (0, 1):
                walk.unit[e], walk.bias[e] = tables.unit[e].data_ptr(), tables.bias[e].data_ptr()
                walk.R[e], walk.B[e] = tables.unit[e].shape[0], tables.bias[e].shape[0]
                walk.per_dim[e] = tables.per_dim[e]
        advance, walk_ref = _lib.lib.sbvr_encode_advance, ctypes.byref(walk)
        # many steps per launch, unless the caller wants to hear of each; one step at a time for what that leaves to the host
        many = _ManySteps(conf, dev) if kernel_search and progress is None and 1 <= conf.mse_window_size <= _ManySteps.WINDOW else None
        own_groups, own_lines, own_index = [], [], []      # groups that keep their own candidate, it, the line it is filed under
        gi = 0
        hits = None
        host_search = False                                # the last step's group was left to the tensor operations; the next one may be too
        while gi < NG:
            if many is not None and not host_search and (book.n < conf.max_cache_lines or book.n < conf.cache_warmup_num):
                if walk.append_at >= 0:
                    book.lines[walk.append_at] = torch.from_numpy(book.host[walk.append_at]).to(dev)
                    walk.append_at = -1
                walk.from_, walk.search = gi, 1
                gi, why = many.run(walk, book, st, own_groups, own_lines, own_index)
                if why == _lib.ENCODE_TIMEOUT:             # its blocks cannot all run at the moment: single steps to the end
                    many = None
                if gi >= NG:
                    hits = NG - walk.misses
                    break
            warm = book.n < conf.cache_warmup_num          # every group searches its own space
            full = book.n >= conf.max_cache_lines          # the best stored line has to do
            walk.from_, walk.line1, walk.warm = gi, book.n, int(warm)
            full = full and not warm
            walk.search = int(kernel_search and not full)
            walk.cutoff = 0.0 if warm else float("inf") if full else book.cutoff()
            _lib.check(advance(walk_ref, st), "sbvr_encode_advance")
            walk.append_at = -1
            if not warm:
                walk.line0 = walk.line1
            g = res.group
            host_search = res.status == 2
            if full:
                hits = gi - walk.misses + int((best_mse[gi:].double() < book.cutoff()).sum())
                break
            if g >= NG:
                hits = NG - walk.misses
                break
            if res.status == 2:
                new_mse, line = _full_search(groups[g], conf, warm or (g - walk.misses) / (g + 1) > 0.6)
                better = new_mse < res.cached_mse
            elif res.status == 1:
                new_mse, line, better = res.mse, _sorted_line(res.line, S, dev), True
            else:
                better = False                             # the codebook already has something at least as good
            walk.misses += 1
            if better:
                at, appended = book.find_or_add(line)
                if appended:
                    walk.append_at = at
                    walk.append[:S] = line.view(np.uint16).tolist()
                own_groups.append(g)                       # selectors of the candidate itself, also when an old line is reused
                own_lines.append(line)
                own_index.append(at)
                book.accept(new_mse)
            gi = g + 1
            if progress:
                progress(gi, NG)
        if progress and gi < NG:
            progress(NG, NG)
        if walk.append_at >= 0:
            book.lines[walk.append_at] = torch.from_numpy(book.host[walk.append_at]).to(dev)

        C = book.n
        cache = book.lines[:C].contiguous()
        sel = torch.empty((NG, GROUP), dtype=torch.uint8, device=dev)
        if own_groups:
            rows = torch.tensor(own_groups, dtype=torch.long, device=dev)
            line_of[rows] = torch.tensor(own_index, dtype=torch.int32, device=dev)
        _select(groups, book.lines, line_of, S, sel)
        if own_groups:
            tmp = torch.empty((len(own_groups), GROUP), dtype=torch.uint8, device=dev)
            _select(groups[rows], torch.from_numpy(np.stack(own_lines)).to(dev), torch.arange(len(own_groups), dtype=torch.int32, device=dev),
                    S, tmp)
            sel[rows] = tmp
        idx = line_of.view(N, Kp // GROUP).T.contiguous()
        idx = idx.to(torch.uint8) if C <= 256 else idx.to(torch.int16).view(torch.uint16)   # C <= 65536: the bits fit
        bvr = pack_selectors(sel.view(N, Kp), S)
        torch.cuda.synchronize(dev)
    stats = {"groups": NG, "cache_lines": C, "cache_hits": NG - walk.misses if hits is None else hits, "searches": len(book.history) - len(conf.mse_history)}
    return bvr, idx, cache, stats
