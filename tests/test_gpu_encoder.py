"""The GPU encoder (`sbvr.sbvr(data, encoder_config)`, sbvr/encoder.py + csrc/encode.cu) against the reference encoder's
golden output and against the CPU restatement of its error function (oracle/encoder_ref.py)."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import encoder_ref as E
from oracle import sbvr_oracle as O

pytestmark = pytest.mark.gpu


def _u16(t):
    return t.cpu().view(torch.int16).numpy().view(np.uint16) if t.dtype == torch.uint16 else t.cpu().numpy()


@pytest.mark.parametrize("S", [1, 2, 3, 4])
def test_error_function_and_selectors_match_the_restatement(S):
    """`sbvr_encode_mse_f16` / `sbvr_encode_select_f16` on seeded groups and lines: the fp16 steps are the reference's, so
    the selectors are identical and the MSEs differ only by the order of the fp32 sum over the 256 values."""
    from sbvr import encoder
    g = torch.Generator().manual_seed(S)
    data = (torch.randn((5, 256), generator=g) * 0.02).half()
    lines = (torch.randn((777, S), generator=g) * 0.02).half()
    ref = E.mse_table(data, lines)
    got = encoder._mse(data.cuda(), lines.cuda(), S).cpu().numpy()
    assert got.shape == ref.shape
    assert np.abs(got - ref).max() <= 2e-6 * ref.max()
    which = torch.tensor([0, 5, 776, 13, 400], dtype=torch.int32)
    sel = torch.empty((5, 256), dtype=torch.uint8, device="cuda")
    encoder._select(data.cuda(), lines.cuda(), which.cuda(), S, sel)
    for b in range(5):
        assert np.array_equal(sel[b].cpu().numpy(), E.selectors(data[b], lines[int(which[b])]))


@pytest.mark.parametrize("S", [2, 3, 4])
def test_pack_selectors_is_the_reference_layout(S):
    from sbvr import encoder
    rng = np.random.default_rng(S)
    sel = rng.integers(0, 2 ** S, size=(7, 512), dtype=np.uint8)
    bvr = encoder.pack_selectors(torch.from_numpy(sel).cuda(), S)
    assert np.array_equal(bvr.cpu().view(torch.int32).numpy().view(np.uint32), O.pack_bvr(sel.astype(np.int64), S))


@pytest.mark.parametrize("name", ["enc_s2", "enc_s3", "enc_s4", "enc_s4_pad"])
def test_encoder_reproduces_the_reference_encoder(golden, name):
    """Same input as the golden case, search spaces generated on the CPU like the reference run that made it: the
    codebook, the indices and the bit-planes are the reference's, bit for bit; and `decode()` gives its decoded weight."""
    import sbvr
    c = golden[name]
    S = int(c["S"])
    W = torch.from_numpy(c["W"])
    w = sbvr.sbvr(W, encoder_config={"num_sums": S, "space_device": "cpu"}, verbose_level=0)
    assert np.array_equal(_u16(w.coeff_cache).view(np.uint16), c["coeff_cache"].view(np.uint16))
    assert np.array_equal(_u16(w.coeff_idx), c["coeff_idx"])
    assert np.array_equal(w.bvr.cpu().view(torch.int32).numpy().view(np.uint32), c["bvr"])
    assert np.array_equal(w.decode().cpu().numpy().view(np.uint16), c["decoded"].view(np.uint16))


def _mse_of(w, W):
    return float(((w.decode().float().cpu() - W.float()) ** 2).mean())


@pytest.mark.parametrize("name", ["enc_s2", "enc_s4", "enc_s4_pad"])
def test_encoder_with_gpu_generated_search_space_is_as_good(golden, name):
    """Search spaces generated on the GPU (the default; what the reference does when it has a GPU): candidates may differ
    from a CPU run in the last fp16 bit, the quality must not."""
    import sbvr
    c = golden[name]
    W = torch.from_numpy(c["W"])
    w = sbvr.sbvr(W, encoder_config={"num_sums": int(c["S"])}, verbose_level=0)
    ref_mse = float(((torch.from_numpy(c["decoded"]).float() - W.float()) ** 2).mean())
    assert _mse_of(w, W) <= 1.02 * ref_mse
    assert tuple(w.decode().shape) == tuple(W.shape)


def _walk(W, conf):
    """The walk one group at a time by the tensor operations (sbvr/core.py:555-653): every stored line against the group, then the
    group's own search space.  Returns what `encoder.encode` returns, without the statistics."""
    from sbvr import encoder
    S = conf.num_sums
    data = W.cuda()
    N, K = data.shape
    Kp = -(-K // 256) * 256
    groups = torch.nn.functional.pad(data, (0, Kp - K)).contiguous().view(-1, 256)
    lines, history, hits, line_of, sel = [], list(conf.mse_history), 0, [], []
    for g in range(len(groups)):
        group = groups[g:g + 1]
        warm = len(lines) < conf.cache_warmup_num
        cached, at = float("inf"), 0
        own = None
        if not warm:
            mse = encoder._mse(group, torch.stack(lines), S)[0]
            at = int(torch.argmin(mse))
            cached = float(mse[at])
            window = history[-min(len(history), conf.mse_window_size):]
            if cached < max(sum(window) / len(window) * 0.99, conf.acceptable_mse):
                hits += 1
                own = False
            elif len(lines) >= conf.max_cache_lines:
                own = False
        if own is None:
            space = encoder.group_search_space(group[0], conf, warm or hits / (g + 1) > 0.6)
            mse = encoder._mse(group, space, S)[0]
            best = int(torch.argmin(mse))
            own = not float(mse[best]) >= cached
            if own:
                line = space[best]
                history.append(float(mse[best]))
                near = [i for i, l in enumerate(lines) if bool((l - line).abs().sum(-1) < line.abs().sum(-1) * 0.0001)]
                at = near[0] if near else len(lines)
                if not near:
                    lines.append(line.clone())
        line_of.append(at)
        out = torch.empty((1, 256), dtype=torch.uint8, device="cuda")
        encoder._select(group.contiguous(), (line if own else lines[at]).view(1, S).contiguous(), torch.zeros(1, dtype=torch.int32, device="cuda"), S, out)
        sel.append(out)
    idx = torch.tensor(line_of).view(N, Kp // 256).T.contiguous()
    return encoder.pack_selectors(torch.cat(sel).view(N, Kp), S), idx, torch.stack(lines)


@pytest.mark.parametrize("kind", ["spread", "full_codebook", "wide_search"])
@pytest.mark.parametrize("S", [2, 3, 4])
def test_the_walk_equals_one_group_at_a_time(S, kind):
    """The device walk (best stored lines kept per group, search kernel, appended and reused lines, the cutoff, the extended switch)
    against the walk by tensor operations, bit for bit; with a codebook that fills up, and search settings that the search
    kernel does not cover."""
    from sbvr import encoder
    g = torch.Generator().manual_seed(S)
    W = (torch.randn((24, 500), generator=g) * 0.02).half()
    W[:, :256] *= torch.linspace(0.5, 3.0, 24).view(-1, 1).half()         # spread the statistics: more misses
    W[20] = W[3]                                                            # groups that come again
    settings = {"num_sums": S}
    if kind == "full_codebook":
        settings["max_cache_lines"] = 12
    if kind == "wide_search":
        if S != 2:
            pytest.skip("more than 2000 grid intervals per axis need two planes")
        settings.update(r_search_num=130, b_search_num=130, s_search_num=130)
        W = W[:4]
    conf = encoder.EncoderConfig(**settings)
    calls = []
    bvr, idx, cache, stats = encoder.encode(W, conf, progress=lambda done, of: calls.append((done, of)))
    ref_bvr, ref_idx, ref_cache = _walk(W, conf)
    assert torch.equal(cache.view(torch.int16), ref_cache.view(torch.int16))
    assert torch.equal(idx.cpu().to(torch.int64), ref_idx)
    assert torch.equal(bvr.view(torch.int32), ref_bvr.view(torch.int32))
    assert stats["cache_lines"] == len(ref_cache) and calls[-1] == (stats["groups"], stats["groups"])
    assert kind == "wide_search" or stats["cache_hits"] > 0


def test_batched_lookup_equals_the_sequential_walk():
    """`batch_groups` is accepted and changes nothing (the walk itself is compared above); trans=True encodes the transpose."""
    import sbvr
    g = torch.Generator().manual_seed(3)
    W = (torch.randn((48, 512), generator=g) * 0.02).half()
    W[:, :256] *= torch.linspace(0.5, 3.0, 48).view(-1, 1).half()         # spread the statistics: more misses
    a = sbvr.sbvr(W, encoder_config={"num_sums": 3, "batch_groups": 1}, verbose_level=0)
    b = sbvr.sbvr(W, encoder_config={"num_sums": 3, "batch_groups": 37}, verbose_level=0)
    assert torch.equal(a.coeff_cache, b.coeff_cache)
    assert torch.equal(a.coeff_idx.view(torch.uint8), b.coeff_idx.view(torch.uint8))
    assert torch.equal(a.bvr.view(torch.int32), b.bvr.view(torch.int32))
    assert a.encoder_stats == b.encoder_stats and a.encoder_stats["cache_hits"] > 0
    t = sbvr.sbvr(W[:, :256].contiguous(), encoder_config={"num_sums": 2}, verbose_level=0, trans=True)
    assert tuple(t.bvr.shape) == (8, 256, 2)                               # W^T is [256, 48], padded to 256 along the bits
    assert tuple(t.decode().shape) == (256, 48)


def test_encode_then_linear_end_to_end():
    """A really encoded weight (not synthetic planes) through the decode GEMV and the batched GEMM: the product with the
    packed weight equals x @ decode().T within the fp16 tolerance, and stays close to the product with the dense weight."""
    import sbvr
    g = torch.Generator().manual_seed(42)
    W = (torch.randn((1024, 4096), generator=g) * 0.02).half().cuda()
    w = sbvr.sbvr(W, encoder_config={"num_sums": 4}, verbose_level=0)
    Wd = w.decode()
    assert float(((Wd.float() - W.float()) ** 2).mean() / (W.float() ** 2).mean()) < 0.02
    for M in (1, 16):
        x = torch.randn((M, 4096), generator=g).half().cuda()
        y = sbvr.linear(x, w).double()
        ref = x.double() @ Wd.double().T
        assert float((y - ref).abs().max() / ref.abs().max()) <= 1e-2
        dense = x.double() @ W.double().T
        assert float((y - dense).abs().max() / dense.abs().max()) < 0.2


@pytest.mark.parametrize("S", [2, 3, 4])
@pytest.mark.parametrize("settings", [{}, {"cache_warmup_num": 1}, {"cache_warmup_num": 40, "mse_window_size": 64}, {"mse_window_size": 1},
                                      {"max_cache_lines": 23}, {"acceptable_mse": 1e-4}, {"mse_history": [1e-7, 3e-6], "cache_warmup_num": 0},
                                      {"mse_window_size": 65}])
def test_many_steps_in_one_launch_equal_one_at_a_time(monkeypatch, S, settings):
    """With a progress callback the walk takes one step per launch and decides on the host; without, on the device: codebook, indices,
    bit-planes and counts are the same.  Among the groups: repeated ones (a winner that is stored already), zeros, a large mean
    and too few distinct values (left to the host); a launch takes seven misses, and once as many as it does."""
    from sbvr import encoder
    g = torch.Generator(device="cuda").manual_seed(S)
    rows = 300 if S == 4 and settings == {"mse_window_size": 1} else 24
    W = torch.randn((rows, 1024), device="cuda", generator=g) * 0.02 * torch.exp(0.4 * torch.randn((rows, 1), device="cuda", generator=g))
    W[5] = W[2]
    W[7] = 0
    W[9] += 0.5
    W[11] = torch.sign(W[11]) * 0.01
    W[13, :256] = W[13, 0]
    one = encoder.encode(W.half(), encoder.EncoderConfig(num_sums=S, **settings), progress=lambda done, of: None)
    for limit in (None, 7):
        why = _watch_runs(monkeypatch, limit)
        many = encoder.encode(W.half(), encoder.EncoderConfig(num_sums=S, **settings))
        assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(one[:3], many[:3]))
        assert one[3] == many[3]
        assert bool(why) == (settings != {"mse_window_size": 65})          # (more errors to look back on than the kernel keeps)


@pytest.mark.parametrize("S", [2, 4])
@pytest.mark.parametrize("settings,mean,reasons", [({"cache_warmup_num": 40}, 0.0, ["LIMIT", "DONE"]), ({"cache_warmup_num": 40}, 0.5, ["LIMIT", "CALLER"]),
                                                   ({"cache_warmup_num": 10, "max_cache_lines": 10}, 0.0, ["LIMIT", "FULL"])])
def test_launches_end_for_every_reason(monkeypatch, S, settings, mean, reasons):
    """A launch of seven steps at most ends because it has taken them, at a group of a large mean, when the codebook is full or at the
    end, and the walk goes on from there as in single steps."""
    from sbvr import _lib, encoder
    g = torch.Generator(device="cuda").manual_seed(S)
    W = torch.randn((24, 1024), device="cuda", generator=g) * 0.02 * torch.exp(0.4 * torch.randn((24, 1), device="cuda", generator=g))
    W[5] += mean
    conf = encoder.EncoderConfig(num_sums=S, **settings)
    one = encoder.encode(W.half(), conf, progress=lambda done, of: None)
    why = _watch_runs(monkeypatch, limit=7)
    many = encoder.encode(W.half(), conf)
    assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(one[:3], many[:3])) and one[3] == many[3]
    assert {getattr(_lib, "ENCODE_" + r) for r in reasons} <= set(why), why


@pytest.mark.parametrize("S", [2, 4])
@pytest.mark.parametrize("settings", [{}, {"cache_warmup_num": 40}])
def test_blocks_that_do_not_meet_leave_the_walk_to_single_steps(monkeypatch, S, settings):
    """A launch of many steps whose blocks could not all run reports so, with the walk as it stands; the rest is walked step by step."""
    from sbvr import _lib, encoder
    g = torch.Generator(device="cuda").manual_seed(S)
    W = (torch.randn((24, 1024), device="cuda", generator=g) * 0.02 * torch.exp(0.4 * torch.randn((24, 1), device="cuda", generator=g))).half()
    conf = encoder.EncoderConfig(num_sums=S, **settings)
    one = encoder.encode(W, conf, progress=lambda done, of: None)
    why = _watch_runs(monkeypatch, limit=5, outcome=_lib.ENCODE_TIMEOUT)
    many = encoder.encode(W, conf)
    assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(one[:3], many[:3])) and one[3] == many[3]
    assert why == [_lib.ENCODE_TIMEOUT]


def _watch_runs(monkeypatch, limit=None, outcome=None):
    """Counts why the launches of many steps end; `limit`: steps of one launch; `outcome`: what each is made to report."""
    from sbvr import _lib, encoder
    why, real = [], _lib.lib.sbvr_encode_run
    if limit:
        monkeypatch.setattr(encoder._ManySteps, "LIMIT", limit)

    def run(walk, args, stream):
        rc = real(walk, args, stream)
        out = ctypes.cast(args._obj.outcome, ctypes.POINTER(ctypes.c_int))
        if outcome:
            out[0] = outcome
        why.append(out[0])
        return rc
    monkeypatch.setattr(_lib.lib, "sbvr_encode_run", run)
    return why


@pytest.mark.parametrize("mean", [0.5, 0.08])
def test_groups_the_kernel_leaves_to_the_host_are_not_looked_for_twice(monkeypatch, mean):
    """A large mean takes every group's search to the tensor operations: after the first the walk goes on in single steps, as with a
    progress callback, and gives the same encoding."""
    from sbvr import encoder
    g = torch.Generator(device="cuda").manual_seed(1)
    W = (torch.randn((16, 1024), device="cuda", generator=g) * 0.02 + mean).half()
    W[3] = torch.randn(1024, device="cuda", generator=g) * 0.02       # (back to the device for a row)
    conf = encoder.EncoderConfig(num_sums=3)
    one = encoder.encode(W, conf, progress=lambda done, of: None)
    why = _watch_runs(monkeypatch)
    many = encoder.encode(W, conf)
    assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(one[:3], many[:3])) and one[3] == many[3]
    assert one[3]["groups"] - one[3]["cache_hits"] > 10 and 1 <= len(why) <= 6, (one[3], why)
