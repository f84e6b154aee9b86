"""Sizes at the edges of the kernels' tiles, through the package API, against the oracle.

Tolerance of the linears: max|y - ref| / max|ref| <= 2e-3 (one fp16 rounding of the result, 2^-11, and weights formed in
fp16 with one rounding per plane, about 2^-11 each: measured near 6e-4)."""
import numpy as np
import pytest
import torch

from oracle import sbvr_oracle as O
from test_gpu_parity import check_status, h2n, to_sbvr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 3, 5, 37, 130])
@pytest.mark.parametrize("N", [40, 128, 129, 1000])
@pytest.mark.parametrize("K", [120, 256, 1000])
@pytest.mark.parametrize("S,mode", [(2, "u8"), (3, "u8"), (4, "u16"), (4, "direct")])
def test_linear_any_rows_any_inner_length(M, N, K, S, mode):
    import sbvr
    Kp = -(-K // 256) * 256
    p = O.make_packed(N, Kp, S, G=256, mode=mode, C=256 if mode == "u8" else 1000, seed=N + K + S)
    w = to_sbvr(p)
    w.original_data_shape = torch.Size((N, K))
    rng = np.random.default_rng(M)
    x = rng.standard_normal((M, K)).astype(np.float16)
    bias = rng.standard_normal(N).astype(np.float16)
    y = h2n(sbvr.linear(torch.from_numpy(x).cuda(), w, torch.from_numpy(bias).cuda()))
    xp = np.zeros((M, Kp), np.float16)
    xp[:, :K] = x
    ref = O.linear_c(xp, p["bvr"], p.get("coeff_idx"), p["coeff"], G=256).astype(np.float64) + bias
    assert y.shape == (M, N)
    assert np.abs(y - ref).max() / np.abs(ref).max() <= 2e-3
    check_status()


@pytest.mark.parametrize("M,N,K,S", [(257, 19072, 256, 4), (257, 19072, 512, 2), (700, 14300, 512, 3), (700, 14336, 1000, 4), (1500, 4000, 256, 2)])
def test_linear_wide_tiles(M, N, K, S):
    """Sizes that take tiles of more than 256 activation rows (288, 352, 384) on a GPU of 148 SMs, with ragged last tiles."""
    test_linear_any_rows_any_inner_length(M, N, K, S, "u16")


@pytest.mark.parametrize("N,K", [(1, 256), (31, 250), (33, 8), (64, 1000), (40, 777)])
@pytest.mark.parametrize("S", [1, 3, 4, 6])
def test_decode_ragged_bit_exact(N, K, S):
    Kp = -(-K // 256) * 256
    p = O.make_packed(N, Kp, S, G=256, mode="u8", C=200, seed=N + K)
    w = to_sbvr(p)
    w.original_data_shape = torch.Size((N, K))
    ref = O.decode_c(p["bvr"], p["coeff_idx"], p["coeff"], G=256)[:, :K]
    assert np.array_equal(h2n(w.decode()).view(np.uint16), np.ascontiguousarray(ref).view(np.uint16))


@pytest.mark.parametrize("tps", [8, 31, 64, 65, 200])
@pytest.mark.parametrize("nh,nkv", [(2, 2), (4, 2), (8, 2), (16, 2)])
def test_prefill_attention_against_softmax(tps, nh, nkv):
    """Query heads per KV head 1, 2, 4, 8; the tokens continue a context that is already in the cache; the last positions fall
    beyond the cache (they attend to all of it).  fp32 scores and weights, one fp16 rounding (2^-11) of the result."""
    from sbvr import _lib
    d, B, mc, start = 128, 2, 150, 7
    g = torch.Generator(device="cuda").manual_seed(tps + nh)
    T = B * tps
    qkv = torch.randn((T, (nh + 2 * nkv) * d), device="cuda", generator=g).half()
    K = torch.randn((B, nkv, mc, d), device="cuda", generator=g).half()
    V = torch.randn((B, nkv, mc, d), device="cuda", generator=g).half()
    pos = (torch.arange(tps, device="cuda", dtype=torch.int32) + start).repeat(B)
    out = torch.full((T, nh * d), float("nan"), dtype=torch.float16, device="cuda")
    _lib.check(_lib.lib.sbvr_attention_f16(qkv.data_ptr(), K.data_ptr(), V.data_ptr(), pos.data_ptr(), out.data_ptr(), None, T, tps,
                                           nh, nkv, d, mc, d ** -0.5, 1, torch.cuda.current_stream().cuda_stream))
    q = qkv[:, :nh * d].view(B, tps, nh, d).permute(0, 2, 1, 3).double()
    kk = K.double().repeat_interleave(nh // nkv, 1)
    vv = V.double().repeat_interleave(nh // nkv, 1)
    s = q @ kk.transpose(2, 3) * d ** -0.5
    lim = torch.clamp(pos[:tps].long() + 1, max=mc)
    s = s.masked_fill(torch.arange(mc, device="cuda")[None, None, None, :] >= lim[None, None, :, None], float("-inf"))
    ref = (torch.softmax(s, -1) @ vv).permute(0, 2, 1, 3).reshape(T, nh * d)
    assert ((out.double() - ref).abs().max() / ref.abs().max()).item() < 1e-3


@pytest.mark.parametrize("S", [2, 3, 4])
@pytest.mark.parametrize("extended", [False, True])
def test_search_kernel_equals_the_tensor_operations(S, extended):
    """The winner of the search kernel, which generates the candidates itself, is bit for bit that of the search space made by
    the tensor operations: data scales over three decades, a stored line good enough to win, groups the kernel leaves to
    its caller."""
    from sbvr import _lib, encoder
    import ctypes
    conf = encoder.EncoderConfig(num_sums=S)
    dev = torch.device("cuda")
    g = torch.Generator(device="cuda").manual_seed(S)
    scale = 10 ** torch.linspace(-3, -0.3, 24, device="cuda")
    data = (torch.randn((24, 256), device="cuda", generator=g) * scale[:, None]).half()
    data[5] = data[5].abs()
    data[7] += 2.0
    tables = encoder._SearchTables(conf, dev)
    stats = torch.empty((24, 4), device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.lib.sbvr_encode_stats_f16(data.data_ptr(), 24, stats.data_ptr(), st))
    assert torch.equal(stats[:, 0], data.float().amax(1)) and torch.equal(stats[:, 1], data.float().amin(1))
    assert torch.equal(stats[:, 2], torch.quantile(data.float(), 0.95, dim=1))
    pinned = torch.empty(ctypes.sizeof(_lib.EncodeResult), dtype=torch.uint8, pin_memory=True)
    res = _lib.EncodeResult.from_address(pinned.data_ptr())
    lines = torch.zeros((4, S), dtype=torch.float16, device="cuda")
    scratch = torch.empty(2, dtype=torch.int64, device="cuda")
    at = torch.zeros(24, dtype=torch.int32, device="cuda")
    for i in range(24):
        # hits / seen of the groups before decides whether the search is extended
        mse = torch.full((24,), float("inf"), device="cuda")
        w = _lib.EncodeWalk(data=data.data_ptr(), stats=stats.data_ptr(), lines=lines.data_ptr(), best_mse=mse.data_ptr(),
                            best_at=at.data_ptr(), scratch=scratch.data_ptr(), result=pinned.data_ptr(), S=S, groups=24,
                            s_search_num=conf.s_search_num, extend_ratio=conf.extend_ratio, append_at=-1, from_=i, search=1,
                            warm=int(extended), misses=i, cutoff=0.0)
        for e in (0, 1):
            w.unit[e], w.bias[e] = tables.unit[e].data_ptr(), tables.bias[e].data_ptr()
            w.R[e], w.B[e], w.per_dim[e] = tables.unit[e].shape[0], tables.bias[e].shape[0], tables.per_dim[e]
        _lib.check(_lib.lib.sbvr_encode_advance(ctypes.byref(w), st))
        assert res.group == i
        if res.status == 2:                        # 7: a large mean; 5: perhaps an empty scale range (max - min below twice the quantile)
            assert i in (5, 7)
            continue
        assert i != 7
        best, line = encoder._full_search(data[i], conf, extended)
        assert res.status == 1 and res.mse == best, (i, res.status, res.mse, best)
        assert np.array_equal(encoder._sorted_line(res.line, S, dev).view(np.uint16), line.view(np.uint16)), i
        # a stored line that is exactly as good keeps its place
        mse[i] = best
        _lib.check(_lib.lib.sbvr_encode_advance(ctypes.byref(w), st))
        assert res.status == (1 if extended else 0)            # (a warm-up step looks at no stored line)


@pytest.mark.parametrize("N,K,G", [(32, 1, 32), (96, 77, 32), (256, 255, 256), (512, 3001, 128), (1024, 5000, 256)])
@pytest.mark.parametrize("S", [2, 3, 4])
@pytest.mark.parametrize("M", [1, 2, 3, 5, 8, 9])
def test_transposed_layout_ragged(N, K, G, S, M):
    """Group lengths down to one word row, odd input counts, both kernels; activations over six decades.  One
    fp16 rounding of the result (2^-11) and 2^-30 of the largest product for every plane bit."""
    from sbvr import sbvr_cuda
    p = O.make_packed(K, N, S, G=G, mode="u8", C=200, seed=N + K + S)
    rng = np.random.default_rng(M)
    x = (rng.standard_normal((M, K)) * 10.0 ** rng.uniform(-4, 2, (M, 1))).astype(np.float16)
    bias = rng.standard_normal(N).astype(np.float16)
    f = lambda a: torch.from_numpy(a).cuda()
    y = sbvr_cuda._sbvr_row_deq_mm_T(f(x), f(p["bvr"].view(np.int32)), f(p["coeff_idx"]), f(p["coeff"]), f(bias))
    ref = O.linear_t_f64(x, p["bvr"], p["coeff_idx"], p["coeff"], bias, G=G)
    err = np.abs(h2n(y).astype(np.float64) - ref).max(1) / np.abs(ref).max(1)
    assert err.max() <= 1e-3, err
    if M > 1:                                      # a non-finite activation stays in its row
        x[1, K // 2] = np.inf
        z = h2n(sbvr_cuda._sbvr_row_deq_mm_T(f(x), f(p["bvr"].view(np.int32)), f(p["coeff_idx"]), f(p["coeff"]), f(bias)))
        assert np.array_equal(z[0], h2n(y)[0]) and not np.isfinite(z[1]).any()
    check_status()


@pytest.mark.parametrize("N", [3, 64, 333])
@pytest.mark.parametrize("K", [256, 768, 4352])
@pytest.mark.parametrize("LS,RS", [(2, 3), (3, 2), (4, 4), (2, 4)])
@pytest.mark.parametrize("M", [1, 2, 5, 17])
def test_product_of_two_encodings_edges(N, K, LS, RS, M):
    """Fewer groups than warps, rows that do not fill a tile, several passes over the activation rows; exact counts and fp32
    sums, one fp16 rounding (2^-11)."""
    import sbvr
    pl = O.make_packed(M, K, LS, G=256, mode="u8", seed=M + LS)
    pr = O.make_packed(N, K, RS, G=256, mode="u16", C=300, seed=N + RS)
    y = h2n(sbvr.mm_T(to_sbvr(pl), to_sbvr(pr))).astype(np.float64)
    ref = O.popc_mm_f64(pl["bvr"], pl["coeff_idx"], pl["coeff"], pr["bvr"], pr["coeff_idx"], pr["coeff"], None)
    assert np.abs(y - ref).max() / np.abs(ref).max() <= 1e-3


@pytest.mark.parametrize("M", [1, 2, 4, 5, 16])
@pytest.mark.parametrize("N,K", [(96, 512), (64, 4096), (160, 8192), (128, 14336)])
@pytest.mark.parametrize("op", ["norm", "norm_nodelta", "silu"])
def test_ops_folded_into_decode_linears(M, N, K, op):
    """The op in front of the linear, applied in its kernels, against the separate kernels followed by the linear: the new
    residual is exact; the product differs where a normalised value lands on the other side of an fp16 rounding (the sum of
    squares is formed in another order), 2^-11 of single elements."""
    import sbvr
    from sbvr import _lib
    from sbvr.core import XOP_ADD_RMSNORM, XOP_SILU_MUL, linear_fused
    p = O.make_packed(N, K, 4, G=256, mode="u8", seed=N + K)
    w = to_sbvr(p)
    g = torch.Generator(device="cuda").manual_seed(M + K)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=g).half()
    st = torch.cuda.current_stream().cuda_stream
    y = torch.empty((M, N), dtype=torch.float16, device="cuda")
    if op == "silu":
        gu, act = rnd(M, 2 * K), torch.empty((M, K), dtype=torch.float16, device="cuda")
        _lib.check(_lib.lib.sbvr_silu_mul_f16(gu.data_ptr(), act.data_ptr(), M, K, st))
        assert linear_fused(XOP_SILU_MUL, gu, w, y)
    else:
        h, d, nw = rnd(M, K), rnd(M, K) if op == "norm" else None, 1 + 0.1 * rnd(K)
        act, ho, ho2 = torch.empty_like(h), torch.empty_like(h), torch.empty_like(h)
        _lib.check(_lib.lib.sbvr_add_rmsnorm_f16(h.data_ptr(), None if d is None else d.data_ptr(), nw.data_ptr(), ho.data_ptr(),
                                                 act.data_ptr(), M, K, 1e-5, st))
        assert linear_fused(XOP_ADD_RMSNORM, h, w, y, delta=d, norm_weight=nw, h_out=ho2, eps=1e-5)
        assert torch.equal(ho, ho2)
    ref = sbvr.linear(act, w).float()
    assert ((y.float() - ref).abs().max() / ref.abs().max()).item() < (1e-6 if op == "silu" and M <= 4 else 2e-3)
    check_status()


def _planes(p, G):
    """Plane bits [S, N, K] and the coefficients of every element [S, N, K], in fp64."""
    KW, N, S = p["bvr"].shape
    bits = ((p["bvr"].transpose(2, 1, 0)[..., None] >> np.arange(32, dtype=np.uint32)) & 1).reshape(S, N, KW * 32)
    c = p["coeff"].astype(np.float64)
    c = c[p["coeff_idx"].astype(np.int64)] if p.get("coeff_idx") is not None else c
    return bits.astype(np.float64), np.repeat(c.transpose(2, 1, 0), G, axis=2)


@pytest.mark.parametrize("M", [5, 16])
@pytest.mark.parametrize("N,K,G,S,mode", [(256, 2048, 256, 4, "u16"), (96, 4096, 128, 3, "u8"), (128, 768, 256, 2, "direct")])
@pytest.mark.parametrize("power", [8, 11, 13, 15])
@pytest.mark.parametrize("algo", [0, 4])
def test_one_large_activation_among_small_ones(M, N, K, G, S, mode, power, algo):
    """One activation of 2^power in every block of 256 values near one; half of the outputs have no plane bit there and must
    come out as if it were not.  Error per output: one fp16 rounding (2^-11 of the value), and fp32 sums of up to K products per
    plane, 2^-18 of the sum of their magnitudes (the activations themselves are held to 2^-33 of their block's largest)."""
    import sbvr
    p = O.make_packed(N, K, S, G=G, mode=mode, C=256 if mode == "u8" else 1000, seed=N + power)
    rng = np.random.default_rng(M + power)
    x = rng.standard_normal((M, K)).astype(np.float16)
    at = np.arange(0, K, 256) + rng.integers(0, 256, K // 256)
    x[:, at] = (np.exp2(power) * rng.uniform(1.0, 1.9, (M, K // 256))).astype(np.float16)
    for k in at:
        p["bvr"][k // 32, :N // 2, :] &= np.uint32(~(1 << (k % 32)) & 0xFFFFFFFF)
    bits, c = _planes(p, G)
    ref = x.astype(np.float64) @ (bits * c).sum(0).T
    mass = np.abs(x.astype(np.float64)) @ (bits * np.abs(c)).sum(0).T
    y = h2n(sbvr.linear(torch.from_numpy(x).cuda(), to_sbvr(p), None, algo=algo)).astype(np.float64)
    ok = np.abs(ref) < 65000
    assert ok[:, :N // 2].all()
    assert (np.abs(y - ref) <= 2.0 ** -11 * np.abs(ref) + 2.0 ** -18 * mass + 2.0 ** -25)[ok].all()
    check_status()


@pytest.mark.parametrize("M", [3, 17, 64, 65, 130, 300])
@pytest.mark.parametrize("N,K,S,mode", [(40, 1024, 3, "u8"), (1000, 2048, 4, "u16"), (129, 512, 2, "direct"), (3000, 768, 4, "u8")])
def test_odd_row_counts_keep_fp32_weights(M, N, K, S, mode):
    """Rows that are no multiple of 128: weights are not rounded to fp16.  Error per output: one fp16 rounding of the result (2^-11 of
    the value) and fp32 sums, 2^-18 of the sum of their products' magnitudes (fp16 weights would add 2^-11 of every product).  An
    infinite activation gives what the CUDA-core kernel gives."""
    import sbvr
    p = O.make_packed(N, K, S, G=256, mode=mode, C=256 if mode == "u8" else 1000, seed=N + K)
    p["coeff"][0] = np.float16(1.5) * np.arange(1, S + 1) / S          # some weights far above the others
    rng = np.random.default_rng(M)
    x = rng.standard_normal((M, K)).astype(np.float16)
    x[0] = 0                                       # an output of almost nothing: a cancelling pair
    x[0, :2] = 1, -1
    bits, c = _planes(p, 256)
    ref = x.astype(np.float64) @ (bits * c).sum(0).T
    mass = np.abs(x.astype(np.float64)) @ (bits * np.abs(c)).sum(0).T
    w = to_sbvr(p)
    y = h2n(sbvr.linear(torch.from_numpy(x).cuda(), w, None)).astype(np.float64)
    assert (np.abs(y - ref) <= 2.0 ** -11 * np.abs(ref) + 2.0 ** -18 * mass + 2.0 ** -25).all()
    x[1, K // 3] = np.inf
    x[2, 5] = -np.inf
    xt = torch.from_numpy(x).cuda()
    y, z = h2n(sbvr.linear(xt, w, None)), h2n(sbvr.linear(xt, w, None, algo=1))
    assert np.array_equal(np.isnan(y), np.isnan(z)) and np.array_equal(np.isinf(y), np.isinf(z))
    assert np.array_equal(np.sign(y[np.isinf(z)]), np.sign(z[np.isinf(z)])) and np.isinf(z).any()
    check_status()


def test_threads_on_one_stream():
    """Calls of several threads on the stream they share: a quantiser and the product that reads its digits, a GEMM and the
    launch that adds its sums, stay together."""
    import threading
    import sbvr
    N, K = 512, 2048
    w = to_sbvr(O.make_packed(N, K, 4, G=256, mode="u16", C=1000, seed=5))
    g = torch.Generator(device="cuda").manual_seed(3)
    xs = [torch.randn((m, K), device="cuda", generator=g).half() for m in (16, 5, 40, 12, 3, 64)]
    want = [sbvr.linear(x, w) for x in xs]
    bad = []

    def work(i):
        for _ in range(200):
            if not torch.equal(sbvr.linear(xs[i], w), want[i]):
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(xs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    check_status()


@pytest.mark.parametrize("N,K,G,S,M", [(1056, 2401, 32, 3, 8), (1024, 4999, 64, 2, 5), (2048, 2816, 128, 4, 3), (1024, 2304, 256, 4, 8),
                                       (4096, 4352, 256, 3, 1), (8192, 2304, 256, 2, 1), (1024, 3000, 256, 4, 17), (512, 700, 256, 4, 6)])
def test_transposed_layout_one_large_product_among_small_ones(N, K, G, S, M):
    """Every digit width and split of the integer form (the last size: the CUDA-core form), one activation in 200 far above the
    others; outputs n % 32 == 0 have no plane bit there.  Error per output: one fp16 rounding (2^-11), fp32 sums of the parts
    (2^-18 of the sum of the products' magnitudes) and half a step, 2^-30 of the largest product, for every plane bit.  A row
    with an infinite activation comes out as products do."""
    from sbvr import sbvr_cuda
    p = O.make_packed(K, N, S, G=G, mode="u16", C=1000, seed=N + K + S)
    rng = np.random.default_rng(M + K)
    x = rng.standard_normal((M, K)).astype(np.float16)
    at = np.arange(7, K, 200)
    x[:, at] = (2.0 ** 13 * rng.uniform(1.0, 1.9, (M, len(at)))).astype(np.float16)
    p["bvr"][:, at, :] &= np.uint32(0xFFFFFFFE)
    f = lambda a: torch.from_numpy(a).cuda()
    bits = ((f(p["bvr"].view(np.int32)).long()[..., None, :] >> torch.arange(32, device="cuda").view(1, 1, 32, 1)) & 1).double()
    c = f(p["coeff"]).double()[f(p["coeff_idx"].astype(np.int64))].repeat_interleave(G // 32, 0)          # [N/32, K, S]
    xd = f(x).double()
    dense = lambda v: torch.einsum("wkns,wks->wnk", bits, v).reshape(N, K)
    W = dense(c)
    ref, mass = xd @ W.T, xd.abs() @ dense(c.abs()).T
    largest = (xd.abs()[:, None, :] * c.abs().amax((0, 2))).amax(2)
    half_steps = dense(torch.ones_like(c)).sum(1) * largest * 2.0 ** -30
    args = [f(p["bvr"].view(np.int32)), f(p["coeff_idx"].view(np.int16)).view(torch.uint16), f(p["coeff"]), torch.zeros(0).half().cuda()]
    y = sbvr_cuda._sbvr_row_deq_mm_T(f(x), *args).double()
    ok = ref.abs() < 65000
    assert ok[:, ::32].all()
    assert ((y - ref).abs() <= 2.0 ** -11 * ref.abs() + 2.0 ** -18 * mass + half_steps + 2.0 ** -25)[ok].all()
    if M > 1:
        xi = x.copy()
        xi[1, K // 2] = -np.inf
        z, want = sbvr_cuda._sbvr_row_deq_mm_T(f(xi), *args).double(), f(xi).double() @ W.T
        assert torch.equal(torch.isnan(z[1]), torch.isnan(want[1]))
        inf = torch.isinf(want[1])
        assert inf.any() and torch.equal(z[1][inf], want[1][inf]) and torch.equal(z[0], y[0])
    check_status()


@pytest.mark.parametrize("N", [7120, 14333])
@pytest.mark.parametrize("K", [256, 1280])
@pytest.mark.parametrize("LS,RS", [(2, 3), (3, 2), (4, 4), (2, 4)])
@pytest.mark.parametrize("M", [1, 2, 3])
def test_product_of_two_encodings_many_rows(N, K, LS, RS, M):
    """One or two activation rows on many weight rows (popcount instructions) and their neighbours (tensor cores); exact counts and
    fp32 sums, one fp16 rounding (2^-11)."""
    test_product_of_two_encodings_edges(N, K, LS, RS, M)


@pytest.mark.parametrize("scale", [-0.05, 0.0, 0.2])
@pytest.mark.parametrize("tps", [31, 130])
def test_prefill_attention_any_scale(scale, tps):
    """A negative scale prefers the smallest products, a scale of zero averages; fp32 scores and weights, one fp16 rounding."""
    from sbvr import _lib
    nh, nkv, d, mc = 4, 2, 128, 150
    g = torch.Generator(device="cuda").manual_seed(tps)
    qkv = torch.randn((tps, (nh + 2 * nkv) * d), device="cuda", generator=g).half()
    K = torch.randn((1, nkv, mc, d), device="cuda", generator=g).half()
    V = torch.randn((1, nkv, mc, d), device="cuda", generator=g).half()
    pos = torch.arange(tps, device="cuda", dtype=torch.int32)
    out = torch.empty((tps, nh * d), dtype=torch.float16, device="cuda")
    _lib.check(_lib.lib.sbvr_attention_f16(qkv.data_ptr(), K.data_ptr(), V.data_ptr(), pos.data_ptr(), out.data_ptr(), None, tps, tps,
                                           nh, nkv, d, mc, scale, 1, torch.cuda.current_stream().cuda_stream))
    q = qkv[:, :nh * d].view(tps, nh, d).transpose(0, 1).double()
    s = q @ K[0].double().repeat_interleave(nh // nkv, 0).transpose(1, 2) * scale
    s = s.masked_fill(torch.arange(mc, device="cuda") > pos[:, None], float("-inf"))
    ref = (torch.softmax(s, -1) @ V[0].double().repeat_interleave(nh // nkv, 0)).transpose(0, 1).reshape(tps, nh * d)
    assert ((out.double() - ref).abs().max() / ref.abs().max()).item() < 1e-3


def test_kernel_choice_does_not_depend_on_earlier_calls():
    """Three rows that the decode GEMV does not take (activations off a 16-byte boundary), on a weight whose partial sums exceed the
    default workspace: the same bits on a fresh stream and after a larger batch has made the workspace grow."""
    import sbvr
    N, K = 262144, 4096
    g = torch.Generator(device="cuda").manual_seed(1)
    bvr = torch.randint(-2 ** 31, 2 ** 31 - 1, (K // 32, N, 2), dtype=torch.int32, device="cuda", generator=g)
    idx = torch.randint(0, 256, (K // 256, N), device="cuda", generator=g).to(torch.uint8)
    w = sbvr.sbvr.from_packed(bvr, idx, (torch.randn((256, 2), device="cuda", generator=g) * 0.01).half(), group_len=256)
    x = torch.randn(3 * K + 2, device="cuda", generator=g).half()[2:].view(3, K)
    big = torch.randn((64, K), device="cuda", generator=g).half()
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        first = sbvr.linear(x, w)
        sbvr.linear(big, w)
        assert torch.equal(first, sbvr.linear(x, w))
        torch.cuda.synchronize()


@pytest.mark.parametrize("K", [2304, 4352, 14592])
@pytest.mark.parametrize("M,G,mode", [(5, 256, "u16"), (16, 256, "direct"), (32, 256, "u16"), (5, 128, "u8"), (16, 128, "direct")])
@pytest.mark.parametrize("S,N", [(2, 192), (3, 96), (4, 416)])
def test_small_batch_kernel_unequal_chunks(K, M, G, mode, S, N):
    """9, 17 and 57 blocks of 256 k: chunks of K that differ in length."""
    import sbvr
    p = O.make_packed(N, K, S, G=G, mode=mode, C=256 if mode == "u8" else 1000, seed=N + K)
    rng = np.random.default_rng(M)
    x = rng.standard_normal((M, K)).astype(np.float16)
    ref = O.linear_c(x, p["bvr"], p.get("coeff_idx"), p["coeff"], G=G).astype(np.float64)
    w = to_sbvr(p)
    y = sbvr.linear(torch.from_numpy(x).cuda(), w, None, algo=4)
    assert np.abs(h2n(y) - ref).max() / np.abs(ref).max() <= 2e-3
    assert torch.equal(y, sbvr.linear(torch.from_numpy(x).cuda(), w, None, algo=4))
    check_status()


@pytest.mark.parametrize("nh,nkv", [(2, 2), (4, 2), (8, 2), (16, 2)])
@pytest.mark.parametrize("ctx,nsplit", [(1, 16), (5, 16), (5, 2), (70, 8), (300, 2), (1300, 16), (1400, 16), (1301, 1)])
def test_decode_attention_splits(nh, nkv, ctx, nsplit):
    """One query token: every number of query heads per KV head, contexts shorter than the number of splits and beyond the cache
    (all of it is attended to); fp32 scores and weights, one fp16 rounding (2^-11) of the result."""
    from sbvr import _lib
    d, B, mc = 128, 2, 1300
    g = torch.Generator(device="cuda").manual_seed(ctx + nh)
    qkv = torch.randn((B, (nh + 2 * nkv) * d), device="cuda", generator=g).half()
    K = torch.randn((B, nkv, mc, d), device="cuda", generator=g).half()
    V = torch.randn((B, nkv, mc, d), device="cuda", generator=g).half()
    pos = torch.full((B,), ctx - 1, dtype=torch.int32, device="cuda")
    out = torch.full((B, nh * d), float("nan"), dtype=torch.float16, device="cuda")
    scratch = torch.empty(B * nh * nsplit * 130, dtype=torch.float32, device="cuda")
    _lib.check(_lib.lib.sbvr_attention_f16(qkv.data_ptr(), K.data_ptr(), V.data_ptr(), pos.data_ptr(), out.data_ptr(),
                                           scratch.data_ptr(), B, 1, nh, nkv, d, mc, d ** -0.5, nsplit,
                                           torch.cuda.current_stream().cuda_stream))
    n = min(ctx, mc)
    q = qkv[:, :nh * d].view(B, nh, 1, d).double()
    kk, vv = (t[:, :, :n].double().repeat_interleave(nh // nkv, 1) for t in (K, V))
    ref = (torch.softmax(q @ kk.transpose(2, 3) * d ** -0.5, -1) @ vv).reshape(B, nh * d)
    assert ((out.double() - ref).abs().max() / ref.abs().max()).item() < 1e-3


@pytest.mark.parametrize("M", [5, 16])
@pytest.mark.parametrize("N,K,G,S,mode", [(192, 4096, 256, 4, "u16"), (64, 512, 128, 3, "u8"), (256, 2304, 256, 2, "direct")])
@pytest.mark.parametrize("op", ["none", "silu"])
def test_non_finite_activations_of_small_batches(M, N, K, G, S, mode, op):
    """The automatic choice multiplies rows with a non-finite activation out: what the CUDA-core kernel gives, infinities with their
    signs; the other rows keep their bits."""
    import sbvr
    from sbvr import _lib
    from sbvr.core import XOP_SILU_MUL, linear_fused
    p = O.make_packed(N, K, S, G=G, mode=mode, C=256 if mode == "u8" else 1000, seed=N + K)
    w = to_sbvr(p)
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn((M, 2 * K if op == "silu" else K), device="cuda", generator=g).half()

    def call(x):
        if op == "none":
            return sbvr.linear(x, w), sbvr.linear(x, w, None, algo=1)
        y, act = torch.empty((M, N), dtype=torch.float16, device="cuda"), torch.empty((M, K), dtype=torch.float16, device="cuda")
        _lib.check(_lib.lib.sbvr_silu_mul_f16(x.data_ptr(), act.data_ptr(), M, K, torch.cuda.current_stream().cuda_stream))
        assert linear_fused(XOP_SILU_MUL, x, w, y)
        return y, sbvr.linear(act, w, None, algo=1)

    clean = call(x)[0]
    x[0, K // 2], x[1, 3], x[2, K - 1] = float("inf"), float("-inf"), float("nan")
    x[3, 7], x[3, K - 9] = float("inf"), float("-inf")
    y, z = call(x)
    assert torch.equal(y[4:], clean[4:])
    assert torch.equal(torch.isnan(y), torch.isnan(z)) and torch.equal(torch.isinf(y), torch.isinf(z))
    assert torch.isinf(z).any() and torch.equal(y[torch.isinf(z)], z[torch.isinf(z)])
    ok = torch.isfinite(z)
    assert ((y[ok].float() - z[ok].float()).abs().max() / z[ok].float().abs().max()).item() < 1e-3
    check_status()


@pytest.mark.parametrize("M", [5, 16])
@pytest.mark.parametrize("S,G,N,K", [(4, 256, 4096, 4096), (4, 256, 4128, 4096), (2, 256, 64, 8192), (3, 128, 96, 1280), (4, 256, 2048, 4352)])
@pytest.mark.parametrize("what", ["random", "zero weight", "zero rows", "odd y"])
def test_small_batch_kernel_merges_its_chunks(M, S, G, N, K, what):
    """Up to 1 MiB of partial sums (4096 x 4096 fills it exactly, 4128 rows are beyond) an arrived sum is told from an empty slot by its
    bits: sums of zero must arrive too, and the slots must be empty again for the next call.  Tolerance: one rounding of the
    result (2^-11) and fp32 sums."""
    import sbvr
    p = O.make_packed(N, K, S, G=G, mode="u16", C=1000, seed=N + K)
    if what == "zero weight":
        p["coeff"][:] = 0
    rng = np.random.default_rng(M)
    x = rng.standard_normal((M, K)).astype(np.float16)
    if what == "zero rows":
        x[1:] = 0
    ref = O.linear_c(x, p["bvr"], p["coeff_idx"], p["coeff"], G=G).astype(np.float64)
    w, xd = to_sbvr(p), torch.from_numpy(x).cuda()
    buf = torch.full((M * N + 1,), float("nan"), dtype=torch.float16, device="cuda")
    out = buf[1:].view(M, N) if what == "odd y" else buf[:-1].view(M, N)
    sbvr.linear(xd, w, None, algo=4, out=out)
    first = out.clone()
    assert np.abs(h2n(first) - ref).max() <= 1e-3 * max(np.abs(ref).max(), 1e-30)
    assert not torch.signbit(first[first == 0]).any() or what == "random"
    for _ in range(3):
        assert torch.equal(first, sbvr.linear(xd, w, None, algo=4))
    check_status()


def _square_sums(h):
    """Sum of squares of each fp16 row in the order of the decode quantiser: 512 threads take chunks of eight values in turn, two squares
    per fp32 addition; then the lanes of a warp in halves, then sixteen warps one after the other."""
    M, K = h.shape
    d = h.double() ** 2
    pairs = (d[:, 0::2] + d[:, 1::2]).float().view(M, K // 8, 4)           # (squares are exact in fp32: one rounding)
    rounds = -(-K // 4096)
    pairs = torch.nn.functional.pad(pairs, (0, 0, 0, rounds * 512 - K // 8)).view(M, rounds, 512, 4)
    s = torch.zeros((M, 512), device=h.device)
    for r in range(rounds):
        for e in range(4):
            s = s + pairs[:, r, :, e]
    s = s.view(M, 16, 32)
    for o in (16, 8, 4, 2, 1):
        s = s + s[:, :, torch.arange(32, device=h.device) ^ o]
    tot = torch.zeros(M, device=h.device)
    for w in range(16):
        tot = tot + s[:, w, 0]
    return tot


@pytest.mark.parametrize("M", [1, 2, 4])
@pytest.mark.parametrize("K,G", [(256, 256), (2048, 128), (3840, 256), (4096, 256), (4352, 256), (8192, 256), (8192, 128), (10496, 256)])
@pytest.mark.parametrize("with_delta", [False, True])
def test_folded_norm_adds_squares_in_one_order(M, K, G, with_delta):
    """The bits of a folded residual add + RMSNorm do not depend on the quantiser's form (rows, K): those of the norm computed apart,
    squares in the stated order, in front of the plain linear."""
    import sbvr
    from sbvr.core import XOP_ADD_RMSNORM, linear_fused
    N, eps = 256, 1e-5
    w = to_sbvr(O.make_packed(N, K, 4, G=G, mode="u16", C=1000, seed=K + M))
    for seed in range(4):
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn((M, K), device="cuda", generator=g).half()
        delta = torch.randn((M, K), device="cuda", generator=g).half() if with_delta else None
        nw = (1 + 0.1 * torch.randn(K, device="cuda", generator=g)).half()
        y, h_out = torch.empty((M, N), dtype=torch.float16, device="cuda"), torch.empty_like(x)
        assert linear_fused(XOP_ADD_RMSNORM, x, w, y, delta=delta, norm_weight=nw, h_out=h_out, eps=eps)
        h = x + delta if with_delta else x
        assert torch.equal(h_out, h)
        rs = torch.rsqrt(_square_sums(h) / torch.full((M,), float(K), device="cuda") + eps)      # (a division by a number would multiply by its inverse)
        normed = (h.float() * rs[:, None]).half() * nw
        assert torch.equal(y, sbvr.linear(normed, w, None, algo=2))
    check_status()


@pytest.mark.parametrize("K", [20736, 21248, 23808, 24064])
@pytest.mark.parametrize("S,mode", [(2, "u8"), (4, "u16")])
def test_two_long_rows_keep_their_precision(K, S, mode):
    """From K = 21 248 on two rows are not the decode kernel's, whose digits end at 2^-16 of a block's largest value: outputs that do not
    see one activation of 2^13 per block keep the precision of the rest (2^-11 of the result, and fp16 weights: 2e-3), a row with an
    infinity has the infinities of a product, and the kernel asked for by name refuses.  Below, the decode kernel's own results."""
    import sbvr
    from sbvr import _lib
    from sbvr.core import XOP_SILU_MUL, linear_fused
    N = 64
    p = O.make_packed(N, K, S, G=256, mode=mode, C=256 if mode == "u8" else 1000, seed=K + S)
    k = np.arange(K // 256) * 256 + np.random.default_rng(K).integers(0, 256, K // 256)
    p["bvr"][k // 32] &= ~(np.uint32(1) << (k % 32).astype(np.uint32))[:, None, None]
    w = to_sbvr(p)
    g = torch.Generator(device="cuda").manual_seed(S)
    x = torch.randn((2, K), device="cuda", generator=g).half()
    x[0, torch.from_numpy(k).cuda()] = 8192.0
    x[1, K - 5] = float("inf")
    gate = torch.full_like(x, 20.0)
    act, y2 = torch.empty_like(x), torch.empty((2, N), dtype=torch.float16, device="cuda")
    both = torch.cat([gate, (x / 20).half()], 1)
    _lib.check(_lib.lib.sbvr_silu_mul_f16(both.data_ptr(), act.data_ptr(), 2, K, torch.cuda.current_stream().cuda_stream))
    assert linear_fused(XOP_SILU_MUL, both, w, y2)
    y = sbvr.linear(x, w)
    if K == 20736:
        assert torch.equal(y.view(torch.int16), sbvr.linear(x, w, None, algo=2).view(torch.int16))
        return
    for got, rows in ((y, x), (y2, act)):
        ref = sbvr.linear(rows, w, None, algo=1)
        assert ((got[0].float() - ref[0].float()).abs().max() / ref[0].float().abs().max()).item() < 2e-3
        assert torch.equal(torch.isnan(got[1]), torch.isnan(ref[1])) and torch.isinf(ref[1]).any()
        assert torch.equal(got[1][torch.isinf(ref[1])], ref[1][torch.isinf(ref[1])])
    with pytest.raises(RuntimeError):
        sbvr.linear(x, w, None, algo=2)
    check_status()


@pytest.mark.parametrize("M", [5, 16])
@pytest.mark.parametrize("S,G,N,K", [(4, 256, 4096, 4096), (4, 256, 4128, 4096), (2, 256, 64, 8192), (3, 128, 96, 1280), (4, 256, 64, 32768), (4, 256, 512, 14336)])
@pytest.mark.parametrize("patience", [0, 2000])
def test_small_batch_chunks_that_do_not_wait(M, S, G, N, K, patience):
    """CTAs that give up at once, or soon, leave their share of the sums to the last of them: the same bits, slots and words empty again."""
    import sbvr
    from sbvr import _lib
    w = to_sbvr(O.make_packed(N, K, S, G=G, mode="u16", C=1000, seed=N + K))
    x = torch.from_numpy(np.random.default_rng(M).standard_normal((M, K)).astype(np.float16)).cuda()
    x[M - 1, K // 3] = float("nan")
    first = sbvr.linear(x, w, None, algo=4)
    ws = _lib.workspace(torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream)
    assert _lib.lib.sbvr_workspace_patience(ws.handle, patience) == 0
    try:
        for _ in range(20):
            assert torch.equal(first[:-1], sbvr.linear(x, w, None, algo=4)[:-1])
    finally:
        _lib.lib.sbvr_workspace_patience(ws.handle, 1 << 18)
    assert torch.isnan(first[-1]).all() and torch.equal(first[:-1], sbvr.linear(x, w, None, algo=4)[:-1])
    check_status()


def test_small_batch_kernel_on_two_streams_at_once():
    """Two streams whose grids each want every SM: calls of both interleave freely, results are those of a call by itself."""
    import sbvr
    shapes = [(4096, 4096), (2048, 16384), (4128, 4096), (64, 32768)]
    ws = [to_sbvr(O.make_packed(N, K, 4, G=256, mode="u16", C=1000, seed=N + K)) for N, K in shapes]
    xs = [torch.from_numpy(np.random.default_rng(K).standard_normal((16, K)).astype(np.float16)).cuda() for _, K in shapes]
    want = [sbvr.linear(x, w, None, algo=4) for x, w in zip(xs, ws)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1)]
    got = []
    for i in range(60):
        for k, s in enumerate(streams):
            with torch.cuda.stream(s):
                j = (i + k) % len(shapes)
                got.append((j, sbvr.linear(xs[j], ws[j], None, algo=4)))
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[j]) for j, y in got)
    for s in streams:
        with torch.cuda.stream(s):
            check_status()


@pytest.mark.parametrize("S,G,N,K,M,algo", [(4, 256, 4096, 4096, 16, 4), (4, 256, 4096, 14336, 16, 4), (4, 256, 4096, 14336, 5, 4), (4, 128, 14336, 8192, 16, 4),
                                            (2, 256, 8192, 8192, 16, 4), (3, 256, 2048, 11008, 16, 4), (2, 256, 128, 14336, 16, 4), (2, 256, 4096, 4352, 16, 3),
                                            (2, 256, 2048, 6144, 16, 3), (3, 256, 4096, 5120, 16, 3), (4, 128, 4096, 6144, 16, 3), (4, 256, 1024, 14336, 16, 3)])
def test_automatic_choice_of_a_few_rows(S, G, N, K, M, algo):
    """Five to sixteen rows go to whichever of the small-batch kernel and the GEMM was measured to be the faster (by 5 to 40 % in these
    calls), and an op is folded where it is the former."""
    import sbvr
    from sbvr import _lib
    w = to_sbvr(O.make_packed(N, K, S, G=G, mode="u16", C=1000, seed=N + K))
    x = torch.from_numpy(np.random.default_rng(M).standard_normal((M, K)).astype(np.float16)).cuda()
    y, small, gemm = (sbvr.linear(x, w, None, algo=a) for a in (0, 4, 3))
    assert torch.equal(y, small if algo == 4 else gemm) and not torch.equal(small, gemm)
    assert _lib.linear_folds(torch.cuda.current_device(), M, N, K, S, G, 2) == (algo == 4)
