"""Prefill attention on the tensor cores (csrc/attention_prefill.cu): blocks of 128 (token, head) pairs, tiles of 64 keys.

Bound: fp32 scores, weights in two fp16 parts (2^-22), fp32 sums, one fp16 rounding of the result: 2^-11 of an element, 2.9e-4 in 2-norm at most;
asserted 4e-4 in 2-norm and 1e-3 of the largest.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu
D = 128


def run(qkv, K, V, pos, tps, nh, nkv, scale=D ** -0.5):
    from sbvr import _lib
    T, mc = qkv.shape[0], K.shape[2]
    out = torch.full((T, nh * D), float("nan"), dtype=torch.float16, device="cuda")
    _lib.check(_lib.lib.sbvr_attention_f16(qkv.data_ptr(), K.data_ptr(), V.data_ptr(), pos.data_ptr(), out.data_ptr(), None, T, tps,
                                           nh, nkv, D, mc, scale, 1, torch.cuda.current_stream().cuda_stream))
    return out


def oracle(qkv, K, V, pos, tps, nh, nkv, scale=D ** -0.5):
    B, mc = K.shape[0], K.shape[2]
    q = qkv[:, :nh * D].view(B, tps, nh, D).permute(0, 2, 1, 3).double()
    s = q @ K.double().repeat_interleave(nh // nkv, 1).transpose(2, 3) * scale
    lim = torch.clamp(pos.view(B, 1, tps, 1).long() + 1, max=mc)
    s = s.masked_fill(torch.arange(mc, device="cuda") >= lim, float("-inf"))
    return (torch.softmax(s, -1) @ V.double().repeat_interleave(nh // nkv, 1)).permute(0, 2, 1, 3).reshape(B * tps, nh * D)


def inputs(B, tps, nh, nkv, mc, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    qkv = torch.randn((B * tps, (nh + 2 * nkv) * D), device="cuda", generator=g).half()
    K = torch.randn((B, nkv, mc, D), device="cuda", generator=g).half()
    V = torch.randn((B, nkv, mc, D), device="cuda", generator=g).half()
    return qkv, K, V, g


def close(out, ref):
    e = out.double() - ref
    assert (e.norm() / ref.norm()).item() < 4e-4 and (e.abs().max() / ref.abs().max()).item() < 1e-3


@pytest.mark.parametrize("B,tps,nh,nkv,start", [
    (8, 128, 8, 8, 0),                             # one block per head
    (6, 129, 8, 8, 0),                             # one token in the second block
    (40, 64, 8, 4, 1),
    (20, 63, 32, 8, 600),                          # a block that is not full, on a long context
    (40, 33, 32, 8, 63),                           # contexts that end around the edge of a tile
    (80, 16, 16, 2, 0), (1, 257, 8, 1, 0), (1, 256, 3, 3, 0),
    (1, 1000, 8, 2, 0),
])
def test_against_softmax(B, tps, nh, nkv, start):
    qkv, K, V, _ = inputs(B, tps, nh, nkv, start + tps + 5, tps)
    K[:, :, start + tps:] = float("nan")           # past the last position: not read
    V[:, :, start + tps:] = float("nan")
    pos = (torch.arange(tps, device="cuda", dtype=torch.int32) + start).repeat(B)
    close(run(qkv, K, V, pos, tps, nh, nkv), oracle(qkv, K[:, :, :start + tps], V[:, :, :start + tps], pos, tps, nh, nkv))


def test_positions_in_any_order():
    """Contexts per token: shuffled, the same twice, none at all (a token without keys gives zeros), past the end of the cache."""
    qkv, K, V, g = inputs(2, 260, 8, 2, 300, 1)
    pos = torch.randint(0, 340, (520,), device="cuda", generator=g, dtype=torch.int32)
    out = run(qkv, K, V, pos, 260, 8, 2)
    close(out, oracle(qkv, K, V, pos, 260, 8, 2))
    pos[5], pos[410:] = -1, -1                     # one token, and a whole block at the end
    out2 = run(qkv, K, V, pos, 260, 8, 2)
    assert not out2[5].any() and not out2[410:].any()
    keep = [i for i in range(410) if i != 5]
    assert torch.equal(out2[keep], out[keep])


@pytest.mark.parametrize("step", [0.02, 0.5])
def test_growing_scores(step):
    """Scores that grow along the keys, slowly and fast: the reference of the weights lags behind the maximum and is moved in steps."""
    qkv, K, V, _ = inputs(1, 400, 4, 1, 400, 2)
    ramp = torch.arange(400, device="cuda") * step
    qkv[:, :4 * D] *= 0.2
    qkv.view(400, 6, D)[:, :4, 0] = 8.0
    K[:, :, :, 0] = (ramp * D ** 0.5 / 8.0).half()
    pos = torch.arange(400, device="cuda", dtype=torch.int32)
    close(run(qkv, K, V, pos, 400, 4, 1), oracle(qkv, K, V, pos, 400, 4, 1))


def test_values_that_are_not_finite_stay_with_the_tokens_that_see_them():
    qkv, K, V, _ = inputs(3, 128, 32, 8, 128, 3)
    pos = torch.arange(128, device="cuda", dtype=torch.int32).repeat(3)
    want = run(qkv, K, V, pos, 128, 32, 8)
    V[0, 1, 20, 3] = float("inf")                  # KV head 1 of the first sequence, seen from token 20 on
    K[0, 0, 90, 5] = float("nan")                  # KV head 0, from token 90 on
    out = run(qkv, K, V, pos, 128, 32, 8)
    a, b = out.view(384, 32, D), want.view(384, 32, D)
    assert torch.equal(a[128:], b[128:]) and torch.equal(a[:, 8:], b[:, 8:])
    assert torch.equal(a[:90, :4], b[:90, :4]) and torch.isnan(a[90:128, :4]).all()
    a, b = a[:128, 4:8], b[:128, 4:8]
    seen = torch.isfinite(a)
    assert not seen[20:, :, 3].any() and seen[:20].all() and seen[:, :, :3].all() and seen[:, :, 4:].all()
    e = torch.where(seen, a.double() - b.double(), torch.zeros_like(b.double()))
    assert e.abs().max() / b.abs().max() < 1e-3    # (one fp16 rounding each)


@pytest.fixture(scope="module")
def impatient(tmp_path_factory):
    """The kernel with a wait that runs out (tests/native/attention_timeout.cu)."""
    import ctypes
    import os
    import shutil
    import subprocess
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    so = str(tmp_path_factory.mktemp("native") / "attention_timeout.so")
    subprocess.check_call([nvcc, "-std=c++17", "-O3", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC",
                           "-I", os.path.join(root, "include"), "-I", os.path.join(root, "sbvr-cpu-arm_b200", "csrc"),
                           "-o", so, os.path.join(root, "tests", "native", "attention_timeout.cu")])
    f = ctypes.CDLL(so).attention_with_a_wait_that_runs_out
    f.argtypes = [ctypes.c_void_p] * 5 + [ctypes.c_int] * 5 + [ctypes.c_float] + [ctypes.c_int] * 3 + [ctypes.c_void_p]
    return f


@pytest.mark.parametrize("warp,bar,parity", [
    (4, 0, 0), (4, 1, 1), (4, 2, 1), (4, 8, 0),    # the issuer's wait for the first and the fourth tile of K, the third of V, the first weights
    (5, 4, 0), (6, 7, 0),                          # the warps that bring K and V, for a place
    (2, 5, 1), (0, 4, 0), (3, 6, 0),               # warps that form weights: for scores, for the output
])
def test_a_wait_that_runs_out_costs_time_and_no_result(impatient, warp, bar, parity):
    qkv, K, V, _ = inputs(2, 300, 8, 2, 310, 7)
    pos = (torch.arange(300, device="cuda", dtype=torch.int32) + 8).repeat(2)
    out = torch.full((600, 8 * D), float("nan"), dtype=torch.float16, device="cuda")
    rc = impatient(qkv.data_ptr(), K.data_ptr(), V.data_ptr(), pos.data_ptr(), out.data_ptr(), 600, 300, 8, 2, 310, D ** -0.5, warp, bar, parity,
                   torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    close(out, oracle(qkv, K, V, pos, 300, 8, 2))
