"""The one-CTA GEMM (csrc/linear_gemm.cu): widths of its tiles of activation rows, row counts that are no multiple of 128, tiles cut into
windows of 256 k and the sums added by the second kernel, windows of two stages, activations that TMA cannot read, every encoding.

Bound: N a multiple of 128: weights formed in fp16 with one rounding per plane (off by at most S fp16 roundings of a partial sum, 2^-11 each),
sums in fp32, the result rounded to fp16: 3.6e-4 of the result in 2-norm at S = 4, asserted 5e-4 and 3e-3 of the largest.  Else weights in
two parts, off by 2^-21: the rounding of the result, 2.1e-4 in 2-norm, beside the reference's weights, which are rounded to fp16 once
(2.1e-4 again): together 3e-4, asserted 4e-4 and 3e-3.
"""
import pytest
import torch

from launched import kernels
from test_gpu_pair import errors, packed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,S,G,mode,bias", [
    (17, 128, 256, 4, 256, "u16", True),           # one tile, one window
    (32, 256, 384, 3, 128, "u8", False),           # K cut, the last window two stages long
    (33, 1024, 4096, 4, 256, "u16", True),
    (64, 4096, 2176, 2, 128, "direct", True),      # cut unevenly, windows of two stages
    (65, 1920, 14592, 3, 256, "u16", False),
    (128, 14336, 1024, 4, 128, "u8", True),        # whole tiles
    (129, 1152, 7936, 2, 256, "u8", True),
    (256, 6144, 1152, 4, 128, "u16", False),
    (40, 1, 512, 4, 256, "u16", True),             # row counts that are no multiple of 128
    (64, 19000, 2048, 4, 256, "u16", False),       # 149 tiles: what is left over has fewer windows than there are CTAs
    (100, 18945, 2048, 2, 128, "u8", True),        # the same, rows that do not start on four bytes
    (130, 3533, 3072, 3, 256, "direct", True),
    (257, 1001, 4096, 4, 128, "u16", True),        # two tiles of 256, the second with one row
    (257, 14336, 512, 4, 256, "u16", True),        # more than 256 rows in one tile
    (300, 4096, 8192, 3, 128, "u8", False),
    (352, 28672, 2176, 4, 128, "u16", True),
    (384, 14336, 1536, 2, 256, "direct", False),
    (700, 8192, 1280, 4, 256, "u8", True),
])
def test_gemm(M, N, K, S, G, mode, bias):
    import sbvr
    w, g = packed(N, K, S, G, mode, M + N + K)
    x = torch.randn((M, K), device="cuda", generator=g).half()
    b = torch.randn(N, device="cuda", generator=g).half() if bias else None
    assert any(f"linear_gemm_kernelILi{S}E" in k for k in kernels(lambda: sbvr.linear(x, w, b)))
    y = sbvr.linear(x, w, b)
    rel, top = errors(y, x, w, b)
    assert rel <= (5e-4 if N % 128 == 0 else 4e-4) and top <= 3e-3, (rel, top)
    assert torch.equal(y, sbvr.linear(x, w, b))    # sums in a fixed order


@pytest.mark.parametrize("M,N,K", [(384, 14336, 2176), (353, 13440, 1408), (384, 28672, 2176), (384, 1024, 2176)])
def test_widest_tile_with_groups_of_128(M, N, K):
    """Four planes, groups of 128: the coefficients of one window at a time beside a tile of 384 rows; windows of two stages, two tiles per CTA,
    tiles that are cut."""
    import sbvr
    w, g = packed(N, K, 4, 128, "u16", M + K)
    x = torch.randn((M, K), device="cuda", generator=g).half()
    assert any("linear_gemm_kernelILi4ELi384E" in k for k in kernels(lambda: sbvr.linear(x, w)))
    y = sbvr.linear(x, w)
    rel, top = errors(y, x, w)
    assert rel <= 5e-4 and top <= 3e-3, (rel, top)
    assert torch.equal(y, sbvr.linear(x, w))


@pytest.mark.parametrize("M,N,kin,offset", [(48, 2048, 1024, 2), (48, 2048, 1003, 0), (300, 14336, 509, 2), (100, 1000, 700, 2),
                                             (19, 500, 255, 0), (152, 256, 4095, 0), (153, 256, 4089, 2)])
def test_activations_that_tma_cannot_read(M, N, kin, offset):
    """x off by 4 bytes, rows of a length that is no multiple of 16 bytes: a copy is read instead, the same values."""
    import sbvr
    w, g = packed(N, kin, 4, 256, "u16", 7)
    flat = torch.randn(M * kin + 8, device="cuda", generator=g).half()
    x = flat[offset:offset + M * kin].view(M, kin)
    y = sbvr.linear(x, w)
    rel, top = errors(y, x, w)
    assert rel <= 5e-4 and top <= 3e-3, (rel, top)
    if kin % 8 == 0:
        assert torch.equal(y, sbvr.linear(x.clone(), w))


def test_back_to_back_calls_keep_their_sums_apart():
    """Calls of different splits after one another on a stream: the kernel in front may still be adding when the next one starts."""
    import sbvr
    ws = [packed(N, K, 4, 256, "u16", N) for N, K in ((512, 4096), (1024, 2048), (3000, 1024), (256, 8192))]
    xs = [torch.randn((M, K), device="cuda", generator=g).half()
          for (w, g), M, K in zip(ws, (40, 100, 20, 64), (4096, 2048, 1024, 8192))]
    want = []
    for (w, _), x in zip(ws, xs):
        want.append(sbvr.linear(x, w))
        torch.cuda.synchronize()
    for _ in range(50):
        got = [sbvr.linear(x, w) for (w, _), x in zip(ws, xs)]
        assert all(torch.equal(a, b) for a, b in zip(got, want))
