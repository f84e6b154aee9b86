"""The GEMM over CTA pairs (csrc/linear_pair.cu), which the automatic choice takes for many activation rows: edges of its blocks of 256
activation rows, item widths that do not divide N, items split over K, every encoding, and the calls that stay with the one-CTA kernel.

Every case asserts which kernel it runs, so that a rule that moves does not leave this file empty.  Bound: weights are formed in fp16 with one
rounding per plane (a weight is off by at most S fp16 roundings of a partial sum, 2^-11 each), sums are fp32, the result is rounded to fp16:
3.4e-4 of the result in 2-norm at S = 4 as for the one-CTA kernel, 6e-4 of the largest; asserted 5e-4 and 3e-3.
"""
import pytest
import torch

from launched import kernels

pytestmark = pytest.mark.gpu


def packed(N, K, S, G, mode, seed, scale=0.01):
    import sbvr
    g = torch.Generator(device="cuda").manual_seed(seed)
    Kp = -(-K // G) * G
    C = {"u8": 200, "u16": 4096, "direct": 0}[mode]
    bvr = torch.randint(-2 ** 31, 2 ** 31 - 1, (Kp // 32, N, S), dtype=torch.int32, device="cuda", generator=g)
    lines = (torch.randn((C, S) if C else (Kp // G, N, S), device="cuda", generator=g) * scale).half()
    idx = None
    if C:
        idx = torch.randint(0, C, (Kp // G, N), dtype=torch.int32, device="cuda", generator=g)
        idx = idx.to(torch.uint8) if C <= 256 else idx.to(torch.int16).view(torch.uint16)
    return sbvr.sbvr.from_packed(bvr, idx, lines, original_shape=(N, K), group_len=G), g


def errors(y, x, w, b=None):
    ref = x.double() @ w.decode().double().T
    if b is not None:
        ref += b.double()
    d = y.double() - ref
    return (d.norm() / ref.norm()).item(), (d.abs().max() / ref.abs().max()).item()


@pytest.mark.parametrize("M,N,K,S,G,which", [      # us by the GEMM over CTA pairs and by the one-CTA GEMM in loops of calls
    (1100, 14336, 2048, 4, 256, "pair"),           # 71, 78
    (1100, 28672, 512, 4, 128, "pair"),            # 50, 61 in tiles of 384 rows, 73 of 288
    (768, 28672, 512, 3, 256, "pair"),             # 36, 47
    (1024, 4096, 14336, 4, 256, "pair"),           # 111, 124
    (2048, 4096, 14336, 4, 256, "pair"),           # 194, 236
    (384, 1024, 4096, 3, 256, "gemm"),             # 22.8, 19.2
    (600, 14336, 2176, 4, 128, "gemm"),            # 46.2, 46.2
    (384, 28672, 8192, 4, 128, "gemm"),            # 193, 177
    (300, 4096, 14336, 4, 256, "gemm"),            # 57, 41
])
def test_the_faster_kernel_is_chosen(M, N, K, S, G, which):
    import sbvr
    w, g = packed(N, K, S, G, "u16", 1)
    x = torch.randn((M, K), device="cuda", generator=g).half()
    runs(lambda: sbvr.linear(x, w), which == "pair", S)


def runs(call, pair, S, cut=None):
    """Asserts which GEMM `call` runs, and whether (`cut`) sums of items that several pairs share are added."""
    names = kernels(call)
    assert any(f"linear_pair_kernelILi{S}E" in k for k in names) == pair and any("linear_gemm_kernel" in k for k in names) != pair, names
    assert cut is None or any("gp_add_kernel" in k for k in names) == cut, names


def product(M, N, K, S, G, mode, bias, pair, cut=None):
    import sbvr
    w, g = packed(N, K, S, G, mode, M + N + K)
    x = torch.randn((M, K), device="cuda", generator=g).half()
    b = torch.randn(N, device="cuda", generator=g).half() if bias else None
    runs(lambda: sbvr.linear(x, w, b), pair, S, cut)
    y = sbvr.linear(x, w, b)
    rel, top = errors(y, x, w, b)
    assert rel <= 5e-4 and top <= 3e-3, (rel, top)
    assert torch.equal(y, sbvr.linear(x, w, b))    # sums in a fixed order


@pytest.mark.parametrize("M,N,K,S,G,mode,bias,cut", [
    (257, 28672, 256, 4, 256, "u16", False, False),            # one row in the second block; a single group
    (512, 28672, 256, 2, 256, "u8", True, False),              # both blocks full
    (513, 28672, 384, 3, 128, "direct", False, False),         # one row in the third block, an odd number of groups of 128
    (768, 14464, 512, 4, 256, "direct", True, False),          # items of one block; 113 tiles of 128 rows, a last item that is narrower
    (768, 7168, 768, 4, 128, "u8", False, False),
    (448, 14336, 768, 4, 256, "u16", True, False),             # a last block that is not full
    (1000, 9600, 1536, 3, 256, "u16", True, False),
    (1280, 6016, 1408, 4, 128, "u16", True, False),            # 11 groups of 128: every slot of their ring several times; items of one block last
    (1280, 5760, 1408, 2, 128, "direct", False, False),
    (1800, 4224, 2432, 4, 128, "direct", True, False),         # 19 groups
    (1280, 28672, 512, 3, 256, "u8", True, False),             # five rounds of items
    (2048, 4096, 4000, 4, 256, "u16", False, False),           # K padded to the group: x ends before the weight
    (511, 1024, 2432, 4, 128, "u16", True, True),              # fewer items than pairs: all split over K
    (512, 640, 3968, 3, 128, "direct", False, True),           # 31 groups
    (511, 1152, 2304, 3, 256, "u8", True, True),
    (512, 896, 2816, 2, 256, "u16", False, True),              # a last item that is narrower
    (1100, 1920, 6400, 4, 256, "direct", True, True),          # items of one block, split
    (1750, 5632, 5248, 4, 128, "u16", False, True),            # whole rounds, items of two blocks and of one split
    (1000, 9600, 4352, 4, 256, "u16", True, True),             # whole rounds and split items
])
def test_pair_gemm(M, N, K, S, G, mode, bias, cut):
    product(M, N, K, S, G, mode, bias, True, cut)


@pytest.mark.parametrize("M,N,K,S,G,mode,bias", [
    (600, 14336, 2176, 4, 128, "u16", True),
    (1030, 13440, 2048, 2, 128, "u8", False),
    (2048, 1024, 4096, 4, 256, "u16", True),
    (300, 4096, 14336, 4, 256, "u8", False),
    (700, 1152, 14336, 3, 128, "u16", True),
    (3000, 4096, 3072, 2, 256, "u16", False),
])
def test_sizes_that_the_one_cta_kernel_serves(M, N, K, S, G, mode, bias):
    product(M, N, K, S, G, mode, bias, False)


def test_pair_gemm_large_coefficients_and_special_rows():
    """|c| >= 3.9 takes the sign-flip form; a row with an infinite or NaN activation spoils itself alone."""
    import sbvr
    w, g = packed(28672, 512, 4, 256, "u16", 5, scale=4.0)
    x = torch.randn((600, 512), device="cuda", generator=g).half() * 0.01
    runs(lambda: sbvr.linear(x, w), True, 4)
    clean = sbvr.linear(x, w)
    rel, top = errors(clean, x, w)
    assert rel <= 6e-4 and top <= 3e-3, (rel, top)          # (sums of coefficients of either sign: partial sums are larger than weights)
    x[255, 7], x[256, 100], x[599, 511] = float("inf"), float("nan"), -float("inf")
    y = sbvr.linear(x, w)
    bad = torch.zeros(600, dtype=torch.bool, device="cuda")
    bad[[255, 256, 599]] = True
    assert torch.equal(y[~bad], clean[~bad]) and not torch.isfinite(y[bad]).any(dim=1).all()


@pytest.mark.parametrize("case", ["x off by 4 bytes", "row of 514", "y off by 2 bytes"])
def test_calls_that_the_copies_cannot_serve(case):
    """Activations or results that do not start on 16 bytes, rows whose length is no multiple of 16 bytes: the one-CTA kernel, as ever."""
    import sbvr
    K = 514 if case == "row of 514" else 512
    w, g = packed(28672, K, 4, 256, "u16", 9)
    x = torch.randn((512, K), device="cuda", generator=g).half()
    if case == "x off by 4 bytes":
        x = torch.empty(512 * K + 2, dtype=torch.float16, device="cuda")[2:].view(512, K).copy_(x)
    out = None
    if case == "y off by 2 bytes":
        out = torch.empty(512 * 28672 + 1, dtype=torch.float16, device="cuda")[1:].view(512, 28672)
    runs(lambda: sbvr.linear(x, w, None, out=out), False, 4)
    y = sbvr.linear(x, w, None, out=out) if out is not None else sbvr.linear(x, w)
    rel, top = errors(y, x, w)
    assert rel <= 5e-4 and top <= 3e-3, (rel, top)


@pytest.mark.parametrize("M,N,K", [(300, 14336, 512), (448, 14336, 512), (40, 512, 2048)])
def test_first_call_of_a_thread(M, N, K):
    """The first thing that a thread does on the GPU: the tensor map of x is a driver call, which needs the thread's context."""
    import threading
    import sbvr
    w, g = packed(N, K, 4, 256, "u16", 11)
    x = torch.randn((M, K), device="cuda", generator=g).half()
    want, out = sbvr.linear(x, w), torch.empty((M, N), dtype=torch.float16, device="cuda")
    same = []

    def work():
        sbvr.linear(x, w, out=out)
        same.append(torch.equal(out, want))

    torch.cuda.synchronize()
    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert same == [True]
