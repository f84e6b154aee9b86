"""Packed weights are read ahead of the wait for the work in front of a call; a weight that is rewritten on the stream right before one is the
weight that the call uses: decoding, and a linear of every kernel."""
import pytest
import torch

from test_gpu_pair import packed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,S,G", [
    (0, 4096, 2048, 4, 256),                       # decode by tables
    (0, 1000, 1000, 3, 256),                       # rows that are stored elsewhere
    (1, 4096, 4096, 4, 256), (3, 1024, 2048, 2, 128), (16, 4096, 4096, 4, 256),
    (64, 4096, 4096, 4, 256), (100, 3001, 1024, 3, 256), (300, 4096, 2048, 4, 128),
    (512, 14336, 512, 4, 256),                     # CTA pairs
    (6, 100, 512, 4, 256),
])
def test_a_weight_rewritten_right_before_a_call(M, N, K, S, G):
    import sbvr
    ws = [packed(N, K, S, G, "u16", seed)[0] for seed in (1, 2)]
    w, g = packed(N, K, S, G, "u16", 3)
    x = torch.randn((max(M, 1), K), device="cuda", generator=g).half()
    call = (lambda v: v.decode()) if M == 0 else (lambda v: sbvr.linear(x, v))
    want = [call(v) for v in ws]
    mine = [w.bvr, w.coeff_idx, w.coeff_cache]
    theirs = [[v.bvr, v.coeff_idx, v.coeff_cache] for v in ws]
    got = []
    for i in range(40):
        for a, b in zip(mine, theirs[i % 2]):
            a.view(torch.uint8).copy_(b.view(torch.uint8))
        got.append(call(w))
    assert not torch.equal(want[0], want[1])
    assert all(torch.equal(y, want[i % 2]) for i, y in enumerate(got))
