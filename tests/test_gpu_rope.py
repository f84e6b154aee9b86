"""Rotary embedding and cache append in pieces of 16 bytes (csrc/glue.cu) against the element-wise kernel, which serves rows that do not start
on 16 bytes: the same fp16 operations, the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,tps,nh,nkv,d", [(2, 33, 4, 2, 128), (1, 5, 3, 1, 16), (3, 7, 6, 2, 48), (1, 40, 96, 8, 128), (2, 9, 1, 1, 512)])
def test_pieces_equal_elements(B, tps, nh, nkv, d):
    from sbvr import _lib
    g = torch.Generator(device="cuda").manual_seed(tps + d)
    T, mc = B * tps, tps + 2
    qkv = torch.randn((T, (nh + 2 * nkv) * d), device="cuda", generator=g).half()
    pos = (torch.arange(tps, device="cuda", dtype=torch.int32) + 4).repeat(B)              # the last two are past the cache
    inv = 500000.0 ** (-torch.arange(0, d, 2, device="cuda").float() / d)
    out = []
    for shift in (0, 1):
        flat = torch.zeros(qkv.numel() + 8, dtype=torch.float16, device="cuda")
        q = flat[shift:shift + qkv.numel()].view_as(qkv).copy_(qkv)
        K = torch.zeros((B, nkv, mc, d), dtype=torch.float16, device="cuda")
        V = torch.zeros_like(K)
        _lib.check(_lib.lib.sbvr_rope_append_f16(q.data_ptr(), pos.data_ptr(), inv.data_ptr(), 1.1, K.data_ptr(), V.data_ptr(), T, tps, nh, nkv,
                                                 d, mc, torch.cuda.current_stream().cuda_stream))
        out.append((q, K, V))
    for a, b in zip(*out):
        assert torch.equal(a, b)
    assert not torch.equal(out[0][0], qkv) and out[0][1][:, :, 4:].any() and not out[0][1][:, :, :4].any()
