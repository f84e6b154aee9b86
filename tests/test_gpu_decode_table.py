"""Decoding by tables of a group's values (csrc/decode.cu): bit for bit what the sums in fp32 in plane order give, rounded once, over ragged
rows and inner lengths, every index form, special coefficients, and destinations and group lengths that stay with the other kernel."""
import numpy as np
import pytest
import torch

from oracle import sbvr_oracle as O
from test_gpu_parity import h2n, to_sbvr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(1, 8), (33, 40), (31, 256), (64, 264), (129, 504), (300, 1000), (96, 2560)])
@pytest.mark.parametrize("S,G,mode", [(2, 256, "u8"), (3, 128, "u16"), (4, 256, "u16"), (4, 128, "direct"), (3, 256, "direct"), (2, 128, "u16")])
def test_decode_table_bit_exact(N, K, S, G, mode):
    Kp = -(-K // G) * G
    p = O.make_packed(N, Kp, S, G=G, mode=mode, C=200 if mode == "u8" else 300, seed=N + K + S)
    c = p["coeff"].reshape(-1, S)                  # special values: signed zeros, the smallest and the largest numbers, infinities, NaN
    c[0] = np.float16(-0.0)
    c[len(c) // 2] = [np.float16(6e-8), np.float16(65504.0), np.float16(-65504.0), np.float16(0.1)][:S]
    c[len(c) // 3] = [np.float16(np.inf), np.float16(-np.inf), np.float16(1.0), np.float16(np.nan)][:S]
    w = to_sbvr(p)
    w.original_data_shape = torch.Size((N, K))
    with np.errstate(over="ignore", invalid="ignore"):
        ref = O.decode_c(p["bvr"], p.get("coeff_idx"), p["coeff"], G=G)[:, :K]
    got, nan = h2n(w.decode()), np.isnan(ref)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got.view(np.uint16)[~nan], np.ascontiguousarray(ref).view(np.uint16)[~nan])
