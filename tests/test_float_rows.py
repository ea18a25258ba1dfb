"""The float kernel that gives a warp four weight rows: rows of x around its block of 4, weight rows that are no
multiple of 4, K that leaves lanes without work, shared between 1 to 8 warps.

Bound: products and sums in float32, in another order than the oracle's float64: |err| <= (K / 8 + 16) * 2^-24 *
sum |x w| (at most K / 256 chunk sums of 8 per lane, 5 shuffle steps, 8 warps)."""
import numpy as np
import pytest
import torch

import locomp_b200 as L
from oracle import qmm_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("m,n,k,g", [(2, 1, 64, 32), (3, 5, 512, 64), (4, 192, 4096, 128), (5, 37, 1032, 8), (8, 1001, 768, 96),
                                     (9, 250, 2048, 2048), (1, 1030, 2056, 8), (1, 16385, 256, 128), (2, 4096, 8192, 32)])
def test_against_oracle(bits, m, n, k, g):
    rng = np.random.default_rng(m + n + k)
    w, s = (O.make_w4 if bits == 4 else O.make_w8)(rng, n, k, g, np.float32)
    x = rng.standard_normal((m, k)).astype(np.float32)
    dq = (O.dequant_int4 if bits == 4 else O.dequant_int8)(w, s, g).astype(np.float64)
    ref, mag = x.astype(np.float64) @ dq.T, np.abs(x).astype(np.float64) @ np.abs(dq).T
    y = L.quantized_matmul(torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda(), torch.from_numpy(s).cuda(), g, bits=bits)
    assert np.all(np.abs(y.double().cpu().numpy() - ref) <= (k / 8 + 16) * 2.0 ** -24 * mag)
