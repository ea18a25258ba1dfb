"""One row of x on int4 weights in float32 math: two octets of weights a lane and load, or one: by K, the groups, the address and how the
warps fill the GPU; K that leaves lanes or whole warps without work, shares of K for 1 to 8 warps, weight rows that are no multiple of 4.

Bound: products and sums in float32, in another order than float64's: |err| <= (K / 8 + 16) * 2^-24 * sum |x w|."""
import numpy as np
import pytest
import torch

import locomp_b200 as L
from oracle import qmm_oracle as O

pytestmark = pytest.mark.gpu

# (n, k, g): beyond 2 Mi weights each; g = 8 and 24 and K = 1032 and 1048 have one octet a lane
CASES = [(2101, 1024, 16), (2050, 1024, 8), (2050, 1032, 8), (2049, 1040, 16), (2003, 1048, 8), (1990, 1056, 48), (1900, 1152, 24), (4097, 2048, 32), (3000, 3072, 128),
         (300, 8192, 64), (270, 16384, 16384), (16387, 272, 16), (9001, 512, 256),
         # on 148 SMs: one octet beyond a wave of two, in 1, 4 and 8 shares; two octets in two waves, in 4 shares (16 lanes and a warp idle), in 8, in a second
         # wave of long shares; K = 256; 768 with more than a wave
         (14300, 512, 32), (4001, 768, 48), (2001, 1152, 32), (19001, 272, 16), (2730, 1040, 16), (1399, 1536, 32), (4001, 3600, 16), (8300, 256, 32), (23700, 768, 64)]


@pytest.mark.parametrize("offset", [0, 4, 8])
@pytest.mark.parametrize("kind", [torch.float32, torch.float16])
@pytest.mark.parametrize("n,k,g", CASES)
def test_against_oracle(n, k, g, kind, offset):
    rng = np.random.default_rng(n + k)
    w, s = O.make_w4(rng, n, k, g, np.float32 if kind == torch.float32 else np.float16)
    x = torch.from_numpy(rng.standard_normal((1, k)).astype(np.float32)).to(kind)
    dq = O.dequant_int4(w, s, g).astype(np.float64)
    ref, mag = x.double().numpy() @ dq.T, np.abs(x.double().numpy()) @ np.abs(dq).T
    raw = torch.zeros(w.size + 512, dtype=torch.uint8, device="cuda")
    placed = raw[offset:offset + w.size].view(n, k // 2)
    placed.copy_(torch.from_numpy(w))
    y = L.quantized_matmul(x.cuda(), placed, torch.from_numpy(s).cuda(), g, algo="simt", out_dtype="f32")
    assert np.all(np.abs(y.double().cpu().numpy() - ref) <= (k / 8 + 16) * 2.0 ** -24 * mag)
