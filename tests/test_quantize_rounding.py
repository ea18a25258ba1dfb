"""The quantisers on quotients at and next to half-integers, where a rounded product in place of the IEEE
quotient would go wrong, and on scales outside the reciprocal's range: bit-identical to the oracle."""
import numpy as np
import pytest
import torch

import locomp_b200 as L
from oracle import qmm_oracle as O

pytestmark = pytest.mark.gpu


def _near_ties(n, k, g, qmax, rng):
    """float32 rows whose groups have amax = qmax * s, so that the scale is s to the bit or next to it, and whose
    other weights are (j + 1/2) * s and its float32 neighbours."""
    s = np.exp2(rng.integers(-6, 3, (n, k // g, 1))).astype(np.float32) * rng.choice([1.0, 1.1, 0.7, 3.0], (n, k // g, 1)).astype(np.float32)
    w = ((rng.integers(-int(qmax), int(qmax), (n, k // g, g)) + 0.5) * s).astype(np.float32)
    step = rng.integers(-2, 3, w.shape).astype(np.int32)
    w = (w.view(np.int32) + step).view(np.float32)
    w[:, :, 0] = (qmax * s)[:, :, 0]
    return w.reshape(n, k)


@pytest.mark.parametrize("g", [8, 32, 256])
@pytest.mark.parametrize("kind", [torch.float32, torch.float16, torch.bfloat16])
def test_ties_and_their_neighbours(g, kind):
    rng = np.random.default_rng(g)
    for bits, qmax, quantise in ((4, 7.0, O.quantize_int4), (8, 127.0, O.quantize_int8)):
        w = torch.from_numpy(_near_ties(33, 1024, g, qmax, rng)).to(kind)
        q_ref, s_ref = quantise(w.float().numpy(), g)
        q = L.quantize(w.cuda(), g, bits=bits)
        assert np.array_equal(q.w.cpu().numpy(), q_ref)
        assert np.array_equal(q.scales.cpu().numpy().view(np.uint32), s_ref.view(np.uint32))


@pytest.mark.parametrize("scale", [1e-38, 1e-31, 1e-29, 1e29, 1e31])
def test_extreme_scales(scale):
    rng = np.random.default_rng(3)
    w = (rng.standard_normal((5, 256)) * scale).astype(np.float32)
    w[1] = 0.0
    for bits, quantise in ((4, O.quantize_int4), (8, O.quantize_int8)):
        q_ref, s_ref = quantise(w, 32)
        q = L.quantize(torch.from_numpy(w).cuda(), 32, bits=bits)
        assert np.array_equal(q.w.cpu().numpy(), q_ref)
        assert np.array_equal(q.scales.cpu().numpy().view(np.uint32), s_ref.view(np.uint32))
