"""Decode calls whose CTAs take whole row blocks, and those next to them that cut row blocks between CTAs: one row block more
than CTAs, row blocks that come in twos and threes, a last one that is not full, partial k tiles, both sides of the rule.

Bound: exact products, float32 sums of K <= 4096 terms in any order (K * 2^-24 of sum |x w|, here 2^-12), and the fp16 / bf16
output half an ulp of the result."""
import ctypes

import pytest
import torch

import locomp_b200 as L
from locomp_b200 import _lib

CASES = [(1, 64, 37889), (1, 512, 49152), (3, 576, 49000), (8, 320, 76001), (1, 1536, 49152), (1, 2048, 49152), (2, 4096, 28672), (4, 2560, 30000),
         (16, 64, 19000), (9, 512, 57000), (16, 832, 18945), (12, 1536, 32000), (16, 2560, 24576)]
CUT = [(1, 2048, 49152), (16, 2560, 24576), (1, 4096, 40000), (16, 2048, 20000), (3, 2112, 49000), (8, 1856, 40001)]
CASES += [case for case in CUT if case not in CASES]


@pytest.mark.parametrize("m,k,n", CASES)
def test_plan_covers_every_tile_once(m, k, n):
    f = (ctypes.c_int * 8)()
    for rows in (n, n - 128, n + 128, n // 2):
        for sms in (148, 132, 16, 1):
            assert _lib.lib().lcq_gemv_tc_plan_check(m, rows, k, sms, f) == 0, (rows, sms, _lib.lib().lcq_last_error())


@pytest.mark.parametrize("m,k,n", CASES)
def test_side_of_the_rule(m, k, n):
    f = (ctypes.c_int * 8)()
    assert _lib.lib().lcq_gemv_tc_plan_check(m, n, k, 148, f) == 0 and _lib.lib().lcq_gemv_tc_plan_cluster(m, n, k, 148) == 1
    assert (f[5] > 1) == ((m, k, n) in CUT)   # more than one slot for partials: row blocks are cut


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,k,n", CASES)
def test_against_64_bits(m, k, n, kind):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    w = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    s = (torch.randn(n, k // 32, device="cuda", generator=g).abs() * 0.02).half()
    x = torch.randn(m, k, device="cuda", generator=g).to(kind)
    w64 = L.dequantize(w, s.float(), n, k, 32).double()
    x64 = x.half().double()                      # activations are converted to fp16: exact for these
    ref, mag = x64 @ w64.t(), x64.abs() @ w64.abs().t()
    out = L.quantized_matmul(x, w, s, 32)
    ulp = 2.0 ** -11 if kind == torch.float16 else 2.0 ** -8
    # high-nibble activations are divided by 16 in fp16: below 2^-10 they lose up to 2^-25 * 16 of absolute value each
    slack = 2.0 ** -21 * w64.abs().sum(1)
    assert bool(((out.double() - ref).abs() <= 2.0 ** -12 * mag + slack + ulp * ref.abs()).all())
    again = torch.full_like(out, float("nan"))
    assert torch.equal(L.quantized_matmul(x, w, s, 32, out=again), out)
    assert _lib.lib().lcq_check_device_status(None) == 0, _lib.lib().lcq_last_error()
