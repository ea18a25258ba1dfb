"""The tcgen05 kernel on single SMs and SM pairs at the edges of its tiles and of its dispatch: rows of x
around the tile heights, weight rows around 128 and 256, K that is no whole number of 256-k stages,
tiles cut along K between CTAs.

Bound: each dequantised weight is rounded once to fp16 (relative error <= 2^-11), products are exact in
float32 and summed over K <= 4096 with float32 rounding; |err| <= 2^-11 * sum_k |x w| + 2^-12 * the same
covers both, and the fp16 / bf16 output adds half an ulp of the result (2^-11 / 2^-8 relative).
"""
import ctypes

import numpy as np
import pytest
import torch

import locomp_b200 as L
from locomp_b200 import _lib
from oracle import qmm_oracle as O


def test_plan_covers_every_stage_once():
    lib, f = _lib.lib(), (ctypes.c_int * 8)()
    for m in (1, 17, 32, 33, 64, 100, 192, 193, 256, 512, 1000, 2048, 8192):
        for n in (1, 100, 256, 257, 1024, 4096, 14336, 28672):
            for k in (64, 256, 320, 576, 4096, 14336):
                for sms in (148, 132, 7, 1):
                    assert lib.lcq_gemm_tc_plan_check(m, n, k, sms, f) == 0, (m, n, k, sms, lib.lcq_last_error())
    assert lib.lcq_gemm_tc_plan_check(64, 100, 96, 148, f) == _lib.ERR_UNSUPPORTED


@pytest.mark.parametrize("m,n,k", [(293, 14066, 5568), (379, 19152, 9024), (1042, 16637, 6976), (90, 9000, 2048), (700, 6000, 4096)])
def test_pairs_multiply_rows_in_multiples_of_32(m, n, k):
    """A pair's MMA takes N in steps of 32, a single SM's in steps of 16: whole tiles and the pieces of the last ones."""
    f = (ctypes.c_int * 8)()
    assert _lib.lib().lcq_gemm_tc_plan_check(m, n, k, 148, f) == 0
    bm, cg, tail = f[1], f[5], f[7]
    assert bm % (16 * cg) == 0 and bm % tail == 0 and (bm // tail) % (16 * cg) == 0


CASES = [(17, 1, 64), (17, 257, 320), (31, 255, 256), (32, 256, 576), (33, 513, 1984), (64, 300, 4096), (96, 1000, 832),
         (128, 129, 4096), (160, 640, 1024), (161, 128, 768), (193, 700, 512), (224, 256, 2048), (250, 384, 448), (257, 2000, 1088),
         (40, 30000, 512), (300, 20000, 320), (1000, 4000, 512), (520, 9600, 1024),
         (64, 300, 256), (65, 300, 256), (96, 200, 512), (128, 400, 768), (116, 9850, 1024)]          # one to four stages, both sides of 64 rows


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k", CASES)
def test_against_oracle(m, n, k, kind):
    rng = np.random.default_rng(m * 31 + n + k)
    wp, s = O.make_w4(rng, n, k, 32, np.float16)
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).to(kind)
    wd, sd = torch.from_numpy(wp).cuda(), torch.from_numpy(s).cuda()
    w = O.dequant_int4(wp, s, 32).astype(np.float64)
    x64 = x.double().numpy()
    ref, mag = x64 @ w.T, np.abs(x64) @ np.abs(w).T
    bound = (2.0 ** -11 + 2.0 ** -12) * mag
    y = L.quantized_matmul(x.cuda(), wd, sd, 32, algo="gemm_tc", out_dtype="f32")
    assert np.all(np.abs(y.double().cpu().numpy() - ref) <= bound)
    z = L.quantized_matmul(x.cuda(), wd, sd, 32, algo="gemm_tc")
    ulp = 2.0 ** -11 if kind == torch.float16 else 2.0 ** -8
    assert np.all(np.abs(z.double().cpu().numpy() - ref) <= bound + ulp * np.abs(ref))
    assert torch.equal(L.quantized_matmul(x.cuda(), wd, sd, 32, algo="gemm_tc"), z)     # fixed order of summation
    assert _lib.lib().lcq_check_device_status(None) == 0, _lib.lib().lcq_last_error()


def test_ragged_k_stays_on_exact_sums_where_the_result_would_show_it():
    select, f32, f16, bf16 = _lib.lib().lcq_matmul_select_algo, _lib.F32, _lib.F16, _lib.BF16
    for m, k in ((17, 64), (64, 576), (500, 6080), (1000, 2112)):
        assert select(4, m, 1000, k, 32, f16, f16, f32) == select(4, m, 1000, k, 32, bf16, f16, f32) == _lib.ALGO_GEMV_TC
        assert select(4, m, 1000, k, 32, f16, f16, f16) == select(4, m, 1000, k, 32, bf16, f16, bf16) == _lib.ALGO_GEMM_TC
    assert select(4, 64, 1000, 6208, 32, f16, f16, f16) == _lib.ALGO_GEMV_TC
    assert select(4, 64, 1000, 6208, 32, bf16, f16, bf16) == _lib.ALGO_GEMM_TC
    for out in (f32, f16, bf16):                  # whole weight stages: as ever
        assert select(4, 64, 1000, 8192, 32, f16, f16, out) == _lib.ALGO_GEMM_TC


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k", [(17, 100, 64), (40, 300, 320), (64, 1000, 2624), (130, 1000, 832), (200, 9000, 1088), (293, 14066, 4032)])
def test_ragged_k_has_exact_products(m, n, k, kind):
    """K % 256 != 0: weights as two fp16 terms, so that only the sums round.  Each of the 2 K / 16 MMAs of an output cuts its
    float32 sum short by less than 2^-23 of it: K / 8 * 2^-23 in the 2-norm (one fp16 term alone gives 1.8e-4, from
    K = 12,000 on no more than that).  Scales down to fp16's subnormals.  A 16-bit result adds its own rounding, and is as close as the decode
    kernel's to the third digit; a float32 result is the decode kernel's."""
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    w = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    x = torch.randn(m, k, device="cuda", generator=g).to(kind)
    for size in (0.02, 1e-6):
        s = (torch.randn(n, k // 32, device="cuda", generator=g).abs() * size).half()
        ref = x.double() @ L.dequantize(w, s.float(), n, k, 32).double().t()

        def error(out):
            return float((out.double() - ref).norm() / ref.norm())
        out = L.quantized_matmul(x, w, s, 32, algo="gemm_tc", out_dtype="f32")
        assert error(out) <= k / 8 * 2.0 ** -23
        assert torch.equal(L.quantized_matmul(x, w, s, 32, algo="gemm_tc", out_dtype="f32"), out)
        wide = torch.empty_like(out)
        assert torch.equal(L.quantized_matmul(x, w, s, 32, out=wide), L.quantized_matmul(x, w, s, 32, algo="gemv_tc", out_dtype="f32"))
        assert error(L.quantized_matmul(x, w, s, 32)) <= 1.003 * error(L.quantized_matmul(x, w, s, 32, algo="gemv_tc"))
    assert _lib.lib().lcq_check_device_status(None) == 0, _lib.lib().lcq_last_error()


# Every form of the schedule, each with whole and with partial weight stages: (m, n, k), then what the plan for 148 SMs must say --
# CTAs per MMA, whether tiles are cut along K, CTAs per cluster that share a tile, rows of a piece of a last tile (0: whole).
FORMS = [((18, 74, 1792), (1, False, 4, 0)), ((18, 77, 832), (1, False, 4, 0)), ((19, 85, 1280), (1, False, 5, 0)), ((19, 73, 1344), (1, False, 6, 0)),
         ((23, 5619, 2048), (1, False, 2, 0)), ((18, 2092, 1472), (1, False, 3, 0)),
         ((20, 26048, 2304), (1, True, 1, 0)), ((20, 25453, 1216), (1, True, 1, 0)), ((64, 28672, 8192), (1, True, 1, 0)),
         ((33, 21092, 2560), (1, False, 1, 32)), ((36, 20259, 1088), (1, False, 1, 32)), ((68, 21774, 1792), (1, False, 1, 48)),
         ((69, 19544, 1088), (1, False, 1, 48)), ((114, 23439, 1024), (1, False, 1, 64)),
         ((142, 12161, 768), (2, False, 1, 0)), ((130, 10336, 448), (2, False, 1, 0)),
         ((103, 20209, 2304), (2, False, 1, 32)), ((371, 19953, 384), (2, False, 1, 32)), ((111, 20595, 1152), (2, False, 1, 32)),
         ((113, 24755, 2304), (2, False, 1, 64)), ((229, 21765, 576), (2, False, 1, 64)),
         ((1264, 3821, 1024), (2, False, 1, 96)), ((190, 19169, 640), (2, False, 1, 96)),
         ((4805, 1170, 1280), (2, False, 1, 128)), ((711, 7733, 640), (2, False, 1, 128))]


def _form(m, n, k, sms):
    f = (ctypes.c_int * 8)()
    assert _lib.lib().lcq_gemm_tc_plan_check(m, n, k, sms, f) == 0, _lib.lib().lcq_last_error()
    return f[5], f[3] > 0, f[6], f[1] // f[7] if f[7] > 1 else 0


@pytest.mark.parametrize("problem,form", FORMS)
def test_the_forms_are_those_the_gpu_test_is_for(problem, form):
    assert _form(*problem, 148) == form


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("problem,form", FORMS)
def test_every_form_of_the_schedule(problem, form, kind):
    """All outputs against the dequantised weights in 64 bits, with the bound at the head of this file: an absolute one on
    each output, from sum |x w|."""
    m, n, k = problem
    assert _form(m, n, k, torch.cuda.get_device_properties(0).multi_processor_count) == form
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    w = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    s = (torch.randn(n, k // 32, device="cuda", generator=g).abs() * 0.02).half()
    x = torch.randn(m, k, device="cuda", generator=g).to(kind)
    w64 = L.dequantize(w, s.float(), n, k, 32).double()
    ref, mag = x.double() @ w64.t(), x.double().abs() @ w64.abs().t()
    out = L.quantized_matmul(x, w, s, 32, algo="gemm_tc", out_dtype="f32")
    assert bool(((out.double() - ref).abs() <= (2.0 ** -11 + 2.0 ** -12) * mag).all())
    narrow = L.quantized_matmul(x, w, s, 32, algo="gemm_tc")
    assert torch.equal(narrow, out.to(kind))                                  # the same sums, rounded once
    assert _lib.lib().lcq_check_device_status(None) == 0, _lib.lib().lcq_last_error()
