"""The dequantisers and quantisers at the edges of their fast paths: one octet, a block's octets and one more or less, several blocks, groups that
are no power of two, and every alignment that the entry points take.  Bit for bit the oracle's results, as the operations are exact or
rounded once."""
import ctypes

import numpy as np
import pytest
import torch

import locomp_b200 as L
from locomp_b200 import _lib
from oracle import qmm_oracle as O

pytestmark = pytest.mark.gpu
KINDS = {"f32": (torch.float32, _lib.F32), "f16": (torch.float16, _lib.F16), "bf16": (torch.bfloat16, _lib.BF16)}
SHAPES = [(1, 8, 8), (1, 32, 32), (3, 24, 24), (2, 4096, 32), (1, 4104, 8), (1, 8184, 24), (5, 8192, 64), (257, 576, 32), (129, 8200, 40), (7, 100, 20), (9, 12, 4), (3, 36, 18)]


def _placed(t, offset):
    """The same values at an address `offset` bytes past a multiple of 512."""
    raw = torch.zeros(t.numel() * t.element_size() + 512, dtype=torch.uint8, device="cuda")
    view = raw[offset:offset + t.numel() * t.element_size()].view(t.dtype).view(t.shape)
    view.copy_(t)
    return view


@pytest.mark.parametrize("n,k,g", SHAPES)
@pytest.mark.parametrize("scales", ["f32", "f16"])
@pytest.mark.parametrize("out", ["f32", "f16", "bf16"])
def test_dequantise_at_every_alignment(n, k, g, scales, out):
    rng = np.random.default_rng(n * k + g)
    for bits, make, dequantise, call in ((4, O.make_w4, O.dequant_int4, _lib.lib().lcq_dequant_int4), (8, O.make_w8, O.dequant_int8, _lib.lib().lcq_dequant_int8)):
        w, s = make(rng, n, k, g, np.float32 if scales == "f32" else np.float16)
        want = O.round_to(dequantise(w, s, g), out).astype(np.float32)
        ws, ss = torch.from_numpy(w).cuda(), torch.from_numpy(s).cuda()
        for w_off, out_off in ((0, 0), (0, 16), (8, 32), (4, 0), (4, 8), (1, 4), (0, 48)):
            placed = _placed(ws, w_off)
            dst = _placed(torch.full((n, k), 77.0, device="cuda").to(KINDS[out][0]), out_off)
            rc = call(ctypes.c_void_p(placed.data_ptr()), ctypes.c_void_p(ss.data_ptr()), ctypes.c_void_p(dst.data_ptr()), n, k, g,
                      KINDS[scales][1], KINDS[out][1], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert rc == 0, _lib.lib().lcq_last_error()
            assert np.array_equal(dst.float().cpu().numpy().view(np.uint32), want.view(np.uint32)), (bits, w_off, out_off)


@pytest.mark.parametrize("n,k,g", [(1, 8, 8), (1, 32, 32), (3, 2048, 16), (1, 4104, 8), (2, 4096, 256), (257, 576, 64), (9, 8192, 128), (1025, 8, 8), (3, 24, 24)])
@pytest.mark.parametrize("kind", ["f32", "f16", "bf16"])
def test_quantise_at_every_alignment(n, k, g, kind):
    gen = torch.Generator(device="cuda").manual_seed(n + k)
    w = (torch.randn(n, k, device="cuda", generator=gen) * 0.1).to(KINDS[kind][0])
    for bits, quantise in ((4, O.quantize_int4), (8, O.quantize_int8)):
        q_ref, s_ref = quantise(w.float().cpu().numpy(), g)
        for offset in (0, 16, 32, 4):
            q = L.quantize(_placed(w, offset), g, bits=bits)
            assert np.array_equal(q.w.cpu().numpy(), q_ref), (bits, offset)
            assert np.array_equal(q.scales.cpu().numpy().view(np.uint32), s_ref.view(np.uint32))


@pytest.mark.parametrize("offset", [0, 16])
@pytest.mark.parametrize("bits", [4, 8])
def test_quantise_a_large_weight(bits, offset):
    """Float32 weights have one octet a thread up to 32 Mi weights and four beyond: a weight just beyond, whole and in two parts."""
    n, k, g = 4099, 8200, 8
    assert n * k > 1 << 25 and n * k // 8 % 1024
    w = _placed(torch.randn(n, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(6)), offset)
    whole, parts = L.quantize(w, g, bits=bits), [L.quantize(part, g, bits=bits) for part in (w[:1000], w[1000:])]
    assert torch.equal(whole.w, torch.cat([q.w for q in parts])) and torch.equal(whole.scales, torch.cat([q.scales for q in parts]))


def _call(name, *args):
    _lib.check(getattr(_lib.lib(), name)(*[ctypes.c_void_p(a.data_ptr()) if isinstance(a, torch.Tensor) else a for a in args],
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))


def _unsynchronised_is_synchronised(rounds, step):
    """step(i) launches a chain of kernels and returns its outputs, in buffers of their own; bit for bit the same with a
    synchronisation behind every kernel (step calls what it is given between them)."""
    torch.cuda.synchronize()
    together = [step(i, lambda: None) for i in range(rounds)]
    torch.cuda.synchronize()
    for i in range(rounds):
        apart = step(i, torch.cuda.synchronize)
        torch.cuda.synchronize()
        for a, b in zip(together[i], apart):
            assert torch.equal(a, b), i


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("kind", ["f32", "f16"])
@pytest.mark.parametrize("before", ["rms_norm", "silu_mul", "add_inplace", "linear"])
def test_input_of_a_kernel_that_lets_its_successor_start(before, kind, bits):
    """The blocks of these kernels are there while such a predecessor still writes what they read, into one buffer whose values change every time."""
    n, k, rounds, dtype = 1500, 2048, 8, KINDS[kind][0]
    gen = torch.Generator(device="cuda").manual_seed(3)
    a = [torch.randn(n, k, device="cuda", generator=gen).to(dtype) for _ in range(rounds)]
    weight = torch.randn(k, device="cuda", generator=gen).to(dtype)
    buffer = torch.zeros(n, k, device="cuda", dtype=dtype)
    layer = L.QuantLinear(torch.randint(0, 256, (k, k // 2), dtype=torch.uint8, device="cuda", generator=gen),
                          torch.rand(k, k // 32, device="cuda", generator=gen).to(dtype) * 0.01, 32, 4)

    def step(i, between):
        if before == "rms_norm":
            L.rms_norm(a[i], weight, out=buffer)
        elif before == "silu_mul":
            L.silu_mul(a[i], a[i - 1], out=buffer)
        elif before == "add_inplace":
            L.add_inplace(buffer.zero_(), a[i])
        else:
            layer(a[i], out=buffer)
        between()
        q = torch.empty(n, k * bits // 8, dtype=torch.uint8, device="cuda")
        s = torch.empty(n, k // 32, device="cuda")
        _call(f"lcq_quantize_int{bits}", buffer, q, s, n, k, 32, KINDS[kind][1], 0)
        between()
        back = torch.empty(n, k, device="cuda")
        _call(f"lcq_dequant_int{bits}", q, s, back, n, k, 32, _lib.F32, _lib.F32)
        return q, s, back
    _unsynchronised_is_synchronised(rounds, step)


def test_scales_from_a_linear_layer():
    """Dequantise behind a kernel that lets it start early and writes its scales."""
    n, k, rounds = 4096, 4096, 8
    gen = torch.Generator(device="cuda").manual_seed(4)
    codes = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen)
    layer = L.QuantLinear(torch.randint(0, 256, (k // 32, 512), dtype=torch.uint8, device="cuda", generator=gen),
                          torch.rand(k // 32, 32, device="cuda", generator=gen).half() * 0.01, 32, 4)
    x = [torch.randn(n, 1024, device="cuda", generator=gen).half() for _ in range(rounds)]
    scales = torch.zeros(n, k // 32, dtype=torch.float16, device="cuda")

    def step(i, between):
        layer(x[i], out=scales)
        between()
        back = torch.empty(n, k, device="cuda", dtype=torch.float16)
        _call("lcq_dequant_int4", codes, scales, back, n, k, 32, _lib.F16, _lib.F16)
        return back,
    _unsynchronised_is_synchronised(rounds, step)


def test_quantise_into_weights_that_a_linear_layer_still_reads():
    n, k, rounds = 16000, 4096, 6
    gen = torch.Generator(device="cuda").manual_seed(5)
    w = [torch.randn(n, k, device="cuda", generator=gen) for _ in range(2)]
    layer = L.QuantLinear(torch.zeros(n, k // 2, dtype=torch.uint8, device="cuda"), torch.zeros(n, k // 32, device="cuda"), 32, 4)
    x = torch.randn(4, k, device="cuda", generator=gen)

    def step(i, between):
        _call("lcq_quantize_int4", w[i % 2], layer.w, layer.scales, n, k, 32, _lib.F32, 0)
        torch.cuda.synchronize()                               # (the weights of a linear layer are to be complete)
        y = layer(x)
        between()
        _call("lcq_quantize_int4", w[1 - i % 2], layer.w, layer.scales, n, k, 32, _lib.F32, 0)
        torch.cuda.synchronize()
        return y,
    _unsynchronised_is_synchronised(rounds, step)


@pytest.mark.parametrize("written", ["weights", "scales"])
def test_a_linear_layer_does_not_start_while_its_weights_are_written(written):
    """Kernels of linear layers fetch weights and scales before they wait for the kernel in front of them, which is why a caller has to synchronise between
    writing weights and the first call.  The quantisers and dequantisers do their part: they do not let a linear layer directly behind them
    start early, so that it does not fetch what was there before.  Other weights every time, in the same buffers."""
    n, k, rounds = 8192, 4096, 12
    gen = torch.Generator(device="cuda").manual_seed(7)
    if written == "weights":
        source = [torch.randn(n, k, device="cuda", generator=gen) for _ in range(4)]
        layer = L.QuantLinear(torch.zeros(n, k // 2, dtype=torch.uint8, device="cuda"), torch.zeros(n, k // 32, device="cuda"), 32, 4)
        x = torch.randn(1, k, device="cuda", generator=gen)
    else:
        source = [torch.randint(0, 256, (n, k // 32), dtype=torch.uint8, device="cuda", generator=gen) for _ in range(4)]
        unit = torch.rand(n, 1, device="cuda", generator=gen) * 0.01
        layer = L.QuantLinear(torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen),
                              torch.zeros(n, k // 32, dtype=torch.float16, device="cuda"), 32, 4)
        x = torch.randn(1, k, device="cuda", generator=gen).half()

    def step(i, between):
        if written == "weights":
            _call("lcq_quantize_int4", source[i % 4], layer.w, layer.scales, n, k, 32, _lib.F32, 0)
        else:
            _call("lcq_dequant_int8", source[i % 4], unit, layer.scales, n, k // 32, k // 32, _lib.F32, _lib.F16)
        between()
        return layer(x),
    _unsynchronised_is_synchronised(rounds, step)
