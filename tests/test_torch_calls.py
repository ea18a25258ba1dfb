"""The native host path for torch CUDA tensors gives what the general path gives, and leaves to the
general path whatever it does not take."""
import copy
import pickle
import sys
import threading

import pytest
import torch

import locomp_b200 as L
from locomp_b200 import _lib


def _linear(m, k, n, bits, group, kind):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    w = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=g) if bits == 4 else \
        torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda", generator=g)
    s = (torch.rand(n, k // group, device="cuda", generator=g) * 0.02).to(torch.float32 if kind == torch.float32 else torch.float16)
    return torch.randn(m, k, device="cuda", generator=g).to(kind), w, s


@pytest.mark.gpu
@pytest.mark.parametrize("m,k,n,bits,group,kind", [(1, 576, 100, 8, 576, torch.float32), (1, 2048, 130, 4, 32, torch.float16),
                                                   (16, 320, 200, 4, 32, torch.bfloat16), (33, 512, 257, 4, 32, torch.float16)])
def test_matmul_same_bits_as_the_general_path(m, k, n, bits, group, kind):
    x, w, s = _linear(m, k, n, bits, group, kind)
    general = L.quantized_matmul(L.DeviceTensor(x), w, s, group, bits=bits)      # a DeviceTensor takes the general path
    native = _lib.calls.matmul(x, w, s, group, bits, None, None)
    assert native is not NotImplemented and torch.equal(native, general)
    out = torch.empty(m, n, dtype=torch.float32, device="cuda")
    assert L.QuantLinear(w, s, group, bits)(x, out=out) is out and torch.equal(out.to(kind), general)
    row = L.quantized_matmul(x[0], w, s, group, bits=bits)
    assert row.shape == (n,)
    side = torch.cuda.Stream()                                                    # a stream that has no workspace yet
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        other = L.quantized_matmul(x, w, s, group, bits=bits)
    side.synchronize()
    assert torch.equal(other, general)
    assert _lib.lib().lcq_check_device_status(None) == 0


@pytest.mark.gpu
def test_the_other_operators_same_bits_as_the_general_path():
    g = torch.Generator(device="cuda").manual_seed(0)
    x, y = (torch.randn(5, 192, device="cuda", generator=g).half() for _ in range(2))
    w = torch.randn(192, device="cuda", generator=g).half()
    D = L.DeviceTensor
    assert torch.equal(L.rms_norm(x, w), L.rms_norm(D(x), w))
    assert torch.equal(L.silu_mul(x, y), L.silu_mul(D(x), y))
    assert torch.equal(L.argmax(x), L.argmax(D(x))) and L.argmax(x[0]).shape == ()
    a, b = x.clone(), x.clone()
    assert torch.equal(L.residual_rms_norm(a, y, w), L.residual_rms_norm(D(b), y, w)) and torch.equal(a, b)
    assert L.add_inplace(a, y) is a and torch.equal(a, L.add_inplace(D(b), y).torch())
    for bits in (4, 8):
        q = L.quantize(x.float(), 32, bits=bits)
        p = L.quantize(D(x.float()), 32, bits=bits)
        assert torch.equal(q.w, p.w) and torch.equal(q.scales, p.scales)
        assert torch.equal(L.dequantize(q.w, q.scales, 5, 192, 32, bits=bits), L.dequantize(D(q.w), q.scales, 5, 192, 32, bits=bits))


@pytest.mark.gpu
def test_errors_are_those_of_the_general_path():
    x, w, s = _linear(2, 256, 64, 4, 32, torch.float16)
    with pytest.raises(ValueError, match="contiguous"):
        L.QuantLinear(w, s)(x.t().contiguous().t())
    with pytest.raises(ValueError, match="K="):
        L.QuantLinear(w, s)(x[:, :128].contiguous())
    with pytest.raises(TypeError, match="uint8"):
        L.quantized_matmul(x, w.to(torch.int8), s)
    with pytest.raises(ValueError, match="workspace_buf"):
        L.quantized_matmul(x, w, s, workspace_buf=torch.zeros(256, dtype=torch.uint8, device="cuda"))


def test_what_is_not_a_cuda_tensor_is_left_to_the_general_path():
    t = torch.zeros(4, 64)
    c = _lib.calls
    assert c.matmul(t, t, t, 32, 4, None, None) is NotImplemented
    assert c.dequantize(t, t, 4, 64, 32, 4, 0) is NotImplemented
    assert c.quantize(t, 32, 4, 0) is NotImplemented
    assert c.rms_norm(t, t, 1e-5, None) is NotImplemented
    assert c.residual_rms_norm(t, t, t, 1e-5, None) is NotImplemented
    assert c.silu_mul(t, t, None) is NotImplemented
    assert c.add_inplace(t, t) is NotImplemented
    assert c.embed_lookup(t, t, t, 1, 64) is NotImplemented
    assert c.argmax(t, None) is NotImplemented
    with pytest.raises(TypeError, match="CUDA"):
        L.quantized_matmul(t, t, t)


def test_a_layer_is_copied_and_pickled_as_any_object():
    layer = L.QuantLinear.__new__(L.QuantLinear)          # (the constructor wants weights on a GPU)
    layer.w, layer.scales, layer.group_size, layer.bits = torch.randint(0, 256, (6, 32), dtype=torch.uint8), torch.rand(6, 2).half(), 32, 4
    layer.out_features, layer.in_features, layer.label = 6, 64, "mine"
    assert set(vars(layer)) == {"w", "scales", "group_size", "bits", "out_features", "in_features", "label"}
    assert copy.copy(layer).w is layer.w
    others = [copy.deepcopy(layer)] + [pickle.loads(pickle.dumps(layer, protocol)) for protocol in range(pickle.HIGHEST_PROTOCOL + 1)]
    for other in others:
        assert type(other) is L.QuantLinear and other.w is not layer.w and vars(other).keys() == vars(layer).keys()
        assert torch.equal(other.w, layer.w) and torch.equal(other.scales, layer.scales) and other.bits == 4 and other.label == "mine"
        with pytest.raises(TypeError, match="CUDA"):
            other(torch.zeros(1, 64).half())
    with pytest.raises(AttributeError, match="scales"):
        del layer.scales
        layer(torch.zeros(1, 64).half())


@pytest.mark.gpu
def test_weights_rebound_during_a_call_outlive_it(monkeypatch):
    """The call on a new stream enters Python for its workspace; what happens there (as in another thread while the GIL is
    released) may drop the layer's last reference to its weights."""
    module = sys.modules["locomp_b200.tensor"]
    x, w, s = _linear(16, 2048, 130, 4, 32, torch.float16)
    want = L.quantized_matmul(x, w, s)
    layer = L.QuantLinear(w, s)
    del w, s

    entered = []

    class Table(dict):
        def get(self, key, default=None):
            entered.append(key)
            layer.w, layer.scales = torch.zeros_like(layer.w), torch.zeros_like(layer.scales)
            return super().get(key, default)
    monkeypatch.setattr(module, "_workspaces", Table(module._workspaces))
    side = torch.cuda.Stream(priority=-1)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        got = layer(x)
        assert torch.equal(layer(x), torch.zeros_like(got))
    side.synchronize()
    assert entered and torch.equal(got, want)


def test_the_scratch_of_a_stream_is_one_threads_at_a_time():
    locked, order = sys.modules["locomp_b200.tensor"].locked_workspace, []

    def other():
        with locked(0, 12345):
            order.append("other")
    thread = threading.Thread(target=other)
    with locked(0, 12345):
        with locked(0, 12345):                             # the same thread may come again
            thread.start()
        with locked(0, 54321):                             # another stream is another lock
            thread.join(0.2)
        order.append("this")
    thread.join(10)
    assert order == ["this", "other"]


@pytest.mark.gpu
def test_threads_that_share_a_stream_do_not_share_scratch():
    """Two threads on the default stream, calls of two launches that pass data through the scratch (bf16, M > 16), sizes that
    make the scratch grow between them; the native and the general path in turn."""
    problems = [_linear(m, k, n, 4, 32, torch.bfloat16) for m, k, n in ((300, 1024, 700), (1100, 4096, 300))]
    want = [L.QuantLinear(w, s)(x, torch.empty(x.shape[0], w.shape[0], dtype=torch.bfloat16, device="cuda")) for x, w, s in problems]
    torch.cuda.synchronize()
    failures = []

    def work(i):
        x, w, s = problems[i]
        layer, operand = L.QuantLinear(w, s), L.DeviceTensor(x)
        got = [layer(x) if r % 3 else L.quantized_matmul(operand, w, s) for r in range(120)]
        torch.cuda.synchronize()
        failures.extend((i, r) for r, g in enumerate(got) if not torch.equal(g, want[i]))
    side = torch.cuda.Stream(priority=-1)                  # no large scratch so far: it grows while the other thread launches

    def on_side(i):
        with torch.cuda.stream(side):
            work(i)
    for form in (work, on_side):
        threads = [threading.Thread(target=form, args=(i,)) for i in (0, 1)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not failures and _lib.lib().lcq_check_device_status(None) == 0
