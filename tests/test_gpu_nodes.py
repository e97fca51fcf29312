"""The layers' native autograd nodes against the Function classes: the same bits, and the same manners in autograd."""
import pytest
import torch

from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.fixture
def functions(monkeypatch):
    """switches the layers to their Function classes"""
    from flashdp4review_b200.layers import layernorm, linear, transformers_conv1d

    def switch(on):
        for m in (linear, transformers_conv1d, layernorm):
            if on:
                monkeypatch.setattr(m, "native_nodes", lambda t: None)
            else:
                monkeypatch.undo()
    return switch


def _layer(kind, n_in, n_out, dtype, bias=True, noise=1.0):
    import flashdp4review_b200 as fdp
    torch.manual_seed(1)
    if kind == "linear":
        m = fdp.DPLinear(n_in, n_out, bias=True if bias else None, C=0.1, noise_multiplier=noise)
    elif kind == "conv1d":
        m = fdp.DPConv1D(n_out, n_in, C=0.1, noise_multiplier=noise)
    else:
        m = fdp.DPLayerNorm(n_in, use_fused=False, bias=True if bias else None, C=0.1, noise_multiplier=noise)
    m = m.to(device=dev(), dtype=dtype)
    m._dp_param_ids = [5, 6]
    return m


def _pass(m, x, g, autocast, dims):
    m._dp_step = 0
    m.zero_grad(set_to_none=True)
    x = x.clone().requires_grad_(dims != "no_dx")
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=autocast):
        y = m(x)
    y.backward(g.to(y.dtype))
    return [y.detach(), x.grad] + [p.grad for p in m.parameters()]


# library products and torch ones (few rows, odd widths), every rank of input, autocast, no bias, frozen parts
@pytest.mark.parametrize("kind,shape,n_in,n_out,dtype,autocast,bias,frozen", [
    ("linear", (4, 64), 128, 192, torch.float32, False, True, ""), ("linear", (3, 50), 72, 40, torch.float32, False, False, ""),
    ("linear", (200,), 128, 136, torch.bfloat16, False, True, ""), ("linear", (2, 3, 40), 128, 128, torch.float16, False, True, ""),
    ("linear", (4, 64), 128, 192, torch.float32, True, True, ""), ("linear", (2, 20), 65, 33, torch.float32, True, True, ""),
    ("linear", (2, 20), 65, 33, torch.bfloat16, False, True, "x"), ("linear", (4, 64), 128, 192, torch.float32, False, True, "weight"),
    ("linear", (4, 64), 128, 192, torch.float32, False, True, "bias"),
    ("conv1d", (4, 64), 128, 192, torch.float32, False, True, ""), ("conv1d", (2, 20), 33, 65, torch.float32, True, True, ""),
    ("conv1d", (4, 64), 128, 192, torch.bfloat16, False, True, "weight"),
    ("layernorm", (4, 30), 128, 128, torch.float32, False, True, ""), ("layernorm", (7,), 100, 100, torch.bfloat16, False, False, ""),
    ("layernorm", (2, 3, 5), 128, 128, torch.float16, False, True, "weight"), ("layernorm", (4, 30), 128, 128, torch.float32, False, True, "x")])
def test_nodes_give_the_functions_bits(functions, kind, shape, n_in, n_out, dtype, autocast, bias, frozen):
    m = _layer(kind, n_in, n_out, dtype, bias)
    gen = torch.Generator(device=dev()).manual_seed(3)
    x = torch.randn(*shape, n_in, device=dev(), generator=gen).to(dtype)
    g = torch.randn(*shape, n_out if kind != "layernorm" else n_in, device=dev(), generator=gen)
    for name, p in m.named_parameters():
        p.requires_grad_(name != frozen)
    dims = "no_dx" if frozen == "x" else ""
    got = _pass(m, x, g, autocast, dims)
    functions(True)
    want = _pass(m, x, g, autocast, dims)
    functions(False)
    assert m._dp_step == 1
    for a, b in zip(got, want):
        assert (a is None) == (b is None) and (a is None or (a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)))


def test_nodes_in_autograd(functions):
    """Saved-tensor hooks see what a node saves, an in-place change of it is an error, a trace records the Function, a call
    for one gradient alone computes that one, an unsupported dtype and a status raise what the operators raise."""
    m = _layer("linear", 128, 192, torch.float32)
    x = torch.randn(4, 64, 128, device=dev(), requires_grad=True)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t.cpu(), lambda t: t.to(dev())):
        y = m(x)
        y.sum().backward()
    assert len(packed) >= 2
    dx, = torch.autograd.grad(m(x).sum(), x)
    assert dx.shape == x.shape and m.weight.grad is not None
    y = m(x * 1.0)
    with torch.no_grad():
        m.weight.mul_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()
    n = _layer("layernorm", 128, 128, torch.float32)
    with pytest.raises(KeyError):
        n(x.double())
    with pytest.raises(KeyError):
        _layer("linear", 128, 192, torch.float64)(x.double()).sum().backward()
    with pytest.raises(RuntimeError):
        torch.func.vmap(m)(x)
    traced = torch.jit.trace(m, (x,), check_trace=False)
    z = torch.randn_like(x)
    assert torch.equal(traced(z), m(z))


def test_nodes_write_into_gradient_buckets(functions):
    """a weight gradient goes where the reducer asks for it"""
    from flashdp4review_b200.layers import _common
    m = _layer("linear", 128, 192, torch.float32, noise=0.0)
    x = torch.randn(4, 64, 128, device=dev())
    slot, done = torch.zeros(192, 128, device=dev()), []

    class Reducer:
        def claim_direct(self, p):
            return slot if p is m.weight else None

        def direct_written(self, p):
            done.append(p)
    before = _common.direct_reducer
    _common.direct_reducer = lambda p: Reducer()
    try:
        m(x).sum().backward()
    finally:
        _common.direct_reducer = before
    assert m.weight.grad is None and len(done) == 1 and done[0] is m.weight
    m(x).sum().backward()
    assert torch.equal(slot, m.weight.grad)


@pytest.mark.parametrize("kind", ["linear", "conv1d"])
def test_nodes_take_and_refuse_what_the_functions_do(functions, kind):
    """A frozen layer in a dtype of torch's alone returns its input gradient; a float64 input under autocast is refused in
    backward, not answered in fp16; a frozen layer takes an empty batch, for which no noise could be formed.  The same
    through the Function classes."""
    for on in (False, True):
        functions(on)
        m = _layer(kind, 128, 192, torch.float64)
        for p in m.parameters():
            p.requires_grad_(False)
        x = torch.randn(4, 64, 128, device=dev(), dtype=torch.float64, requires_grad=True)
        m(x).sum().backward()
        w = m.weight if kind == "linear" else m.weight.t()
        assert torch.allclose(x.grad, w.sum(0).expand_as(x))
        for width in (192, 33):              # a product of the library's, one of torch's
            m = _layer(kind, 128, width, torch.float32)
            y = None
            with torch.autocast("cuda", dtype=torch.bfloat16):
                y = m(x)
            with pytest.raises(KeyError):
                y.float().sum().backward()
        m = _layer(kind, 128, 192, torch.float32)
        for p in m.parameters():
            p.requires_grad_(False)
        e = torch.zeros(0, 64, 128, device=dev(), requires_grad=True)
        m(e).sum().backward()
        assert e.grad.shape == e.shape and m._dp_step == 1


def test_a_forward_leaves_the_interpreter_to_other_threads(tmp_path):
    """While one thread is in the library (here an entry point that only sleeps and reports an error) another goes on."""
    import ctypes
    import shutil
    import subprocess
    import threading
    import time
    from flashdp4review_b200 import _lib
    if shutil.which("gcc") is None:
        pytest.skip("no C compiler")
    src = tmp_path / "slow.c"
    src.write_text("#include <unistd.h>\nint slow(void) { usleep(400000); return -1; }\n")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "slow.so"), str(src)], check=True)
    slow = ctypes.cast(ctypes.CDLL(str(tmp_path / "slow.so")).slow, ctypes.c_void_p).value
    lib, host = _lib.load(), _lib.host()
    real = {n: ctypes.cast(getattr(lib, n), ctypes.c_void_p).value for n in _lib.SIGNATURES}
    x = torch.randn(4, 64, 128, device=dev())
    for kind, entry in (("linear", "fdp_linear_fwd"), ("layernorm", "fdp_layernorm_fwd")):
        m = _layer(kind, 128, 192 if kind == "linear" else 128, torch.float32)
        m(x)
        gaps, stop = [0.0], threading.Event()

        def tick():
            last = time.perf_counter()
            while not stop.is_set():
                time.sleep(0.002)
                now = time.perf_counter()
                gaps.append(now - last)
                last = now
        t = threading.Thread(target=tick)
        host.bind({**real, entry: slow})
        try:
            t.start()
            with pytest.raises(ValueError):
                m(x)
        finally:
            stop.set()
            t.join()
            host.bind(real)
        assert max(gaps) < 0.3, (kind, max(gaps))


@pytest.mark.parametrize("kind", ["linear", "conv1d", "layernorm"])
def test_a_node_does_not_keep_its_layer_alive(kind):
    """A layer that keeps its own output goes when the program lets go of it; a graph outlives its layer, with the
    values and the noise that the layer would have given it."""
    import gc
    import weakref
    x = torch.randn(4, 64, 128, device=dev())
    m = _layer(kind, 128, 192 if kind != "layernorm" else 128, torch.float32)
    m.register_forward_hook(lambda mod, i, o: setattr(mod, "act", o))
    m(x)
    gone = weakref.ref(m)
    del m
    gc.collect()
    assert gone() is None

    grads = []
    for keep in (True, False):
        m = _layer(kind, 128, 192 if kind != "layernorm" else 128, torch.float32)
        m._dp_step = 4
        params = list(m.parameters())
        ys = [m(x), m(2.0 * x)]
        if not keep:
            del m
            gc.collect()
        for y in ys:
            y.sum().backward()
        grads.append([p.grad for p in params])
        if keep:
            assert m._dp_step == 6
            m.C = 0.01                # read when a backward runs, as the Function classes do
            a = torch.autograd.grad(m(x).sum(), params)
            m._dp_step -= 1
            m.C = 0.1
            y = m(x)
            m.C = 0.01
            b = torch.autograd.grad(y.sum(), params)
            assert all(torch.equal(s, t) for s, t in zip(a, b))
    assert all(torch.equal(s, t) for s, t in zip(*grads))
