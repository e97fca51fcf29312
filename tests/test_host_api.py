"""CPU-side checks: the shared library loads and exports the whole C ABI, and the wrap API keeps
the reference's selection rules and errors (flashdp/api/wrap_model.py)."""
import os
import re

import pytest
import torch
import torch.nn as nn

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_exports_every_declared_symbol():
    from flashdp4review_b200 import _lib
    lib = _lib.load()
    header = open(os.path.join(ROOT, "include", "fdp_b200.h")).read()
    declared = set(re.findall(r"\b(fdp_[a-z0-9_]+)\s*\(", header))
    assert declared, "no declarations found"
    for name in declared:
        assert hasattr(lib, name), f"{name} declared in include/fdp_b200.h but not exported"
    assert declared == set(_lib.SIGNATURES), declared ^ set(_lib.SIGNATURES)
    assert lib.fdp_abi_version() == _lib.ABI_VERSION
    assert lib.fdp_status_string(0) == b"ok"
    assert b"workspace" in lib.fdp_status_string(_lib.FDP_ERR_WORKSPACE)
    # pure host-side queries work without a device
    assert lib.fdp_linear_wgrad_workspace_bytes(4, 128, 768, 768, _lib.FDP_F32, 0) > 0
    assert lib.fdp_linear_wgrad_workspace_bytes(0, 128, 768, 768, _lib.FDP_F32, 0) == 0
    assert lib.fdp_bias_grad_workspace_bytes(4, 128, 768, _lib.FDP_BF16) > 0
    assert lib.fdp_layernorm_bwd_workspace_bytes(16, 1024, 1024) > 0


def test_no_cpu_fallback():
    from flashdp4review_b200.core import ops
    with pytest.raises(RuntimeError, match="no CPU path"):
        ops.dp_linear_weight_grad(torch.zeros(1, 2, 8), torch.zeros(1, 2, 8), 1.0, 1.0)
    with pytest.raises(RuntimeError, match="no CPU path"):
        ops.dp_bias_grad(torch.zeros(1, 2, 8), 1.0, 1.0)


def _model():
    return nn.Sequential(nn.Linear(8, 8), nn.LayerNorm(8),
                         nn.Sequential(nn.Linear(8, 4, bias=False), nn.ReLU()), nn.Linear(4, 2))


def test_wrap_argument_errors():
    from flashdp4review_b200 import wrap_with_flashdp_layers
    with pytest.raises(ValueError):
        wrap_with_flashdp_layers(_model())
    with pytest.raises(ValueError):
        wrap_with_flashdp_layers(_model(), target_modules=[])
    with pytest.raises(ValueError):
        wrap_with_flashdp_layers(_model(), target_layers=["0"])          # target_layers alone is rejected
    with pytest.raises(ValueError):
        wrap_with_flashdp_layers(_model(), target_modules=[nn.Conv2d])


def test_wrap_selection_rules():
    import flashdp4review_b200 as fdp
    m = fdp.wrap_with_flashdp_layers(_model(), target_modules=[nn.Linear, nn.LayerNorm], skip_layers=["3"],
                                     C=0.3, noise_multiplier=0.7, clamp_value=0.9, feedback=False)
    assert isinstance(m[0], fdp.DPLinear) and isinstance(m[1], fdp.DPLayerNorm)
    assert isinstance(m[2][0], fdp.DPLinear) and m[2][0].bias is None
    assert type(m[3]) is nn.Linear
    assert (m[0].C, m[0].noise_multiplier, m[0].clamp_value) == (0.3, 0.7, 0.9)
    # skipping a container does not skip its children (exact-name match only)
    m = fdp.wrap_with_flashdp_layers(_model(), target_modules=[nn.Linear], skip_layers=["2"], feedback=False)
    assert isinstance(m[2][0], fdp.DPLinear)
    # target_layers restricts the candidates
    m = fdp.wrap_with_flashdp_layers(_model(), target_modules=[nn.Linear], target_layers=["0"], feedback=False)
    assert isinstance(m[0], fdp.DPLinear) and type(m[3]) is nn.Linear


def test_wrap_keeps_weights_dtype_mode_and_ties():
    import flashdp4review_b200 as fdp

    class Tied(nn.Module):
        def __init__(self):
            super().__init__()
            self.emb = nn.Embedding(10, 8)
            self.body = nn.Linear(8, 8)
            self.lm_head = nn.Linear(8, 10, bias=False)
            self.lm_head.weight = self.emb.weight
    src = Tied().to(torch.bfloat16).eval()
    ref_w = src.body.weight.detach().clone()
    m = fdp.wrap_with_flashdp_layers(src, target_modules=[nn.Linear], skip_layers=["lm_head"], feedback=False)
    assert torch.equal(m.body.weight.detach(), ref_w)
    assert m.body.weight.dtype == torch.bfloat16 and not m.body.training
    assert m.lm_head.weight is m.emb.weight
    assert set(m.state_dict()) == set(Tied().state_dict())            # parameter names round-trip


def test_conv1d_twin_and_constructor_attributes():
    import flashdp4review_b200 as fdp
    from flashdp4review_b200.layers import Conv1D
    m = nn.Sequential(Conv1D(24, 8))
    fdp.wrap_with_flashdp_layers(m, target_modules=[Conv1D], feedback=False)
    assert isinstance(m[0], fdp.DPConv1D) and m[0].weight.shape == (8, 24) and m[0].nf == 24
    lin = fdp.DPLinear(4, 6, C=2.0, clamp_value=0.5, noise_multiplier=0.1, auto_tune=False)
    assert lin.dp and lin.runtime_tuner.enable is False and lin.weight.requires_dp
    ln = fdp.DPLayerNorm(6, use_fused=False, bias=None)
    assert ln.bias is None and ln.use_fused is False


def test_workspace_queries_are_pure_host_functions():
    """The *_workspace_bytes queries run without a GPU, reject nonsense with 0 and grow with the
    problem; every plan the launch would pick (tensor-core, short-sequence, generic) fits them."""
    from flashdp4review_b200 import _lib
    lib = _lib.load()
    q = lib.fdp_linear_wgrad_workspace_bytes
    assert q(0, 128, 256, 256, _lib.FDP_BF16, 0) == 0 and q(4, 128, 256, 256, 7, 0) == 0
    sizes = [q(B, T, 256, 384, dt, 0) for dt in (_lib.FDP_F32, _lib.FDP_BF16)
             for (B, T) in ((2, 7), (512, 1), (4, 128), (32, 1024))]
    assert all(s > 0 and s % 256 == 0 for s in sizes)
    assert q(64, 1024, 256, 384, _lib.FDP_BF16, 0) >= q(32, 1024, 256, 384, _lib.FDP_BF16, 0)
    b = lib.fdp_bias_grad_workspace_bytes
    assert b(0, 1, 1, _lib.FDP_F32) == 0
    assert 0 < b(4, 128, 768, _lib.FDP_F32) <= b(8, 128, 768, _lib.FDP_F32) <= b(8, 4096, 768, _lib.FDP_F32)
    ln = lib.fdp_layernorm_bwd_workspace_bytes
    assert ln(0, 1, 1) == 0
    assert 0 < ln(4, 9, 40) <= ln(16, 1024, 1024) <= ln(32, 1024, 4096)
    assert lib.fdp_linear_dgrad_workspace_bytes(4096, 256, 384, _lib.FDP_BF16) >= 0
    # fp32 on the tensor cores: the flag adds room for the bf16 halves of the operands where the shape
    # qualifies (64-aligned contracted dimension, at least 128 of everything) and nothing elsewhere
    t3 = _lib.FDP_F32 | _lib.FDP_FP32_TENSOR
    d = lib.fdp_linear_dgrad_workspace_bytes
    rows, n_in, n_out = 8192, 1024, 3072
    assert d(rows, n_in, n_out, _lib.FDP_F32) == 256
    assert d(rows, n_in, n_out, t3) >= 256 + 4 * (rows * n_out + n_out * n_in)
    assert d(rows, n_in, 1000, t3) == 256 and d(64, n_in, n_out, t3) == 256     # K % 64, too few rows
    w = lib.fdp_linear_wgrad_workspace_bytes
    plain, flagged = w(8, 1024, 4096, 4096, _lib.FDP_F32, 0), w(8, 1024, 4096, 4096, _lib.FDP_F32, _lib.FDP_FP32_TENSOR)
    assert flagged >= plain + 4 * 8 * 1024 * (4096 + 4096) - (1 << 20)
    assert w(8, 1000, 4096, 4096, _lib.FDP_F32, _lib.FDP_FP32_TENSOR) == w(8, 1000, 4096, 4096, _lib.FDP_F32, 0)
    assert w(8, 1024, 4096, 4096, _lib.FDP_BF16, _lib.FDP_FP32_TENSOR) == w(8, 1024, 4096, 4096, _lib.FDP_BF16, 0)


def test_gram_work_units_cover_the_block_triangle_once(tmp_path):
    """The Gram norm pass deals units of (t-block, two s-blocks); compiled for the host, the
    enumeration must cover every unordered block pair exactly once, with at most one single-block
    unit per sample, for every block count."""
    import shutil
    import subprocess
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    hdr = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                       "flashdp4review_b200", "csrc", "fdp_gram_units.h")
    src = tmp_path / "units.cpp"
    src.write_text('#include <cstdio>\n#include <set>\n#include <utility>\n#include "%s"\n' % hdr + r'''
int main() {
  for (int nb = 1; nb <= 160; ++nb) {
    std::set<std::pair<int, int>> seen;
    const int units = fdp::gram_units(nb);
    int singles = 0;
    for (int u = 0; u < units; ++u) {
      int i, j1, j2;
      fdp::gram_decode(nb, u, i, j1, j2);
      if (i < 0 || i >= nb || j1 < 0 || j1 >= nb || j2 >= nb) { std::printf("range nb=%d u=%d\n", nb, u); return 1; }
      if (j2 < 0) ++singles;
      const int js[2] = {j1, j2};
      for (int k = 0; k < 2; ++k) {
        if (js[k] < 0) continue;
        const std::pair<int, int> key(i < js[k] ? i : js[k], i < js[k] ? js[k] : i);
        if (!seen.insert(key).second) { std::printf("twice nb=%d (%d,%d)\n", nb, key.first, key.second); return 1; }
      }
    }
    if (static_cast<int>(seen.size()) != nb * (nb + 1) / 2) { std::printf("missing nb=%d\n", nb); return 1; }
    if (singles > 1 || units != (nb * (nb + 1) / 2 + 1) / 2) { std::printf("count nb=%d\n", nb); return 1; }
  }
  std::printf("ok\n");
  return 0;
}
''')
    exe = tmp_path / "units"
    subprocess.run([gxx, "-O1", "-std=c++17", "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout


def test_forward_and_input_gradient_gemm_selection():
    """`set_input_grad_impl`: "library" never uses the package's GEMMs, "auto" (default) only where a
    tensor-core kernel takes the shape, "native" also the generic 16-bit kernels; fp32 only in fp32 mode
    "tensor" and with the contracted dimension a multiple of 64."""
    import torch
    from flashdp4review_b200 import runtime
    from flashdp4review_b200.core import ops
    before, before32 = runtime.input_grad_impl(), runtime.fp32_mode()
    try:
        assert before == "auto" and before32 == "tensor"
        bf, f32 = torch.bfloat16, torch.float32
        cases = {  # (dtype, rows, K, N): (library, auto, native)
            (bf, 8192, 1024, 3072): (False, True, True),
            (bf, 8192, 100, 3072): (False, False, True),      # K not a multiple of 8: generic kernel
            (bf, 64, 1024, 1024): (False, False, True),       # too few rows for a tile
            (f32, 8192, 1024, 3072): (False, True, True),
            (f32, 8192, 1000, 3072): (False, False, False),   # K not a multiple of 64: cuBLAS
            (f32, 96, 1024, 1024): (False, False, False),
            (torch.float64, 8192, 1024, 1024): (False, False, False),
        }
        for i, impl in enumerate(("library", "auto", "native")):
            runtime.set_input_grad_impl(impl)
            for (dt, rows, K, N), want in cases.items():
                assert ops.native_product_ok(dt, rows, K, N) == want[i], (impl, dt, rows, K, N)
        runtime.set_input_grad_impl("auto")
        runtime.set_fp32_mode("exact")
        assert not ops.native_product_ok(f32, 8192, 1024, 3072)
        with pytest.raises(ValueError):
            runtime.set_input_grad_impl("cublas")
    finally:
        runtime.set_input_grad_impl(before)
        runtime.set_fp32_mode(before32)


@pytest.fixture
def no_launch(monkeypatch):
    """The operator layer on CPU tensors, with a call layer that fails the test when it is entered."""
    from flashdp4review_b200 import _lib
    from flashdp4review_b200.core import ops

    class Launched(Exception):
        pass

    class Host:
        def __getattr__(self, name):
            def call(*args):
                raise Launched(name, args)
            return call
    monkeypatch.setattr(_lib, "host", Host)
    monkeypatch.setattr(ops, "_require_cuda", lambda *tensors: None)
    return ops, Launched


@pytest.mark.parametrize("layout", ["out_in", "in_out"])
def test_operands_that_do_not_fit_are_refused_before_a_launch(monkeypatch, layout):
    """The kernels take the weight as a bare pointer: another shape than (out, in) or (in, out) would be misread, a
    smaller one read past its end.  (On CPU tensors: the call layer looks before it touches a device.)"""
    from flashdp4review_b200.core import ops
    monkeypatch.setattr(ops, "_require_cuda", lambda *tensors: None)
    X, G = torch.zeros(2, 3, 16), torch.zeros(2, 3, 8)
    right = (8, 16) if layout == "out_in" else (16, 8)
    shapes = [right[::-1], (right[0], right[1] + 1), (right[0] + 1, right[1]), (right[0] - 1, right[1]), (4, 4), right + (1,), (128,)]
    refused = "weight does not fit"
    for shape in shapes:
        with pytest.raises(RuntimeError, match=refused):
            ops.dp_linear_backward(X, G, torch.zeros(shape), 1.0, 1.0, layout=layout)
        if len(shape) != 2 or shape[0 if layout == "out_in" else 1] != 8:
            with pytest.raises(RuntimeError, match=refused):
                ops.linear_input_grad(G, torch.zeros(shape), layout)
        if len(shape) != 2 or shape[1 if layout == "out_in" else 0] != 16:
            with pytest.raises(RuntimeError, match=refused):
                ops.linear_forward(X, torch.zeros(shape), None, layout)
    W = torch.zeros(right)
    monkeypatch.setattr(ops, "_aligned", lambda t: t)          # (a meta tensor has no address to look at)
    for call in (lambda: ops.dp_linear_backward(X, G, W.to("meta"), 1.0, 1.0, layout=layout),
                 lambda: ops.linear_input_grad(G, W.to("meta"), layout), lambda: ops.linear_forward(X, W.to("meta"), None, layout)):
        with pytest.raises(RuntimeError, match="weight is on another device"):
            call()
    with pytest.raises(RuntimeError, match="input is on another device"):
        ops.dp_linear_backward(X.to("meta"), G, W, 1.0, 1.0, layout=layout)
    for bias in (torch.zeros(7), torch.zeros(8).to("meta")):
        with pytest.raises(RuntimeError, match="bias does not fit"):
            ops.linear_forward(X, W, bias, layout)


def test_layernorm_operands_that_do_not_fit_are_refused_before_a_launch(monkeypatch):
    """Parameters, statistics and upstream gradient of a layer norm go to the kernels as bare pointers too: a layer that
    was never moved to the input's device, or another size, stops in the call layer, through the layers' nodes and
    through the operators.  (On CPU tensors, as above; the other device is torch's meta device.)"""
    from flashdp4review_b200 import _lib
    from flashdp4review_b200.core import ops
    monkeypatch.setattr(ops, "_require_cuda", lambda *tensors: None)
    host = _lib.host()
    x, w, b = torch.zeros(2, 3, 16), torch.ones(16), torch.zeros(16)
    for fwd in (lambda *a: ops.layernorm_fwd_fused(*a, 1e-5), lambda *a: host.dp_layernorm(*a, None, 1e-5)):
        for args in ((x, w.to("meta"), b), (x, w, b.to("meta")), (x.to("meta"), w, b)):
            with pytest.raises(RuntimeError, match="not on one device"):
                fwd(*args)
        for args in ((x, torch.ones(15), b), (x, w, torch.zeros(8)), (x, torch.ones(17), torch.zeros(17))):
            with pytest.raises(RuntimeError, match="parameters do not fit"):
                fwd(*args)
    mean, rstd = torch.zeros(6), torch.ones(6)
    for args, refused in (((x, x, w.to("meta"), mean, rstd), "not on one device"), ((x, x, torch.ones(8), mean, rstd), "parameters do not fit"),
                          ((x, x, w, mean.to("meta"), rstd), "statistics"), ((x, x, w, mean, torch.ones(5)), "statistics"),
                          ((x, x, w, mean.double(), rstd), "statistics"), ((torch.zeros(2, 2, 16), x, w, mean, rstd), "grad_output"),
                          ((x.to("meta"), x, w, mean, rstd), "grad_output")):
        with pytest.raises(RuntimeError, match=refused):
            ops.dp_layernorm_backward(*args, 1.0, 1.0)


def test_partial_backward_takes_only_what_it_needs(no_launch):
    """Without the weight gradient (a frozen weight, a bias alone) the workspace of a whole backward is that of the
    remaining outputs, and the layer input stays out of the call: no cast, no copy."""
    from flashdp4review_b200 import _lib
    lib = _lib.load()
    q, d, b = lib.fdp_linear_bwd_workspace_bytes, lib.fdp_linear_dgrad_workspace_bytes, lib.fdp_bias_grad_workspace_bytes
    w = lib.fdp_linear_wgrad_workspace_bytes
    DX, DW, DB = 1, 2, 4
    wide = _lib.FDP_FP32_TENSOR | _lib.FDP_FP32_WIDE
    for (B, T, n_in, n_out) in ((4, 128, 768, 768), (3, 197, 264, 320), (2, 100, 136, 196), (64, 1, 1024, 1000), (3, 50, 72, 40)):
        for dt in (_lib.FDP_F32, _lib.FDP_BF16):
            algo = wide if dt == _lib.FDP_F32 else 0
            dx = d(B * T, n_in, n_out, dt | (algo & _lib.FDP_FP32_TENSOR))
            db = b(B, T, n_out, dt)
            assert q(B, T, n_in, n_out, dt, algo, DX) == dx
            assert q(B, T, n_in, n_out, dt, algo, DB) == db
            assert q(B, T, n_in, n_out, dt, algo, DX | DB) == max(dx, db)
            assert q(B, T, n_in, n_out, dt, algo, DW) == w(B, T, n_in, n_out, dt, algo)
    ops, Launched = no_launch
    X, G, W = torch.zeros(2, 3, 16, dtype=torch.float64), torch.zeros(2, 3, 8), torch.zeros(8, 16)
    for need in ((True, False, True), (True, False, False), (False, False, True)):
        with pytest.raises(Launched) as e:
            ops.dp_linear_backward(X, G, W, 1.0, 1.0, need_dx=need[0], need_dw=need[1], need_db=need[2])
        passed_X = e.value.args[1][1]
        assert passed_X is None
    with pytest.raises(Launched) as e:
        ops.dp_linear_backward(X, G, W, 1.0, 1.0)
    assert e.value.args[1][1].dtype == torch.float32


def test_input_gradient_of_a_whole_backward_needs_its_own_flag():
    """FDP_FP32_WIDE alone asks for six products in the weight gradient; the input gradient's three products are
    FDP_FP32_TENSOR's.  Without it nothing is shared, so the workspace holds no parts of W."""
    from flashdp4review_b200 import _lib
    q = _lib.load().fdp_linear_bwd_workspace_bytes
    w = _lib.load().fdp_linear_wgrad_workspace_bytes
    wide, both = _lib.FDP_FP32_WIDE, _lib.FDP_FP32_WIDE | _lib.FDP_FP32_TENSOR
    for (B, T, n_in, n_out) in ((2, 130, 128, 256), (4, 128, 256, 384), (3, 197, 264, 320)):
        plain = w(B, T, n_in, n_out, _lib.FDP_F32, wide)
        assert q(B, T, n_in, n_out, _lib.FDP_F32, wide, 3) == plain
        assert q(B, T, n_in, n_out, _lib.FDP_F32, both, 3) > w(B, T, n_in, n_out, _lib.FDP_F32, both)


def test_call_layer_is_rebuilt_for_another_torch(monkeypatch, tmp_path):
    """_fdp_host.so fits the torch that it was built against only: newer sources or another torch rebuild it."""
    import shutil
    import types
    from flashdp4review_b200 import build
    copy = tmp_path / "_fdp_host.so"
    shutil.copy(build.HOST_LIB, copy)           # (a new time of modification)
    compiled = []
    monkeypatch.setattr(build, "HOST_LIB", str(copy))
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **kw: compiled.append(cmd) or types.SimpleNamespace(returncode=0, stderr=""))
    build.build_host()
    assert not compiled
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    build.build_host()
    assert len(compiled) == 1 and str(copy) in compiled[0]
