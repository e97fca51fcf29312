"""Edge sizes of the kernels' tiles, boxes and dispatch rules, against float64 on the same rounded inputs."""
import pytest
import torch

from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from flashdp4review_b200.core import ops
    return ops


def _randn(*shape, seed, dtype, scale=1.0):
    gen = torch.Generator(device=dev()).manual_seed(seed)
    return (torch.randn(*shape, device=dev(), generator=gen) * scale).to(dtype)


def _close_to_sum(got, want, absum, k, unit):
    """|got - want| <= rounding of the result (unit, relative) + k fp32 additions of terms whose
    magnitudes add up to absum (one unit in the last place each, 2^-23)."""
    err = (got.double() - want).abs()
    bound = unit * want.abs() + (k * 2.0 ** -23) * absum + 1e-30
    assert bool((err <= bound).all()), float((err / bound).max())


UNIT = {torch.float32: 2.0 ** -23, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10}


# rows and columns around the 32-row x 128-byte output boxes and the 256 x 256 tiles
@pytest.mark.parametrize("rows,K,N", [(128, 64, 128), (129, 72, 136), (257, 200, 264), (511, 136, 328), (300, 64, 1000)])
@pytest.mark.parametrize("dtype,out_dtype", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32),
                                             (torch.float16, torch.float16)])
@pytest.mark.parametrize("bias", [True, False])
def test_output_boxes(ops, rows, K, N, dtype, out_dtype, bias):
    X, W = _randn(rows, K, seed=1, dtype=dtype), _randn(N, K, seed=2, dtype=dtype, scale=0.1)
    b = _randn(N, seed=3, dtype=dtype) if bias else None
    Y = ops.linear_forward(X, W, b, "out_in", out_dtype=out_dtype)
    want = X.double() @ W.double().t()
    absum = X.double().abs() @ W.double().abs().t()
    if bias:
        want, absum = want + b.double(), absum + b.double().abs()
    _close_to_sum(Y, want, absum, K + 1, UNIT[out_dtype])


# fp32 through six bf16 products: the ends of samples against 64-row K stages, sequences too short for the product
# form of the norm (T < 64), the smallest widths and row counts, widths whose rows are not multiples of 16 bytes
@pytest.mark.parametrize("B,T,n_in,n_out", [(1, 64, 64, 64), (2, 65, 72, 328), (3, 127, 257, 130), (5, 197, 520, 64),
                                            (64, 1, 65, 129), (9, 63, 333, 100), (2, 1000, 300, 515), (400, 70, 66, 66)])
@pytest.mark.parametrize("layout", ["out_in", "in_out"])
def test_fp32_six_products(ops, B, T, n_in, n_out, layout):
    X = _randn(B, T, n_in, seed=1, dtype=torch.float32)
    G = _randn(B, T, n_out, seed=2, dtype=torch.float32, scale=1e-2)
    G[0] *= 30.0
    dW, norms, factors = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, layout=layout, return_norms=True, fp32_tensor=True)
    per = torch.einsum("bto,bti->boi", G.double(), X.double())
    want_n = per.flatten(1).norm(dim=1)
    assert float(((norms.double() - want_n) / want_n).abs().max()) < 4 * 2.0 ** -23
    f = (1.0 / (want_n + 1e-10)).clamp(max=1.0)
    want = torch.einsum("boi,b->oi", per, f) / B
    absum = torch.einsum("bto,bti,b->oi", G.double().abs(), X.double().abs(), f) / B
    if layout == "in_out":
        want, absum = want.t(), absum.t()
    # 24 truncating steps within an accumulator, one rounded addition per 64 rows of a sample, the clip factor (4)
    _close_to_sum(dW, want, absum, 28 + B * ((T + 63) // 64), 2.0 ** -23)
    # the noise is the stream of the generic kernels, element for element, whatever the row pitch and alignment
    noise = ops.NoiseSpec(0.01, 5, 2, 0, 9)
    zero = torch.zeros_like(G)
    flat = torch.zeros(n_in * n_out + 1, device=dev())
    out = flat[1:].view(dW.shape)
    ops.dp_linear_weight_grad(X, zero, 1.0, 1.0, layout=layout, noise=noise, fp32_tensor=True, out=out)
    assert torch.equal(out, ops.dp_linear_weight_grad(X, zero, 1.0, 1.0, layout=layout, noise=noise, fp32_tensor=False))
    assert float(flat[0]) == 0.0


# many samples of few rows (at most 16 rows and more than 64 samples take kernels of their own): both sides of that line,
# widths off the 16-byte vectors, one row a sample
@pytest.mark.parametrize("B,T,n", [(64, 1, 256), (65, 1, 1000), (1025, 1, 257), (300, 3, 72), (66, 16, 130), (66, 17, 130), (4000, 2, 8)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_bias_gradient_of_short_samples(ops, B, T, n, dtype):
    G = _randn(B, T, n, seed=3, dtype=dtype, scale=0.1)
    db, norms, factors = ops.dp_bias_grad(G, 0.5, 1.0, out_dtype=torch.float32, return_norms=True)
    want_n = G.double().flatten(1).norm(dim=1)
    # sums of squares over T * n elements in chains of at most T * n / 32, then the root halves the error
    assert float(((norms.double() - want_n) / want_n).abs().max()) < (T * n / 64 + 8) * 2.0 ** -23
    f = (0.5 / (want_n + 1e-10)).clamp(max=1.0)
    assert float(((factors.double() - f) / f).abs().max()) < (T * n / 64 + 10) * 2.0 ** -23
    want = torch.einsum("bto,b->o", G.double(), f) / (B * T)
    absum = torch.einsum("bto,b->o", G.double().abs(), f) / (B * T)
    _close_to_sum(db, want, absum, B * T / 8 + T * n / 64 + 20, 2.0 ** -23)


# the norm of samples of one row is the product of the rows' norms
@pytest.mark.parametrize("B,n_in,n_out", [(1, 8, 8), (9, 1000, 1024), (300, 129, 65)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_norms_of_one_row_samples(ops, B, n_in, n_out, dtype):
    X, G = _randn(B, 1, n_in, seed=4, dtype=dtype), _randn(B, 1, n_out, seed=5, dtype=dtype, scale=1e-2)
    _, norms, _ = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, return_norms=True)
    want = G.double().flatten(1).norm(dim=1) * X.double().flatten(1).norm(dim=1)
    assert float(((norms.double() - want) / want).abs().max()) < ((n_in + n_out) / 64 + 12) * 2.0 ** -23


# one call for the whole backward: bit for bit what the three calls give, whether or not the split copies are shared
# (fp32: three products, six products with and without 16-byte rows, short sequences; 16 bit: plain)
@pytest.mark.parametrize("dtype,B,T,n_in,n_out", [
    (torch.float32, 4, 128, 256, 384), (torch.float32, 3, 197, 264, 320), (torch.float32, 2, 100, 136, 196), (torch.float32, 5, 70, 130, 128),
    (torch.float32, 40, 7, 128, 128), (torch.float32, 2, 130, 128, 129), (torch.bfloat16, 3, 256, 264, 136), (torch.float16, 4, 77, 128, 192)])
@pytest.mark.parametrize("layout", ["out_in", "in_out"])
@pytest.mark.parametrize("need", [(True, True, True), (True, True, False), (False, True, True), (True, False, True)])
def test_whole_backward_equals_its_parts(ops, dtype, B, T, n_in, n_out, layout, need):
    X, G = _randn(B, T, n_in, seed=6, dtype=dtype), _randn(B, T, n_out, seed=7, dtype=dtype, scale=1e-2)
    W = _randn(*((n_out, n_in) if layout == "out_in" else (n_in, n_out)), seed=8, dtype=dtype, scale=0.05)
    nw, nb = ops.NoiseSpec(0.01, 5, 2, 0, 9), ops.NoiseSpec(0.01, 5, 3, 0, 9)
    dX, dW, db = ops.dp_linear_backward(X, G, W, 0.7, 1.0, need_dx=need[0], need_dw=need[1], need_db=need[2], noise=nw,
                                        noise_bias=nb, layout=layout, dw_dtype=torch.float32, db_dtype=torch.float32)
    assert (dX is not None, dW is not None, db is not None) == need
    if need[0]:
        assert torch.equal(dX, ops.linear_input_grad(G, W, layout))
    if need[1]:
        assert torch.equal(dW, ops.dp_linear_weight_grad(X, G, 0.7, 1.0, noise=nw, layout=layout, out_dtype=torch.float32))
    if need[2]:
        assert torch.equal(db, ops.dp_bias_grad(G, 0.7, 1.0, noise=nb, out_dtype=torch.float32))


# LayerNorm backward with rows whose ring stages are 64 KB (wide fp32): a chunk shorter than the ring, a ragged last
# stage, widths that do and do not fill the threads' columns
@pytest.mark.parametrize("B,T,d", [(2, 3, 1024), (3, 37, 1000), (2, 70, 4096), (2, 33, 8192), (1, 130, 5000)])
def test_layernorm_backward_of_wide_fp32_rows(ops, B, T, d):
    x, dy = _randn(B, T, d, seed=9, dtype=torch.float32), _randn(B, T, d, seed=10, dtype=torch.float32, scale=0.1)
    w, b = 1.0 + _randn(d, seed=11, dtype=torch.float32, scale=0.1), torch.zeros(d, device=dev())
    _, buf, _ = ops.layernorm_fwd_fused(x, w, b, 1e-5)
    dx, dg, db = ops.dp_layernorm_backward(dy, x, w, buf["mean"], buf["rstd"], 1e6, 1.0, batch_divisor=1)
    xd, dyd, wd = x.double(), dy.double(), w.double()
    rs = 1.0 / torch.sqrt(xd.var(-1, unbiased=False, keepdim=True) + 1e-5)
    xh = (xd - xd.mean(-1, keepdim=True)) * rs
    wdy = dyd * wd
    want = rs * (wdy - xh * (wdy * xh).mean(-1, keepdim=True) - wdy.mean(-1, keepdim=True))
    absum = rs * (wdy.abs() + xh.abs() * (wdy * xh).abs().mean(-1, keepdim=True) + wdy.abs().mean(-1, keepdim=True))
    # a row's sums run in chains of at most d / 32 additions; mean and rstd carry as many
    _close_to_sum(dx, want, absum, d / 16 + 16, 2.0 ** -23)
    _close_to_sum(dg, (dyd * xh).sum((0, 1)), (dyd * xh).abs().sum((0, 1)) + rs.mean() * dyd.abs().sum((0, 1)), B * T + d / 32 + 16, 2.0 ** -23)
    _close_to_sum(db, dyd.sum((0, 1)), dyd.abs().sum((0, 1)), B * T + 8, 2.0 ** -23)


# 16-bit weight gradients whose samples end inside a K stage: factors in the epilogue or in a copy of G, norms by product
# tiles or by Gram blocks
@pytest.mark.parametrize("B,T,n_in,n_out", [(3, 257, 136, 264), (2, 300, 520, 128), (12, 500, 256, 256), (2, 319, 2048, 128), (5, 65, 128, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("algo", ["auto", "direct", "gram"])
def test_ragged_samples_16bit(ops, B, T, n_in, n_out, dtype, algo):
    X, G = _randn(B, T, n_in, seed=12, dtype=dtype), _randn(B, T, n_out, seed=13, dtype=dtype, scale=1e-2)
    G[0] *= 30.0
    dW, norms, _ = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, norm_algo=algo, out_dtype=torch.float32, return_norms=True)
    per = torch.einsum("bto,bti->boi", G.double(), X.double())
    want_n = per.flatten(1).norm(dim=1)
    assert float(((norms.double() - want_n) / want_n).abs().max()) < 1e-4
    f = (1.0 / (want_n + 1e-10)).clamp(max=1.0)
    absum = torch.einsum("bto,bti,b->oi", G.double().abs(), X.double().abs(), f) / B
    # fp32 sums; the pre-scaled copy rounds c_b G to the input type, half a unit each
    err = (dW.double() - torch.einsum("boi,b->oi", per, f) / B).abs()
    assert bool((err <= (UNIT[dtype] / 2 + (B * T / 16 + 32) * 2.0 ** -23) * absum).all())


def test_six_products_fall_back_where_their_workspace_does_not_fit(ops):
    """fp32 shapes that ran in little memory before still do: without room for the split copies and the parking area
    (38.8 MB) the FMA kernels take the call."""
    X, G = _randn(4, 100, 256, seed=14, dtype=torch.float32), _randn(4, 100, 192, seed=15, dtype=torch.float32)
    want = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, fp32_tensor=False)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (24 << 20)) / total)
        got = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, fp32_tensor=True)
        _, dW, _ = ops.dp_linear_backward(X, G, None, 1.0, 1.0, need_dx=False)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(got, want) and torch.equal(dW, want)


# FDP_FP32_WIDE without FDP_FP32_TENSOR through the C ABI: the input gradient is that of the FMA kernels, bit for bit,
# whatever the pointers' alignment lets the weight gradient do
@pytest.mark.parametrize("B,T,n_in,n_out", [(2, 130, 128, 256), (4, 128, 256, 384), (40, 7, 128, 128)])
@pytest.mark.parametrize("layout", ["out_in", "in_out"])
def test_wide_flag_alone_leaves_the_input_gradient_exact(ops, B, T, n_in, n_out, layout):
    from flashdp4review_b200 import _lib
    lib = _lib.load()
    X, G = _randn(B, T, n_in, seed=16, dtype=torch.float32), _randn(B, T, n_out, seed=17, dtype=torch.float32, scale=1e-2)
    W = _randn(*((n_out, n_in) if layout == "out_in" else (n_in, n_out)), seed=18, dtype=torch.float32, scale=0.05)
    dX, dW = torch.empty_like(X), torch.empty_like(W)
    p = _lib.DPParams(1.0, 1.0, 0.0, 0, 0, 0, 0, 0, 0, 1, None)
    algo, lay = _lib.FDP_FP32_WIDE, _lib.FDP_OUT_IN if layout == "out_in" else _lib.FDP_IN_OUT
    ws = torch.empty(lib.fdp_linear_bwd_workspace_bytes(B, T, n_in, n_out, _lib.FDP_F32, algo, 3), dtype=torch.uint8, device=dev())
    st = lib.fdp_linear_bwd(G.data_ptr(), X.data_ptr(), W.data_ptr(), dX.data_ptr(), dW.data_ptr(), None, B, T, n_in, n_out,
                            *[_lib.FDP_F32] * 4, lay, algo, p, p, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    assert st == _lib.FDP_OK
    assert torch.equal(dX, ops.linear_input_grad(G, W, layout, fp32_tensor=False))
    assert _lib.load().fdp_device_status(None, torch.cuda.current_stream().cuda_stream) == _lib.FDP_OK


@pytest.mark.parametrize("T", [128, 130])
def test_whole_backward_one_output_at_a_time_where_its_workspace_does_not_fit(ops, T):
    """Where the workspace of the whole call does not fit, that of one output after the other may: the same bits, with
    three products (T = 128) and with six (T = 130)."""
    from flashdp4review_b200 import _lib
    B, n = 4, 4096
    X, G = _randn(B, T, n, seed=19, dtype=torch.float32), _randn(B, T, n, seed=20, dtype=torch.float32, scale=1e-2)
    W = _randn(n, n, seed=21, dtype=torch.float32, scale=0.05)
    want = [t.cpu() for t in ops.dp_linear_backward(X, G, W, 1.0, 1.0)]
    q = lambda outputs: _lib.load().fdp_linear_bwd_workspace_bytes(B, T, n, n, _lib.FDP_F32, _lib.FDP_FP32_TENSOR | _lib.FDP_FP32_WIDE, outputs)
    # what the results (dX in a segment of 20 MB, db in one of 2 MB, dW) and the largest single workspace take, 6 MB for
    # the allocator's rounding; dW and the whole call's workspace alone take more
    room = (22 << 20) + 4 * n * n + max(q(1), q(2), q(4)) + (6 << 20)
    assert 4 * n * n + q(7) > room + (2 << 20)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + room) / total)
        got = ops.dp_linear_backward(X, G, W, 1.0, 1.0)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for a, b in zip(got, want):
        assert torch.equal(a.cpu(), b)


# a sample with an infinity or a NaN: its norm is infinite, its clip factor 0, and only the rows (columns) that hold the
# element are lost; every norm algorithm and every kernel that derives factors
@pytest.mark.parametrize("dtype,B,T,n_in,n_out,algo,fp32_tensor", [
    (torch.float32, 3, 197, 128, 136, "auto", True), (torch.float32, 3, 128, 128, 192, "auto", True),
    (torch.float32, 40, 7, 128, 136, "auto", True), (torch.float32, 130, 1, 128, 136, "auto", True),
    (torch.float32, 3, 197, 40, 40, "direct", False), (torch.float32, 3, 197, 40, 40, "gram", False), (torch.float32, 3, 50, 40, 40, "auto", False),
    (torch.bfloat16, 3, 256, 128, 128, "direct", None), (torch.bfloat16, 3, 256, 128, 128, "gram", None),
    (torch.float16, 3, 300, 136, 128, "auto", None), (torch.bfloat16, 400, 64, 128, 128, "auto", None)])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("where", ["input", "grad_output"])
def test_non_finite_samples_are_clipped_away(ops, dtype, B, T, n_in, n_out, algo, fp32_tensor, value, where):
    X, G = _randn(B, T, n_in, seed=22, dtype=dtype), _randn(B, T, n_out, seed=23, dtype=dtype, scale=1e-2)
    X[1] *= 4.0
    rest = [b for b in range(B) if b != 1]
    row, col = (T - 1) // 2, 5
    (X if where == "input" else G)[1, row, col] = value
    dW, norms, factors = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, norm_algo=algo, return_norms=True, out_dtype=torch.float32,
                                                   fp32_tensor=fp32_tensor)
    assert float(norms[1]) == float("inf") and float(factors[1]) == 0.0
    assert bool(norms[rest].isfinite().all()) and bool((factors[rest] > 0).all())
    # the other elements are the sums of the other samples, at the same divisor
    want = ops.dp_linear_weight_grad(X[rest].contiguous(), G[rest].contiguous(), 1.0, 1.0, batch_divisor=B, norm_algo=algo,
                                     out_dtype=torch.float32, fp32_tensor=fp32_tensor)
    lost = ~dW.isfinite()
    mask = torch.zeros_like(lost)
    (mask[:, col] if where == "input" else mask[col]).fill_(True)
    assert bool((lost <= mask).all())
    err = (dW - want)[~mask].abs().max() / want.abs().max()
    assert float(err) < 1e-2 if dtype != torch.float32 else float(err) < 1e-5
    if where == "grad_output":
        db, norms, factors = ops.dp_bias_grad(G, 1.0, 1.0, out_dtype=torch.float32, return_norms=True)
        assert float(norms[1]) == float("inf") and float(factors[1]) == 0.0
        keep = [o for o in range(n_out) if o != col]
        assert bool(db[keep].isfinite().all())


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_non_finite_samples_of_a_layernorm_are_clipped_away(ops, value):
    B, T, d = 3, 17, 96
    x, dy = _randn(B, T, d, seed=24, dtype=torch.float32), _randn(B, T, d, seed=25, dtype=torch.float32)
    w, b = torch.ones(d, device=dev()), torch.zeros(d, device=dev())
    _, buf, _ = ops.layernorm_fwd_fused(x, w, b, 1e-5)
    dy[1, 3, 5] = value
    _, dg, db, ng, nb = ops.dp_layernorm_backward(dy, x, w, buf["mean"], buf["rstd"], 1.0, 1.0, return_norms=True)
    assert float(ng[1]) == float("inf") and float(nb[1]) == float("inf")
    keep = [c for c in range(d) if c != 5]
    rest = [0, 2]
    _, wg, wb = ops.dp_layernorm_backward(dy[rest].contiguous(), x[rest].contiguous(), w, buf["mean"].view(B, T)[rest].reshape(-1).contiguous(),
                                          buf["rstd"].view(B, T)[rest].reshape(-1).contiguous(), 1.0, 1.0, batch_divisor=B)
    for got, want in ((dg, wg), (db, wb)):
        assert float((got - want)[keep].abs().max() / want.abs().max()) < 1e-5


# norms of short samples with long rows: as close to float64 as those of the general kernels (64 samples and fewer)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,n", [(300, 1, 8192), (300, 4, 4096), (300, 8, 4096), (300, 2, 4097)])
def test_norms_of_short_samples_are_as_accurate(ops, dtype, B, T, n):
    G = _randn(B, T, n, seed=26, dtype=dtype, scale=0.1)
    want = G[:64].double().flatten(1).norm(dim=1)
    rms = []
    for part in (G[:64], G):
        _, norms, _ = ops.dp_bias_grad(part, 1.0, 1.0, return_norms=True)
        rms.append(float(((norms[:64].double() - want) / want).square().mean().sqrt()))
    # half as much again, and half a unit in the last place for the root
    assert rms[1] < 1.5 * rms[0] + 2.0 ** -25, rms


# ... and long rows against few samples take the general kernels: both sides of the line, by the launches of a call
# (three of the short kernels, two of the general ones) and against float64
@pytest.mark.parametrize("dtype,B,T,n,short", [
    (torch.float32, 65, 16, 11008, False), (torch.float32, 65, 16, 4096, False), (torch.bfloat16, 65, 16, 4096, False),
    (torch.float32, 65, 1, 11008, True), (torch.float32, 65, 11, 1000, True), (torch.float32, 65, 12, 1000, False),
    (torch.bfloat16, 65, 16, 1000, True), (torch.float32, 200, 16, 1000, True), (torch.float16, 128, 16, 11008, False)])
def test_bias_gradient_of_short_samples_with_long_rows(ops, dtype, B, T, n, short):
    from flashdp4review_b200 import _lib
    G = _randn(B, T, n, seed=27, dtype=dtype, scale=0.1)
    before = _lib.load().fdp_launch_count()
    db, norms, _ = ops.dp_bias_grad(G, 0.5, 1.0, out_dtype=torch.float32, return_norms=True)
    assert _lib.load().fdp_launch_count() - before == (3 if short else 2)
    want_n = G.double().flatten(1).norm(dim=1)
    assert float(((norms.double() - want_n) / want_n).abs().max()) < (T * n / 256 + 8) * 2.0 ** -23
    f = (0.5 / (want_n + 1e-10)).clamp(max=1.0)
    want = torch.einsum("bto,b->o", G.double(), f) / (B * T)
    absum = torch.einsum("bto,b->o", G.double().abs(), f) / (B * T)
    _close_to_sum(db, want, absum, B * T / 8 + T * n / 256 + 20, 2.0 ** -23)


def _parts(v):
    """the three bf16 parts of an fp32 number"""
    v, out = torch.tensor(v, dtype=torch.float32), []
    for _ in range(3):
        p = v.to(torch.bfloat16).float()
        out.append(float(p))
        v = v - p
    assert float(v) == 0.0
    return out


# every one of the six products is there, in the gradient and in the norms: with constant operands what a product
# contributes adds up over all elements instead of averaging out
@pytest.mark.parametrize("B,T,n_in,n_out", [(2, 64, 72, 130), (1, 65, 257, 100), (3, 127, 64, 300), (2, 192, 136, 264)])
@pytest.mark.parametrize("layout", ["out_in", "in_out"])
def test_fp32_six_products_are_six(ops, B, T, n_in, n_out, layout):
    g = 1.0 + 2.0 ** -9 + 2.0 ** -10 + 2.0 ** -18 + 2.0 ** -19 + 2.0 ** -20
    x = 1.0 + 2.0 ** -9 + 2.0 ** -11 + 2.0 ** -18 + 2.0 ** -19 + 2.0 ** -21
    G, X = torch.full((B, T, n_out), g, device=dev()), torch.full((B, T, n_in), x, device=dev())
    assert float(G[0, 0, 0]) == g and float(X[0, 0, 0]) == x
    dW, norms, _ = ops.dp_linear_weight_grad(X, G, 1e9, 1.0, batch_divisor=1, layout=layout, return_norms=True, fp32_tensor=True)
    # steps on a large accumulator (4 of the 24 of a hand-off; 2 of the norm pass) truncate up to a unit each, the
    # additions of the hand-offs in registers round up to half a unit each; the norm's sums of squares 8 more
    n = (T + 63) // 64
    bound = (4 + B * n / 2 + 2) * 2.0 ** -23
    bound_n = (2 + 2 * n / 2 + 8) * 2.0 ** -23
    rel = ((dW.double() - B * T * g * x).abs() / (B * T * g * x)).max()
    want_n = T * g * x * (n_in * n_out) ** 0.5
    rel_n = ((norms.double() - want_n).abs() / want_n).max()
    assert float(rel) < bound and float(rel_n) < bound_n, (float(rel), float(rel_n))
    # what a missing product would make of it: further off than the bounds allow, each of the six
    pg, px = _parts(g), _parts(x)
    for i in range(3):
        for j in range(3 - i):
            assert pg[i] * px[j] / (g * x) > 2 * max(bound, bound_n), (i, j)


# the FMA kernels on the same ragged shapes: the path of "exact" mode and of a card without room for the split copies
@pytest.mark.parametrize("B,T,n_in,n_out", [(1, 64, 64, 64), (2, 65, 72, 328), (3, 127, 257, 130), (5, 197, 520, 64),
                                            (64, 1, 65, 129), (9, 63, 333, 100), (2, 1000, 300, 515), (400, 70, 66, 66)])
@pytest.mark.parametrize("layout", ["out_in", "in_out"])
def test_fp32_ragged_shapes_on_fma_kernels(ops, B, T, n_in, n_out, layout):
    X = _randn(B, T, n_in, seed=1, dtype=torch.float32)
    G = _randn(B, T, n_out, seed=2, dtype=torch.float32, scale=1e-2)
    G[0] *= 30.0
    dW, norms, _ = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, layout=layout, return_norms=True, fp32_tensor=False)
    per = torch.einsum("bto,bti->boi", G.double(), X.double())
    want_n = per.flatten(1).norm(dim=1)
    assert float(((norms.double() - want_n) / want_n).abs().max()) < 1e-5
    f = (1.0 / (want_n + 1e-10)).clamp(max=1.0)
    want = torch.einsum("boi,b->oi", per, f) / B
    absum = torch.einsum("bto,bti,b->oi", G.double().abs(), X.double().abs(), f) / B
    if layout == "in_out":
        want, absum = want.t(), absum.t()
    _close_to_sum(dW, want, absum, B * T + 100, 2.0 ** -23)      # one chain over all rows; 1e-5 of the factor is 84 units
