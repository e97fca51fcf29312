"""Weight gradients whose per-sample products are kept and summed: tile edges, every input form, noise, against float64."""
import pytest
import torch

from gpu_util import dev
from test_gpu_edges import UNIT, _close_to_sum, _randn, ops  # noqa: F401

pytestmark = pytest.mark.gpu


def _kept(call):
    """whether `call` sums kept products"""
    call()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return any("weighted_sum_kernel" in e.name for e in p.events())


# edges of the 256 x 256 tiles and their 32 x 32 boxes, one tile and several, samples that end inside a K stage, 8 and
# more samples to a sum, three and six products
@pytest.mark.parametrize("B,T,n_in,n_out,dtype", [
    (1, 256, 128, 128, torch.bfloat16), (3, 270, 200, 264, torch.float16), (9, 319, 520, 136, torch.bfloat16),
    (17, 300, 264, 776, torch.bfloat16), (2, 1000, 256, 512, torch.float16), (4, 128, 256, 320, torch.float32),
    (9, 192, 512, 256, torch.float32), (2, 64, 64, 64, torch.float32), (3, 100, 130, 1001, torch.float32),
    (11, 70, 259, 97, torch.float32)])
@pytest.mark.parametrize("layout", ["out_in", "in_out"])
def test_kept_products(ops, B, T, n_in, n_out, dtype, layout):  # noqa: F811
    X, G = _randn(B, T, n_in, seed=1, dtype=dtype), _randn(B, T, n_out, seed=2, dtype=dtype, scale=1e-2)
    G[0] *= 30.0
    assert _kept(lambda: ops.dp_linear_weight_grad(X, G, 1.0, 1.0, layout=layout))
    per = torch.einsum("bto,bti->boi", G.double(), X.double())
    want_n = per.flatten(1).norm(dim=1)
    f = (1.0 / (want_n + 1e-10)).clamp(max=1.0)
    want = (f.view(-1, 1, 1) * per).sum(0) / B
    absum = (f.view(-1, 1, 1) * torch.einsum("bto,bti->boi", G.double().abs(), X.double().abs())).sum(0) / B
    if layout == "in_out":
        want, absum = want.t(), absum.t()
    # three products leave out what lies below 2^-16 of a product of two elements (2^-8 of each), the others nothing
    dropped = 2.0 ** -16 if dtype == torch.float32 and n_in % 64 == 0 and n_out % 64 == 0 and T % 64 == 0 and T >= 128 else 0.0
    for out_dtype in (torch.float32, torch.bfloat16):
        dW, norms, factors = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, layout=layout, out_dtype=out_dtype, return_norms=True)
        k = T // 16 + B + 8        # additions on the way to an element: one a K step, one a sample, the factor's roundings
        _close_to_sum(dW, want, absum * (1 + dropped * 2 ** 23 / k), k, UNIT[out_dtype])
        assert float(((norms.double() - want_n) / want_n).abs().max()) < (T / 16 + 8) * 2.0 ** -23 + dropped
        assert float(((factors.double() - f) / f).abs().max()) < (T / 16 + 12) * 2.0 ** -23 + dropped


@pytest.mark.parametrize("B,T,n_in,n_out", [(1, 4096, 1024, 1024), (2, 8192, 256, 256), (4, 4096, 264, 512), (1, 4000, 130, 520)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_long_samples_do_not_drift(ops, B, T, n_in, n_out, dtype):  # noqa: F811
    """An accumulator takes 32 truncated steps at most, each of which loses a unit of 2^-23 of what it holds at most, whatever the
    plan; what it holds is added with rounding.  Terms of one sign, clipping off: nothing hides a drift."""
    X, G = _randn(B, T, n_in, seed=1, dtype=dtype).abs(), _randn(B, T, n_out, seed=2, dtype=dtype, scale=1e-2).abs()
    per = torch.einsum("bto,bti->boi", G.double(), X.double())
    want, n = per.sum(0) / B, per.flatten(1).norm(dim=1)
    dW, norms, _ = ops.dp_linear_weight_grad(X, G, 1e9, 1.0, out_dtype=torch.float32, return_norms=True)
    bound = 32 * 2.0 ** -23 + (B * T / 512 + 8) ** 0.5 * 2.0 ** -24
    assert float((dW.double() - want).norm() / want.norm()) < bound
    if _kept(lambda: ops.dp_linear_weight_grad(X, G, 1.0, 1.0)):
        assert float(((norms.double() - n) / n).abs().max()) < bound


@pytest.mark.parametrize("B,T,n_in,n_out", [(4, 2387, 72, 1024), (8, 3264, 128, 136), (5, 1984, 70, 1648)])
def test_long_samples_in_six_products_are_summed_in_two_levels(ops, B, T, n_in, n_out):  # noqa: F811
    """Registers sum two hand-offs a stage over at most max(4, half a part) stages and the kept tile sums what they leave: the
    rounding errors (2^-24 / sqrt(3) of the running sum each, independent) of a chain of n are sqrt(n / 2) of one, and the
    truncation of the hand-offs is a unit of 2^-24."""
    X, G = _randn(B, T, n_in, seed=1, dtype=torch.float32), _randn(B, T, n_out, seed=2, dtype=torch.float32, scale=1e-2)
    assert _kept(lambda: ops.dp_linear_weight_grad(X, G, 1e9, 1.0))
    want = torch.einsum("bto,bti->oi", G.double(), X.double()) / B
    stages, parts = (T + 63) // 64, min(16, 2 * 74 // (-(-n_in // 256) * -(-n_out // 256)))
    F = max(4, B * stages // parts // 2 + 1)
    dW = ops.dp_linear_weight_grad(X, G, 1e9, 1.0)
    assert float((dW.double() - want).norm() / want.norm()) < (((2 * F + stages / F + 1) / 2 / 3) ** 0.5 + 1) * 2.0 ** -24


def test_kept_products_noise_and_infinities(ops):  # noqa: F811
    """A zero gradient returns the noise stream of the direct form bit for bit, with rows of any pitch; a sample that is
    not finite has norm inf and factor 0 and leaves the others' elements alone."""
    spec = ops.NoiseSpec(std=0.5, seed=77, param_id=3, step=2, rank=1, world=2)
    for (n_in, n_out, dtype) in ((264, 200, torch.bfloat16), (259, 97, torch.float32)):
        T = 256 if dtype == torch.bfloat16 else 128
        X, G = _randn(4, T, n_in, seed=1, dtype=dtype), torch.zeros(4, T, n_out, device=dev(), dtype=dtype)
        assert _kept(lambda: ops.dp_linear_weight_grad(X, G, 1.0, 1.0))
        kw = dict(batch_divisor=8, noise=spec, out_dtype=torch.float32)
        assert torch.equal(ops.dp_linear_weight_grad(X, G, 1.0, 1.0, **kw),
                           ops.dp_linear_weight_grad(X, G, 1.0, 1.0, norm_algo="direct", **kw))
        G = _randn(4, T, n_out, seed=2, dtype=dtype, scale=1e-2)
        clean = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, out_dtype=torch.float32)
        G[2, 5, 7] = float("inf")
        dW, norms, factors = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, out_dtype=torch.float32, return_norms=True)
        assert norms[2] == float("inf") and factors[2] == 0 and bool(torch.isfinite(norms[[0, 1, 3]]).all())
        rows = torch.arange(n_out, device=dev()) != 7
        G[2] = 0.0
        rest = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, out_dtype=torch.float32)
        assert torch.equal(dW[rows], rest[rows]) and not torch.equal(dW[rows], clean[rows])


def test_kept_products_give_way(ops):  # noqa: F811
    """Where the products do not fit the card the call contracts twice."""
    B, T, n = 8, 2048, 2048                      # 134 MB of products
    X, G = _randn(B, T, n, seed=1, dtype=torch.bfloat16), _randn(B, T, n, seed=2, dtype=torch.bfloat16, scale=1e-2)
    call = lambda: ops.dp_linear_weight_grad(X, G, 1.0, 1.0, out_dtype=torch.float32)   # noqa: E731
    assert _kept(call)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        # the result and the parking area (38.8 MB) have room, the products have not
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (96 << 20)) / total)
        got = call()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(got, ops.dp_linear_weight_grad(X, G, 1.0, 1.0, out_dtype=torch.float32, norm_algo="direct"))


# products whose last round of tiles is cut in two along N: behind full rounds, alone, with halves that overhang or miss
# the matrix, K-major and MN-major weights, 16-bit and fp32 (three products)
@pytest.mark.parametrize("rows,K,N", [(256 * 80, 64, 256), (256 * 25 + 3, 128, 776), (200, 320, 264), (130, 128, 136)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("layout", ["out_in", "in_out"])
def test_cut_tiles(ops, rows, K, N, dtype, layout):  # noqa: F811
    if dtype == torch.float32 and K < 128:
        K = 128
    X, W = _randn(rows, K, seed=1, dtype=dtype), _randn(*((N, K) if layout == "out_in" else (K, N)), seed=2, dtype=dtype, scale=0.1)
    b = _randn(N, seed=3, dtype=dtype)
    w = W if layout == "in_out" else W.t()
    want, absum = X.double() @ w.double() + b.double(), X.double().abs() @ w.double().abs() + b.double().abs()
    # three products leave out what lies below 2^-16 of a product of two elements
    k = K / 16 + 8 + (2.0 ** 7 if dtype == torch.float32 else 0)
    _close_to_sum(ops.linear_forward(X, W, b, layout), want, absum, k, UNIT[dtype])
    G = _randn(rows, N, seed=4, dtype=dtype)
    _close_to_sum(ops.linear_input_grad(G, W, layout), G.double() @ w.double().t(), G.double().abs() @ w.double().abs().t(),
                  N / 16 + 8 + (2.0 ** 7 if dtype == torch.float32 else 0), UNIT[dtype])


# fp32 forward and input gradient in six products: widths of any number (rows that are no multiple of 16 bytes, K stages and
# tiles that end past the last column), the smallest sizes, cut along K and not, misaligned operands
@pytest.mark.parametrize("rows,K,N", [(128, 64, 65), (130, 65, 64), (129, 100, 257), (200, 1999, 70), (1000, 333, 515), (300, 2000, 100)])
@pytest.mark.parametrize("layout", ["out_in", "in_out"])
@pytest.mark.parametrize("offset", [0, 1])
def test_fp32_products_in_six(ops, rows, K, N, layout, offset):  # noqa: F811
    def tensor(*shape, seed, scale=1.0):
        n = 1
        for d in shape:
            n *= d
        return _randn(n + offset, seed=seed, dtype=torch.float32, scale=scale)[offset:].view(*shape)
    X, G, b = tensor(rows, K, seed=1), tensor(rows, N, seed=2), tensor(N, seed=3)
    W = tensor(*((N, K) if layout == "out_in" else (K, N)), seed=4, scale=0.1)
    w = W if layout == "in_out" else W.t()
    # each hand-off of 24 steps of which four meet a large accumulator, then one rounded addition a stage, and the parts
    bound = lambda k: k / 64 * 2 + 8        # noqa: E731
    _close_to_sum(ops.linear_forward(X, W, b, layout), X.double() @ w.double() + b.double(),
                  X.double().abs() @ w.double().abs() + b.double().abs(), bound(K), UNIT[torch.float32])
    _close_to_sum(ops.linear_input_grad(G, W, layout), G.double() @ w.double().t(), G.double().abs() @ w.double().abs().t(),
                  bound(N), UNIT[torch.float32])


@pytest.mark.parametrize("layout", ["out_in", "in_out"])
def test_whole_backward_in_six_products(ops, layout):  # noqa: F811
    """One split of G serves the weight gradient and an input gradient in six products: the same bits as the calls alone."""
    B, T, n_in, n_out = 3, 100, 330, 1001
    X, G = _randn(B, T, n_in, seed=1, dtype=torch.float32), _randn(B, T, n_out, seed=2, dtype=torch.float32, scale=1e-2)
    W = _randn(*((n_out, n_in) if layout == "out_in" else (n_in, n_out)), seed=3, dtype=torch.float32, scale=0.1)
    dX, dW, db = ops.dp_linear_backward(X, G, W, 1.0, 1.0, layout=layout)
    assert torch.equal(dX, ops.linear_input_grad(G, W, layout))
    assert torch.equal(dW, ops.dp_linear_weight_grad(X, G, 1.0, 1.0, layout=layout))
    assert torch.allclose(db, ops.dp_bias_grad(G, 1.0, 1.0), rtol=1e-5, atol=1e-9)


# 16-bit and three-product outputs whose parts are parked and added, with and without bias
@pytest.mark.parametrize("rows,K,N", [(300, 8192, 264), (972, 3520, 688), (128, 4096, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("layout", ["out_in", "in_out"])
def test_products_cut_along_k(ops, rows, K, N, dtype, layout):  # noqa: F811
    from flashdp4review_b200 import _lib
    q = _lib.load().fdp_linear_dgrad_workspace_bytes
    code = {torch.bfloat16: _lib.FDP_BF16, torch.float32: _lib.FDP_F32 | _lib.FDP_FP32_TENSOR}[dtype]
    assert q(rows, N, K, code | _lib.FDP_GEMM_SPLIT_K) > q(rows, N, K, code)
    X, W = _randn(rows, K, seed=1, dtype=dtype), _randn(*((N, K) if layout == "out_in" else (K, N)), seed=2, dtype=dtype, scale=0.1)
    w = W if layout == "in_out" else W.t()
    want, absum = X.double() @ w.double(), X.double().abs() @ w.double().abs()
    k = K / 16 + 8 + (2.0 ** 7 if dtype == torch.float32 else 0)     # (as in test_cut_tiles)
    for b in (None, _randn(N, seed=3, dtype=dtype)):
        bd = 0.0 if b is None else b.double()
        _close_to_sum(ops.linear_forward(X, W, b, layout), want + bd, absum + (0.0 if b is None else bd.abs()), k, UNIT[dtype])


# 16-bit layers of any width from 64 on: rows that are no multiple of 16 bytes (one operand, both, none), samples that end
# inside a K stage, samples of one row, kept and contracted twice, noise with rows of any pitch
@pytest.mark.parametrize("B,T,n_in,n_out", [(2, 64, 64, 64), (3, 300, 129, 1001), (5, 100, 72, 65), (1, 700, 333, 128), (40, 65, 130, 66),
                                            (9, 20, 515, 70), (3, 2, 600, 100), (30, 1, 257, 129), (200, 1, 100, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("layout", ["out_in", "in_out"])
def test_16bit_of_any_width(ops, B, T, n_in, n_out, dtype, layout):  # noqa: F811
    X, G = _randn(B, T, n_in, seed=1, dtype=dtype), _randn(B, T, n_out, seed=2, dtype=dtype, scale=1e-2)
    G[0] *= 30.0
    per = torch.einsum("bto,bti->boi", G.double(), X.double())
    want_n = per.flatten(1).norm(dim=1)
    f = (1.0 / (want_n + 1e-10)).clamp(max=1.0)
    want = (f.view(-1, 1, 1) * per).sum(0) / B
    absum = (f.view(-1, 1, 1) * torch.einsum("bto,bti->boi", G.double().abs(), X.double().abs())).sum(0) / B
    if layout == "in_out":
        want, absum = want.t(), absum.t()
    k = 4 + B * (T + 63) // 64 + 8        # four steps an accumulator, one addition a stage, the factor's roundings
    for out_dtype in (torch.float32, dtype):
        dW, norms, _ = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, layout=layout, out_dtype=out_dtype, return_norms=True)
        # below 2^-14 an fp16 result is rounded to a multiple of 2^-24, whatever its size
        steps = absum + (2.0 ** -25 / (k * 2.0 ** -23) if out_dtype == torch.float16 else 0.0)
        _close_to_sum(dW, want, steps, k, UNIT[out_dtype])
        assert float(((norms.double() - want_n) / want_n).abs().max()) < 8 * 2.0 ** -23
    zero = torch.zeros_like(G)
    spec = ops.NoiseSpec(std=0.5, seed=77, param_id=3, step=2)
    kw = dict(layout=layout, noise=spec, out_dtype=torch.float32)
    stream = ops.dp_linear_weight_grad(X.float(), zero.float(), 1.0, 1.0, fp32_tensor=False, **kw)      # of the FMA kernels
    assert torch.equal(ops.dp_linear_weight_grad(X, zero, 1.0, 1.0, **kw), stream)


@pytest.mark.parametrize("rows,K,N", [(128, 65, 64), (130, 64, 65), (300, 999, 130), (1000, 515, 1001), (129, 72, 100), (256, 4001, 72)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("layout", ["out_in", "in_out"])
def test_16bit_products_of_any_width(ops, rows, K, N, dtype, layout):  # noqa: F811
    X, W = _randn(rows, K, seed=1, dtype=dtype), _randn(*((N, K) if layout == "out_in" else (K, N)), seed=2, dtype=dtype, scale=0.1)
    G, b = _randn(rows, N, seed=3, dtype=dtype), _randn(N, seed=4, dtype=dtype)
    w = W if layout == "in_out" else W.t()
    _close_to_sum(ops.linear_forward(X, W, b, layout), X.double() @ w.double() + b.double(),
                  X.double().abs() @ w.double().abs() + b.double().abs(), K / 16 + 8, UNIT[dtype])
    for out_dtype in (dtype, torch.float32):
        _close_to_sum(ops.linear_input_grad(G, W, layout, out_dtype=out_dtype), G.double() @ w.double().t(),
                      G.double().abs() @ w.double().abs().t(), N / 16 + 8, UNIT[out_dtype])


@pytest.mark.parametrize("rows,K,N", [(130, 64, 65), (300, 999, 130), (256, 4001, 72), (128, 3648, 100)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("layout", ["out_in", "in_out"])
def test_fp32_outputs_of_16bit_products_of_any_width(ops, rows, K, N, dtype, layout):  # noqa: F811
    """In fp32 these are no further from float64 than the FMA kernels that computed them before: an accumulator takes four
    truncated steps (4 units of 2^-23 at most, of what it holds), its K / 64 contents are added with rounding to nearest, whose
    errors of at most 2^-24 of the sum are independent.  With terms of one sign no cancellation hides a drift."""
    X, W = _randn(rows, K, seed=1, dtype=dtype).abs(), _randn(*((N, K) if layout == "out_in" else (K, N)), seed=2, dtype=dtype).abs()
    G, b = _randn(rows, N, seed=3, dtype=dtype).abs(), _randn(N, seed=4, dtype=dtype).abs()
    w = (W if layout == "in_out" else W.t()).double()

    def check(got, want, k):
        assert float((got.double() - want).norm() / want.norm()) < 4 * 2.0 ** -23 + (k / 64 + 1) ** 0.5 * 2.0 ** -24
    f32 = torch.float32
    check(ops.linear_forward(X, W, b, layout, out_dtype=f32), X.double() @ w + b.double(), K)
    check(ops.linear_forward(X, W, None, layout, out_dtype=f32), X.double() @ w, K)
    check(ops.linear_input_grad(G, W, layout, out_dtype=f32), G.double() @ w.t(), N)
    wide = _randn(rows, K, seed=5, dtype=dtype).abs()        # the long contraction of an input gradient
    check(ops.linear_input_grad(wide, W, "in_out" if layout == "out_in" else "out_in", out_dtype=f32), wide.double() @ w, K)


# few short samples of wide layers in the product form, every type; and noise drawn by the fix-up kernel
@pytest.mark.parametrize("B,T,n_in,n_out,dtype", [(3, 44, 1024, 512, torch.bfloat16), (2, 2, 2000, 136, torch.float16), (8, 63, 256, 768, torch.bfloat16),
                                                  (3, 44, 512, 260, torch.float32), (2, 3, 1200, 123, torch.float32), (40, 20, 300, 300, torch.float32)])
def test_short_samples_as_products(ops, B, T, n_in, n_out, dtype):  # noqa: F811
    X, G = _randn(B, T, n_in, seed=1, dtype=dtype), _randn(B, T, n_out, seed=2, dtype=dtype, scale=1e-1)
    G[0] *= 30.0
    per = torch.einsum("bto,bti->boi", G.double(), X.double())
    want_n = per.flatten(1).norm(dim=1)
    f = (1.0 / (want_n + 1e-10)).clamp(max=1.0)
    dW, norms, _ = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, out_dtype=torch.float32, return_norms=True)
    absum = (f.view(-1, 1, 1) * torch.einsum("bto,bti->boi", G.double().abs(), X.double().abs())).sum(0) / B
    _close_to_sum(dW, (f.view(-1, 1, 1) * per).sum(0) / B, absum, 4 + B + 8, 2.0 ** -23)
    assert float(((norms.double() - want_n) / want_n).abs().max()) < 8 * 2.0 ** -23


@pytest.mark.parametrize("B,T,n_in,n_out", [(2, 71, 576, 1472), (5, 92, 512, 512), (300, 4, 256, 136)])
def test_noise_of_short_contractions(ops, B, T, n_in, n_out):  # noqa: F811
    X, G = _randn(B, T, n_in, seed=1, dtype=torch.bfloat16), _randn(B, T, n_out, seed=2, dtype=torch.bfloat16, scale=1e-2)
    spec = ops.NoiseSpec(std=0.5, seed=77, param_id=3, step=2)
    stream = ops.dp_linear_weight_grad(X.float(), torch.zeros_like(G).float(), 1.0, 1.0, fp32_tensor=False, noise=spec)
    kw = dict(out_dtype=torch.float32)
    assert torch.equal(ops.dp_linear_weight_grad(X, torch.zeros_like(G), 1.0, 1.0, noise=spec, **kw), stream)
    plain, noisy = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, **kw), ops.dp_linear_weight_grad(X, G, 1.0, 1.0, noise=spec, **kw)
    assert float((noisy - (plain + stream)).abs().max()) <= 2.0 ** -23 * float(noisy.abs().max())


_SINGLE_CTA_CHILD = r"""
import sys, torch
sys.path.insert(0, %r)
from flashdp4review_b200.core import ops
worst = 0.0
# padded 16-bit widths, samples of one K stage, fp32 parts: more tiles along the input's columns than along the output's, and
# the reverse; enough samples that the products are not kept
for (B, T, n_in, n_out, dtype) in [(200, 128, 520, 72, torch.bfloat16), (100, 128, 72, 520, torch.float16), (150, 100, 300, 65, torch.bfloat16),
                                   (300, 20, 600, 100, torch.float16), (2, 50, 2000, 136, torch.bfloat16), (3, 40, 1400, 260, torch.float32),
                                   (150, 70, 600, 72, torch.float32), (4, 300, 200, 648, torch.bfloat16)]:
    gen = torch.Generator(device="cuda").manual_seed(B)
    X = torch.randn(B, T, n_in, device="cuda", generator=gen).to(dtype)
    G = (torch.randn(B, T, n_out, device="cuda", generator=gen) * torch.linspace(1e-3, 1e-1, B, device="cuda").view(B, 1, 1)).to(dtype)
    per = torch.einsum("bto,bti->boi", G.double(), X.double())
    n = per.flatten(1).norm(dim=1)
    f = (1.0 / (n + 1e-10)).clamp(max=1.0)
    want = (f.view(-1, 1, 1) * per).sum(0) / B
    for layout in ("out_in", "in_out"):
        dW, norms, factors = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, layout=layout, out_dtype=torch.float32, return_norms=True)
        w = want if layout == "out_in" else want.t()
        worst = max(worst, float(((norms.double() - n) / n).abs().max()), float(((factors.double() - f) / f).abs().max()),
                    float((dW.double() - w).norm() / w.norm()) * 1e-3 if dtype != torch.float32 else float((dW.double() - w).norm() / w.norm()))
torch.cuda.synchronize()
print("WORST", worst)
"""


def test_single_cta_tiles_of_any_width():
    """FDP_TC_CTAS=1 (tiles of 128 x 256, whose number depends on the orientation) on the plans for any width and for short
    samples: norms and factors within the truncation of their chains (300 rows at most: 20 steps of half a unit), dW likewise or, where G is
    rounded once more to 16 bits, within 2^-9."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _SINGLE_CTA_CHILD % root], env={**os.environ, "FDP_TC_CTAS": "1"},
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    worst = float(r.stdout.strip().split("WORST")[-1])
    assert worst < 20 * 2.0 ** -23, worst


# fp32 operands that three bf16 parts cannot stand for: what cuBLAS's and the FMA kernels return.  Cut along K and not
# (300 x 2000 -> 100), both layouts, every place the operand can be in
@pytest.mark.parametrize("rows,K,N", [(130, 200, 65), (300, 2000, 100), (1000, 333, 515)])
@pytest.mark.parametrize("layout", ["out_in", "in_out"])
def test_fp32_products_of_numbers_that_bf16_lacks(ops, rows, K, N, layout):  # noqa: F811
    f32, inf = torch.float32, float("inf")
    X, b = _randn(rows, K, seed=1, dtype=f32), _randn(N, seed=3, dtype=f32)
    W = _randn(*((N, K) if layout == "out_in" else (K, N)), seed=2, dtype=f32, scale=0.1)
    G = _randn(rows, N, seed=4, dtype=f32)

    def same(got, want64):
        want = want64.to(f32)
        finite = torch.isfinite(want)
        assert torch.equal(torch.isfinite(got), finite)
        assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(got[~finite & ~torch.isnan(want)], want[~finite & ~torch.isnan(want)])
        assert float((got[finite].double() - want64[finite]).norm()) <= 2e-6 * float(want64[finite].norm())

    def check(x, w, g):
        wkn = (w if layout == "in_out" else w.t()).double()
        same(ops.linear_forward(x, w, b, layout), x.double() @ wkn + b.double())
        same(ops.linear_input_grad(g, w, layout), g.double() @ wkn.t())
        # the whole backward (N and K a multiple of four or not: G's parts come with its statistics or alone)
        dX, _, _ = ops.dp_linear_backward(x[: rows // 2 * 2].view(2, rows // 2, K), g[: rows // 2 * 2].view(2, rows // 2, N), w, 1.0, 1.0, layout=layout)
        same(dX.view(-1, K), g[: rows // 2 * 2].double() @ wkn.t())

    def put(t, value, *where):
        t = t.clone()
        t[where] = value
        return t
    for value in (inf, -inf, float("nan"), 3.4e38, -3.39999e38):
        check(put(X, value, 3, 5), W, put(G, value, rows - 1, N - 1))
        check(X, put(W, value, 1, 2), G)
    check(put(put(X, inf, 7, 0), -inf, 7, 1), W, put(put(G, inf, 0, 0), inf, 0, 1))
    check(X * 1e-33, W, G * 1e-33)           # everything below 2^-100
    check(X, W * 1e-33, G)
    check(torch.zeros_like(X), W, torch.zeros_like(G))


@pytest.mark.parametrize("B,T,n_in,n_out", [(3, 44, 256, 512), (5, 20, 1024, 128)])
@pytest.mark.parametrize("what", ["out", "X", "G"])
def test_short_samples_take_pointers_of_any_alignment(ops, B, T, n_in, n_out, what):  # noqa: F811
    """Fewer than 256 rows of short samples ran on the FMA kernels, which take any pointer; where their products are kept
    now, a pointer off 16 bytes goes where it went (a gradient slice through the operator, operands through the C interface)."""
    import ctypes
    from flashdp4review_b200 import _lib
    bf = torch.bfloat16

    def off(t):
        flat = torch.empty(t.numel() + 1, device=dev(), dtype=t.dtype)
        flat[1:] = t.flatten()
        return flat[1:].view(t.shape)
    X, G = _randn(B, T, n_in, seed=1, dtype=bf), _randn(B, T, n_out, seed=2, dtype=bf, scale=1e-1)
    want, norms, _ = ops.dp_linear_weight_grad(X, G, 1.0, 1.0, out_dtype=torch.float32, return_norms=True)
    assert _kept(lambda: ops.dp_linear_weight_grad(X, G, 1.0, 1.0))
    if what == "out":
        out = off(torch.zeros(n_out, n_in, device=dev()))
        ops.dp_linear_weight_grad(X, G, 1.0, 1.0, out=out)
    else:
        lib, algo = _lib.load(), _lib.FDP_KEEP_PRODUCTS | _lib.FDP_PAD_16BIT
        X, G = (off(X), G) if what == "X" else (X, off(G))
        out = torch.zeros(n_out, n_in, device=dev())
        ws = torch.empty(lib.fdp_linear_wgrad_workspace_bytes(B, T, n_in, n_out, _lib.FDP_BF16, algo), dtype=torch.uint8, device=dev())
        p = _lib.DPParams(1.0, 1.0, 0.0, 0, 0, 0, 0, 0, 0, 1)
        st = lib.fdp_linear_wgrad(G.data_ptr(), X.data_ptr(), out.data_ptr(), None, None, B, T, n_in, n_out, _lib.FDP_BF16, _lib.FDP_F32, 0,
                                  algo, ctypes.byref(p), ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
        assert st == 0
    assert float((out - want).norm()) < 2.0 ** -19 * float(want.norm())       # both in fp32, sums of at most 132 terms
