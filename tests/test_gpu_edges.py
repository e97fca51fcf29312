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
