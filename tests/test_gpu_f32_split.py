"""The float32 products on tensor cores: the same bits however a tile's segments are shared; operands that are no finite numbers or whose
parts overflow; no wait that gave up."""
import pytest
import torch

from test_gpu_kernels import rand

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def K():
    from holon_b200.kernels import load_kernels
    k = load_kernels(torch.device(DEV))
    yield k
    k.lib.hb_gemm_f32_split(0)


def product(K, x, w, split=0):
    out = torch.full((x.shape[0], w.shape[0]), 7.0, device=DEV)
    K.lib.hb_gemm_f32_split(split)
    K.linear(out, x.to(DEV), w.to(DEV))
    assert K.tcgen05_status() == 0
    return out.cpu()


@pytest.mark.parametrize("m", [1, 16, 17, 95, 96, 97, 200])
@pytest.mark.parametrize("n,k", [(1, 1), (127, 64), (129, 65), (300, 512), (256, 513), (130, 1100), (128, 4096)])
def test_the_same_bits_however_segments_are_shared(K, m, n, k):
    x, w = rand(m, k, seed=m), rand(n, k, seed=n)
    outs = [product(K, x, w, split) for split in (1, 2, 4, 8, 0)]
    want = x.double() @ w.double().T
    assert torch.linalg.norm(outs[0] - want) <= 4e-7 * torch.linalg.norm(want)      # (each step's sum is cut off at 2^-23 of it)
    assert all(torch.equal(outs[0], o) for o in outs[1:])


@pytest.mark.parametrize("m", [3, 40])
@pytest.mark.parametrize("split", [0, 1, 8])
def test_operands_that_are_no_finite_numbers(K, m, split):
    x, w = rand(m, 700, seed=1), rand(200, 700, seed=2)
    clean = product(K, x, w, split)
    x[1, 5], x[1, 600], w[7, 9] = float("inf"), 3.0, float("nan")
    x[2, 650] = float("-inf")
    w[11, 5] = 0.0
    out = product(K, x, w, split)
    want = x.double() @ w.double().T
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isinf(), want.isinf())
    assert torch.equal(out[out.isinf()].double(), want[want.isinf()])
    w[11, 5] = rand(200, 700, seed=2)[11, 5]                                         # rows and columns without them keep their bits
    out, good = product(K, x, w, split), [i for i in range(200) if i != 7]
    assert torch.equal(out[0, good], clean[0, good]) and torch.equal(out[3:][:, good], clean[3:][:, good])


def test_numbers_whose_parts_overflow(K):
    """The nearest bfloat16 of the largest numbers is infinite; their products are not."""
    x, w = torch.zeros(5, 130), torch.zeros(130, 130)
    x[:, 3], x[2, 70] = 3.4e38, -3.4e38
    w[:, 3], w[:, 70] = 0.25, 0.125
    w[9, 3] = 8.0
    out, want = product(K, x, w), x.double() @ w.double().T
    assert out[:, 9].isinf().all() and out[:, 10:].isfinite().all()
    assert ((out - want)[:, 10:].abs() <= 2e-7 * want[:, 10:].abs()).all()
