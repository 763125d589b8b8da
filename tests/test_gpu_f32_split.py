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


def bound(x, w):
    """Of multiply-adds in up to eight segments and their sums: 2^-24 of the terms' sizes each; and half of the smallest number a term."""
    k = x.shape[1]
    return (k / 8 + 72) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + k * 2.0 ** -149


@pytest.mark.parametrize("m", [2, 16, 40, 130])
@pytest.mark.parametrize("split", [0, 1, 8])
@pytest.mark.parametrize("k,small,large", [(130, -112, 100), (700, -118, 110), (700, -126, 0), (513, -140, 120), (64, -105, 90), (300, -105, -40), (1100, -70, -75)])
def test_numbers_whose_parts_lie_below_the_smallest_bfloat16(K, m, split, k, small, large):
    """Small operands against large ones, on either side, alone or beside numbers of ordinary size."""
    x, w = rand(m, k, seed=3) * 2.0 ** small, rand(200, k, seed=4) * 2.0 ** large
    x[1, 5] = 0.0
    if m > 2:
        x[2, ::3] = rand(1, len(x[2, ::3]), seed=5)[0] * 2.0 ** (small + 3)
    for a, b in ((x, w), (rand(m, k, seed=6) * 2.0 ** large, rand(200, k, seed=7) * 2.0 ** small)):
        out, want = product(K, a, b, split), a.double() @ b.double().T
        assert ((out - want).abs() <= bound(a, b)).all()


@pytest.mark.parametrize("m", [3, 40])
def test_whether_an_element_is_made_again_does_not_depend_on_its_neighbours(K, m):
    x, w = rand(m, 700, seed=1), rand(200, 700, seed=2)
    clean = product(K, x, w)
    x[1], w[7] = x[1] * 2.0 ** 100, w[7] * 2.0 ** -120
    x[2] = 0.0
    out, rows, good = product(K, x, w), [i for i in range(m) if i not in (1, 2)], [i for i in range(200) if i != 7]
    assert torch.equal(out[rows][:, good], clean[rows][:, good]) and not out[2].any()
    want = x.double() @ w.double().T
    assert ((out - want).abs() <= bound(x, w)).all()
    x[1] = 2.0 ** -130                                                                # (a row of the smallest numbers beside ordinary ones)
    out = product(K, x, w)
    assert torch.equal(out[rows][:, good], clean[rows][:, good])
    assert ((out - x.double() @ w.double().T).abs() <= bound(x, w)).all()


@pytest.mark.parametrize("m", [2, 60])
def test_rows_of_zeros_stay_zero(K, m):
    x, w = rand(m, 300, seed=1), rand(200, 300, seed=2)
    clean = product(K, x, w)
    w[5::7] = 0.0
    out = product(K, x, w)
    assert not out[:, 5::7].any() and torch.equal(out[:, ::7], clean[:, ::7])
    x[0] = 0.0
    assert not product(K, x, w)[0].any()
    one = torch.zeros(m, 300)
    one[:, 9] = 2.0
    assert torch.equal(product(K, one, w), (2.0 * w[:, 9]).expand(m, 200))             # (products of zeros with other numbers)
