"""The experts' products for prompts at the edges of their tiles: experts without rows, of one row, around the multiples of 32 that a tile
is wide and around the 256 rows that one holds; columns that end inside a lane's block, inside the second accumulator and behind it; fewer
tiles than pairs of CTAs and more."""
import pytest
import torch

from ref_kernels import RefKernels
from test_gpu_kernels import close, rand

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
REF = RefKernels()
COUNTS = [0, 1, 31, 0, 32, 33, 255, 256, 257, 300, 513, 97, 0]


@pytest.fixture(scope="module")
def K():
    from holon_b200.kernels import load_kernels
    k = load_kernels(torch.device(DEV))
    k.expert_products = "tcgen05"
    return k


def case(counts, n, k, gather):
    rows = sum(counts)
    starts = torch.tensor([0] + counts, dtype=torch.int32).cumsum(0).to(torch.int32)
    tokens = max(1, rows // 3)
    token_of = torch.randint(0, tokens, (rows,), generator=torch.Generator().manual_seed(n)).to(torch.int32) if gather else None
    x = rand(tokens if gather else rows, k, dtype=torch.bfloat16, seed=1)
    return rows, starts, token_of, x, rand(len(counts), n, k, dtype=torch.bfloat16, seed=2, scale=k ** -0.5)


@pytest.mark.parametrize("counts", [COUNTS, [700], [5, 0, 9] * 60])
@pytest.mark.parametrize("n,k", [(8, 64), (136, 72), (392, 200), (512, 64), (520, 320), (1288, 136)])
@pytest.mark.parametrize("gather,act", [(False, 0), (True, 1)])
def test_products(K, counts, n, k, gather, act):
    rows, starts, token_of, x, w = case(counts, n, k, gather)
    out, want = torch.full((rows, n), 7.0, dtype=torch.bfloat16, device=DEV), torch.empty(rows, n, dtype=torch.bfloat16)
    K.expert_linear(out, x.to(DEV), token_of.to(DEV) if gather else None, w.to(DEV), starts.to(DEV), act)
    REF.expert_linear(want, x, token_of, w, starts, act)
    assert K.tcgen05_status() == 0
    close(out, want, torch.bfloat16, scale=4.0)                      # (results of up to about 4, squares of up to 16, rounded to bfloat16)


@pytest.mark.parametrize("counts", [COUNTS, [5, 0, 9] * 60])
@pytest.mark.parametrize("inter,k", [(8, 64), (136, 72), (256, 64), (264, 328), (776, 136)])
@pytest.mark.parametrize("gather,scaled", [(False, False), (True, True)])
def test_clamped_units(K, counts, inter, k, gather, scaled):
    rows, starts, token_of, x, w = case(counts, 2 * inter, k, gather)
    scale = rand(rows, seed=5).abs() if scaled else None
    out, want = torch.full((rows, inter), 7.0, dtype=torch.bfloat16, device=DEV), torch.empty(rows, inter, dtype=torch.bfloat16)
    K.expert_glu(out, x.to(DEV), token_of.to(DEV) if gather else None, w.to(DEV), starts.to(DEV), 1.5, 1.702, scale.to(DEV) if scaled else None)
    REF.expert_glu(want, x, token_of, w, starts, 1.5, 1.702, scale)
    assert K.tcgen05_status() == 0
    close(out, want, torch.bfloat16, scale=2.0)                      # (limits keep the unit's results below 4)


def test_more_experts_than_the_kernel_counts(K):
    """1,025 experts stay with the other kernels."""
    counts = [1] * 1025
    rows, starts, _, x, w = case(counts, 8, 16, False)
    out, want = torch.full((rows, 8), 7.0, dtype=torch.bfloat16, device=DEV), torch.empty(rows, 8, dtype=torch.bfloat16)
    for products in ("tcgen05", "fast"):
        K.expert_products = products
        K.expert_linear(out, x.to(DEV), None, w.to(DEV), starts.to(DEV), 0)
        REF.expert_linear(want, x, None, w, starts, 0)
        close(out, want, torch.bfloat16, scale=2.0)
    K.expert_products = "tcgen05"


@pytest.mark.parametrize("clamped", [False, True])
def test_gates_far_below_zero(K, clamped):
    """silu(-88) is -5.3e-37: no zero, although what it is divided by is beyond 2^126."""
    rows, k, inter = 300, 64, 8
    x, w = torch.zeros(rows, k, dtype=torch.bfloat16), torch.zeros(1, 2 * inter, k, dtype=torch.bfloat16)
    x[:, 3], w[0, :inter, 3], w[0, inter:, 3] = 1.0, torch.linspace(-88.5, -86.5, inter), 2.0
    starts, out = torch.tensor([0, rows], dtype=torch.int32), torch.empty(rows, inter, dtype=torch.bfloat16, device=DEV)
    if clamped:
        K.expert_glu(out, x.to(DEV), None, w.to(DEV), starts.to(DEV), 100.0, 1.0, None)
    else:
        K.expert_swiglu(out, x.to(DEV), None, w.to(DEV), starts.to(DEV))
    gate, up = w[0, :inter, 3].double(), 2.0
    want = (gate * torch.sigmoid(gate) * (up + 1.0 if clamped else up)).expand(rows, inter)
    assert ((out.cpu().double() - want).abs() <= 2.0 ** -8 * want.abs()).all()           # (a bfloat16 rounding, and 88 log2(e) to 2^-17)


@pytest.mark.parametrize("act", [1, 2, 3])
@pytest.mark.parametrize("n,k", [(136, 72), (520, 320)])
def test_activations(K, act, n, k):
    """Each that experts may have (parts/experts.py: EXPERT_ACTIVATIONS), as the kernels for fewer rows apply it."""
    rows, starts, _, x, w = case(COUNTS, n, k, False)
    out, want = torch.full((rows, n), 7.0, dtype=torch.bfloat16, device=DEV), torch.empty(rows, n, dtype=torch.bfloat16)
    K.expert_linear(out, x.to(DEV), None, w.to(DEV), starts.to(DEV), act)
    REF.expert_linear(want, x, None, w, starts, act)
    close(out, want, torch.bfloat16, scale=4.0)
    K.expert_products = "mma"
    other = torch.empty_like(out)
    K.expert_linear(other, x.to(DEV), None, w.to(DEV), starts.to(DEV), act)
    K.expert_products = "tcgen05"
    close(out, other.cpu(), torch.bfloat16, scale=4.0)
