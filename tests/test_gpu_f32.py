"""The float32 engine's products where their forms meet: rows around the limit between the kernel for few rows and the
tiles, k around its segments, tiles that a cluster shares."""
import math

import pytest
import torch

from test_gpu_kernels import rand

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def K():
    from holon_b200.kernels import load_kernels
    return load_kernels(torch.device(DEV))


# k: one segment, a remainder in the last of eight, segments of 64 + 16, no multiple of 4; n: a cluster of eight, of four
# and no cluster at 65 rows (1, 33 to 120 and more tiles of 64 x 128)
@pytest.mark.parametrize("k", [4, 16, 60, 128, 132, 636, 1030, 3072])
@pytest.mark.parametrize("n", [7, 130, 2200, 9000])
def test_products_do_not_depend_on_the_kernel(K, n, k):
    x, w = rand(130, k, seed=n), rand(n, k, seed=k)
    xd, wd = x.to(DEV), w.to(DEV)
    want = x.double() @ w.double().T
    whole = None
    for m in (130, 65, 64, 17, 16, 9, 8, 5, 4, 1):
        out = torch.full((m, n), float("nan"), device=DEV)
        K.linear(out, xd[:m], wd)
        if whole is None:
            whole = out
            # every step of a sum rounds by at most half a unit in 2^24 of the partial sum; sqrt(k) of them add up at random
            assert (out.cpu() - want).abs().max().item() <= 6e-8 * 8 * math.sqrt(k) * math.sqrt(k)
            assert torch.linalg.norm(out.cpu() - want) <= 1e-6 * torch.linalg.norm(want)
        assert torch.equal(out, whole[:m]), m


@pytest.mark.parametrize("m", [3, 16, 17, 200])
@pytest.mark.parametrize("heads,n,k", [(5, 64, 36), (40, 130, 128), (3, 96, 30)])
def test_products_per_head_on_views(K, m, heads, n, k):
    x, w = rand(m, heads, k + 4, seed=m), rand(heads, n, k, seed=n)
    wide = torch.full((m, heads, n + 3), 7.0, device=DEV)
    K.linear_heads(wide[..., :n], x.to(DEV)[..., :k], w.to(DEV))
    want = torch.einsum("thk,hnk->thn", x[..., :k].double(), w.double())
    assert (wide[..., :n].cpu() - want).abs().max().item() <= 6e-8 * 8 * k
    assert (wide[..., n:] == 7.0).all()
