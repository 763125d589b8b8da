"""Latent attention of prompt portions on tcgen05: ranks whose output fits tensor memory once and ranks that two CTAs share,
tiles that end inside a token's heads, rows that end inside a cache tile whose other rows hold no numbers."""
import pytest
import torch

from ref_kernels import RefKernels
from test_gpu_kernels import close, on_device, rand
from holon_b200.engine.batch import Rows

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
REF = RefKernels()


@pytest.fixture(scope="module")
def K():
    from holon_b200.kernels import load_kernels
    return load_kernels(torch.device(DEV))


SIZES = [(16, 512, 64, 64), (1, 512, 64, 64), (40, 256, 32, 64), (3, 64, 16, 128), (5, 384, 32, 64), (7, 128, 80, 64), (130, 192, 64, 64)]


@pytest.mark.parametrize("heads,rank,rot,page", SIZES)
@pytest.mark.parametrize("window", [0, 1, 65, 200])
@pytest.mark.parametrize("sink", [False, True])
def test_portions(K, heads, rank, rot, page, window, sink):
    new, lens = [1, 2, 37, 64, 129, 9, 130], [70, 2, 300, 64, 129, 641, 193]
    dk = rank + rot
    need = [-(-n // page) for n in lens]
    pages = sum(need) + 2
    cache = rand(pages, page, dk, dtype=torch.bfloat16, seed=rank)
    order = torch.randperm(pages - 1, generator=torch.Generator().manual_seed(3)).tolist()
    table = torch.full((len(lens), max(need) + 1), pages - 1, dtype=torch.int32)
    at = 0
    for b, n in enumerate(need):
        table[b, :n] = torch.tensor(order[at:at + n], dtype=torch.int32)
        at += n
        if lens[b] % page:                                        # what lies behind a row's end is no number
            cache[table[b, n - 1], lens[b] % page:] = float("nan")
    qs = torch.tensor([0] + new, dtype=torch.int32).cumsum(0).to(torch.int32)
    t = int(qs[-1])
    host = Rows(torch.arange(len(new), dtype=torch.int32), qs, torch.tensor(lens, dtype=torch.int32), len(new), t, 1, max(new), max(lens))
    qa = rand(t, heads, dk, dtype=torch.bfloat16, seed=9, scale=3.0)
    sinks = rand(heads, seed=4, scale=3.0) if sink else None
    scale = dk ** -0.5
    want = torch.empty(t, heads, rank)
    REF.latent_attention(want, qa, cache, table, host, scale, rank, window, sinks=sinks)
    out = torch.full((t, heads, rank), float("nan"), dtype=torch.bfloat16, device=DEV)
    assert K._latent_tcgen05_takes(heads, rank, rot, pages, page)
    K.latent_attention(out, qa.to(DEV), cache.to(DEV), table.to(DEV), on_device(host), scale, rank, window, sinks=None if sink is False else sinks.to(DEV))
    assert K.tcgen05_status() == 0
    # a weight and an output are rounded to bfloat16 once each (2^-9 of values up to about 4)
    close(out, want, torch.bfloat16, scale=2.0)


def test_sizes_that_stay_with_the_other_kernel(K):
    for heads, rank, rot, pages, page in [(4, 80, 16, 9, 64), (4, 512, 0, 9, 64), (4, 320, 32, 9, 64), (4, 64, 32, 9, 32), (4, 512, 256, 9, 64)]:
        assert not K._latent_tcgen05_takes(heads, rank, rot, pages, page)


def small_case(heads=16, rank=512, rot=64, page=64):
    new, lens, dk = [70, 5, 40], [170, 133, 40], rank + rot
    cache = rand(9, page, dk, dtype=torch.bfloat16, seed=1)
    table = torch.tensor([[3, 1, 6], [0, 4, 7], [5, 8, 8]], dtype=torch.int32)
    qs = torch.tensor([0] + new, dtype=torch.int32).cumsum(0).to(torch.int32)
    host = Rows(torch.arange(3, dtype=torch.int32), qs, torch.tensor(lens, dtype=torch.int32), 3, sum(new), 0, max(new), max(lens))
    return rand(sum(new), heads, dk, dtype=torch.bfloat16, seed=2, scale=3.0), cache, table, host


def latent(K, qa, cache, table, host, rank=512, scale=0.04, window=0, sinks=None):
    out = torch.full((qa.shape[0], qa.shape[1], rank), 7.0, dtype=torch.bfloat16, device=DEV)
    assert K._latent_tcgen05_takes(qa.shape[1], rank, qa.shape[2] - rank, cache.shape[0], cache.shape[1])
    K.latent_attention(out, qa.to(DEV), cache.to(DEV), table.to(DEV), on_device(host), scale, rank, window, sinks=sinks)
    assert K.tcgen05_status() == 0
    return out.cpu()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("column", [0, 300, 560])
@pytest.mark.parametrize("sink", [False, True])
def test_what_is_no_number_stays_none(K, bad, column, sink):
    """A cached number of the second row's context that is none: every query of that row sees it and has no answer (and not zeros);
    the other rows keep their bits."""
    qa, cache, table, host = small_case()
    qa[..., column] = qa[..., column].abs() + 1.0                     # (an infinity then scores one: a weight without bounds)
    sinks = rand(16, seed=5).to(DEV) if sink else None
    clean = latent(K, qa, cache, table, host, sinks=sinks)
    cache[4, 10, column] = bad
    out = latent(K, qa, cache, table, host, sinks=sinks)
    assert out[70:75].isnan().all() and clean.isfinite().all()
    assert torch.equal(out[:70], clean[:70]) and torch.equal(out[75:], clean[75:])


def test_a_page_that_the_table_does_not_name(K):
    """Reads as rows of zeros, as in the other kernel."""
    qa, cache, table, host = small_case()
    cache[8] = 0
    table[1, 0] = 8
    want = latent(K, qa, cache, table, host)
    for nowhere in (-1, 9, 1 << 30):
        table[1, 0] = nowhere
        assert torch.equal(latent(K, qa, cache, table, host), want), nowhere
