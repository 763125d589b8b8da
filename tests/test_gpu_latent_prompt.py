"""Latent attention of prompt portions with every head's keys and values made first: rows that end inside tiles of 64 keys and 128 and
256 queries, contexts, windows whose first tile is not the cache's, both head sizes, one-token rows beside them; and the part that chooses
between this form and the folded one."""
import pytest
import torch

from test_gpu_kernels import close, on_device, rand
from holon_b200.engine.batch import Rows

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def K():
    from holon_b200.kernels import load_kernels
    return load_kernels(torch.device(DEV))


def case(heads, dim, rank, page, new, lens, seed=1):
    rot, dk = dim // 2, rank + dim // 2
    need = [-(-n // page) for n in lens]
    pages = sum(need) + 1
    cache = rand(pages, page, dk, dtype=torch.bfloat16, seed=seed)
    order = torch.randperm(pages - 1, generator=torch.Generator().manual_seed(3)).tolist()
    table = torch.full((len(lens), max(need) + 1), pages - 1, dtype=torch.int32)
    at = 0
    for b, n in enumerate(need):
        table[b, :n] = torch.tensor(order[at:at + n], dtype=torch.int32)
        at += n
        if lens[b] % page:                                        # what lies behind a row's end is no number
            cache[table[b, n - 1], lens[b] % page:] = float("nan")
    qs = torch.tensor([0] + new, dtype=torch.int32).cumsum(0).to(torch.int32)
    t, ones = int(qs[-1]), sum(n == 1 for n in new)
    rows = Rows(torch.arange(len(new), dtype=torch.int32), qs, torch.tensor(lens, dtype=torch.int32), len(new), t, ones, max(new), max(lens),
                qs.numpy(), torch.tensor(lens).numpy())
    first = rand(t, heads * 3 * rot + 24, dtype=torch.bfloat16, seed=seed + 1, scale=2.0)
    qa = torch.full((t, heads, dk), float("nan"), dtype=torch.bfloat16)
    qa[:, :, rank:] = rand(t, heads, rot, dtype=torch.bfloat16, seed=seed + 2, scale=2.0)
    weight = rand(heads * 2 * dim, rank, dtype=torch.bfloat16, seed=seed + 3, scale=rank ** -0.5)
    return first, qa, cache, table, rows, weight


def plain(first, qa, cache, table, rows, weight, heads, dim, rank, scale, window, sinks):
    """In 64 bits, keys and values rounded to bfloat16 once as the engine keeps them."""
    t, rot, page = qa.shape[0], dim // 2, cache.shape[1]
    out = torch.zeros(t, heads, dim, dtype=torch.float64)
    q = torch.cat((first[:, :heads * (dim + rot)].view(t, heads, dim + rot)[:, :, :dim], qa[:, :, rank:]), -1).double()
    for b in range(rows.n_decode, rows.n_rows):
        s, e, n = int(rows.query_start[b]), int(rows.query_start[b + 1]), int(rows.kv_len[b])
        j = torch.arange(n)
        lat = cache[table[b, j // page].long(), j % page]
        made = (lat[:, :rank].double() @ weight.double().T).bfloat16().double().view(n, 2, heads, dim)
        k = torch.cat((made[:, 0], lat[:, None, rank:].double().expand(n, heads, rot)), -1)
        score = torch.einsum("qhd,khd->hqk", q[s:e], k) * scale
        i = torch.arange(n - (e - s), n)[:, None]
        score = score.masked_fill((j > i) | ((i - j >= window) if window else (j < 0)), float("-inf"))
        if sinks is not None:
            score = torch.cat((score, sinks.double()[:, None, None].expand(-1, e - s, 1)), -1)
        out[s:e] = torch.einsum("hqk,khd->qhd", score.softmax(-1)[..., :n], made[:, 1])
    return out


def attend(K, c, heads, dim, rank, scale, window, sinks, tile=None):
    first, qa, cache, table, rows, weight = (x.to(DEV) if torch.is_tensor(x) else on_device(x) for x in c)
    rows.host_query_start, rows.host_kv_len = c[4].host_query_start, c[4].host_kv_len
    out = torch.full((qa.shape[0], heads, dim), 7.0, dtype=torch.bfloat16, device=DEV)
    q = first[:, :heads * 3 * dim // 2]
    assert K.latent_expands(rows, heads, dim, dim // 2, dim, rank, window, scale, q, qa, out, cache, weight)
    K.prefill_tile = tile
    K.latent_prompt(out, q, qa, cache, table, rows, scale, weight, dim, dim, rank, window, None if sinks is None else sinks.to(DEV))
    K.prefill_tile = None
    assert K.tcgen05_status() == 0
    return out.cpu()


NEW, LENS = [1, 2, 63, 129, 70, 300, 257], [70, 2, 63, 129, 290, 300, 641]


@pytest.mark.parametrize("heads,dim,rank,page", [(3, 128, 512, 64), (16, 128, 64, 128), (5, 64, 256, 64), (1, 64, 80, 16)])
@pytest.mark.parametrize("window", [0, 1, 65, 200])
@pytest.mark.parametrize("sink", [False, True])
@pytest.mark.parametrize("tile", [128, 256])
def test_portions(K, heads, dim, rank, page, window, sink, tile):
    c = case(heads, dim, rank, page, NEW, LENS)
    sinks = rand(heads, seed=4, scale=3.0) if sink else None
    scale = (1.5 * dim) ** -0.5
    want = plain(*c, heads, dim, rank, scale, window, sinks)
    out = attend(K, c, heads, dim, rank, scale, window, sinks, tile)
    assert (out[0] == 7.0).all()                                   # the one-token row is not this kernel's
    # weights, outputs and, by another order of summation, a few keys and values are rounded to bfloat16 (2^-9 of values up to about 4)
    close(out[1:], want[1:].float(), torch.bfloat16, scale=2.0)


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("column", [0, 500, 560])
def test_what_is_no_number_stays_none(K, bad, column):
    """A cached number that is none, in one row's context: that row's queries have no answer, the other rows keep their bits."""
    c = case(4, 128, 512, 64, [70, 5, 40], [170, 8, 40])
    c[1][..., 512:] = c[1][..., 512:].abs() + 1.0                  # (an infinity then scores one: a weight without bounds)
    clean = attend(K, c, 4, 128, 512, 0.07, 0, None)
    c[2][c[3][0, 0], 10, column] = bad
    out = attend(K, c, 4, 128, 512, 0.07, 0, None)
    assert out[:70].isnan().all() and clean.isfinite().all() and torch.equal(out[70:], clean[70:])


def test_a_page_that_the_table_does_not_name(K):
    """Reads as rows of zeros."""
    c = case(4, 64, 256, 64, [70, 50], [130, 70])
    c[2][c[3][0, 0]] = 0
    want = attend(K, c, 4, 64, 256, 0.1, 0, None)
    for nowhere in (-1, c[2].shape[0], 1 << 30):
        c[3][0, 0] = nowhere
        assert torch.equal(attend(K, c, 4, 64, 256, 0.1, 0, None), want), nowhere


@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("own_query_latent", [False, True])
def test_the_part_gives_the_same_either_way(K, window, own_query_latent):
    """A step of one-token rows and portions through the part, with keys and values made and with folded queries."""
    from holon_b200.config.spec import PartRef
    from holon_b200.parts.base import BuildContext
    from holon_b200.parts.latent import LatentAttention
    from holon_b200.parts.model import LayerCache
    from holon_b200.engine.batch import GroupStep
    import types
    heads, dim, rot, rank, hidden = 4, 128, 64, 512, 256
    new, lens = [1, 1, 90, 300], [50, 129, 90, 350]
    ctx = BuildContext(torch.device(DEV), torch.bfloat16, K, max_positions=512, max_step_tokens=512)
    part = LatentAttention(ctx, heads=heads, dim=dim, rot_dim=rot, vdim=dim, rank=rank, scale=192 ** -0.5, hidden=hidden, norm=PartRef.of("norm", "rmsnorm", eps=1e-6),
                           position=None, window=window, q_rank=96 if own_query_latent else None, sink=True)
    for i, (name, p) in enumerate(part.params()):
        p.tensor = (rand(*p.shape, seed=i) * (p.shape[-1] ** -0.5 if len(p.shape) > 1 else 1.0)).to(torch.float32 if p.kind == "coef" else torch.bfloat16).to(DEV)
    part.finalize()
    pages, qs = 40, torch.tensor([0] + new, dtype=torch.int32).cumsum(0).to(torch.int32)
    table = torch.arange(24, dtype=torch.int32).view(4, 6)
    write = torch.cat([table[b, torch.arange(n - a, n) // 64] * 64 + torch.arange(n - a, n) % 64 for b, (a, n) in enumerate(zip(new, lens))]).to(torch.int32)
    rows = on_device(Rows(torch.arange(4, dtype=torch.int32), qs, torch.tensor(lens, dtype=torch.int32), 4, sum(new), 2, 300, 350))
    rows.host_query_start, rows.host_kv_len = qs.numpy(), torch.tensor(lens).numpy()
    kept = rand(pages, 64, rank + rot, dtype=torch.bfloat16, seed=77).to(DEV)
    x = rand(sum(new), hidden, dtype=torch.bfloat16, seed=78).to(DEV)
    outs = []
    for way in ("tcgen05", "mma"):
        K.prefill_attention = way
        step = types.SimpleNamespace(rows=rows, positions=torch.zeros(sum(new), dtype=torch.int32, device=DEV))
        outs.append(part.forward(x, step, LayerCache(kept.clone(), GroupStep(table.to(DEV), write.to(DEV), 64), True, {})).float())
    K.prefill_attention = "tcgen05"
    assert torch.equal(outs[0][:2], outs[1][:2])                   # one-token rows: the same kernel
    # folded queries and mixed latents on one side, keys and values on the other are rounded to bfloat16, 2^-9 each
    assert torch.linalg.norm(outs[0] - outs[1]) <= 4 * 2 ** -9 * torch.linalg.norm(outs[1])
