"""The float32 engine's products and attention where their forms meet: rows around the limit between the kernel for few
rows and the tiles, k around its segments, tiles that a cluster shares; head sizes around the padded ones, rows of one
token beside rows of many."""
import math

import pytest
import torch

import ref_kernels
from test_gpu_kernels import on_device, paged_case, rand

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
REF = ref_kernels.RefKernels()


@pytest.fixture(scope="module")
def K():
    from holon_b200.kernels import load_kernels
    return load_kernels(torch.device(DEV))


# k: one segment, two, a remainder in the last of eight, segments of 64 and of 80, no multiple of 4; n: a cluster of eight, of four
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


@pytest.mark.parametrize("k", [4100, 6144])
def test_products_whose_stages_are_filled_again(K, k):
    """Few rows and columns with more pieces of k than the ring of the kernel for few rows has stages."""
    test_products_do_not_depend_on_the_kernel(K, 130, k)


@pytest.mark.parametrize("m", [3, 16, 17, 200])
@pytest.mark.parametrize("heads,n,k", [(5, 64, 36), (40, 130, 128), (3, 96, 30)])
def test_products_per_head_on_views(K, m, heads, n, k):
    x, w = rand(m, heads, k + 4, seed=m), rand(heads, n, k, seed=n)
    wide = torch.full((m, heads, n + 3), 7.0, device=DEV)
    K.linear_heads(wide[..., :n], x.to(DEV)[..., :k], w.to(DEV))
    want = torch.einsum("thk,hnk->thn", x[..., :k].double(), w.double())
    assert (wide[..., :n].cpu() - want).abs().max().item() <= 6e-8 * 8 * k
    assert (wide[..., n:] == 7.0).all()


# (heads, kv heads, head size, page): padded sizes and their neighbours, groups of 1 to 7, one size of the generic kernel
GEOMETRIES = [(3, 3, 4, 5), (4, 2, 64, 16), (7, 1, 68, 64), (5, 5, 128, 7), (8, 2, 128, 64), (2, 1, 132, 16), (4, 4, 256, 8), (6, 2, 30, 16)]
SPEC = [(0, 1), (31, 1), (300, 1), (0, 63), (0, 64), (5, 65), (200, 2), (70, 129)]


@pytest.mark.parametrize("geometry", GEOMETRIES)
@pytest.mark.parametrize("window", [0, 1, 33, 100])
@pytest.mark.parametrize("sink", [False, True])
def test_attention_float32(K, geometry, window, sink):
    heads, kv_heads, head_dim, page = geometry
    q, kv, table, rows = paged_case(heads, kv_heads, head_dim, page, SPEC, torch.float32, seed=head_dim + window)
    sinks = rand(heads, seed=9, scale=2.0) if sink else None
    scale = 1 / math.sqrt(head_dim)
    want = torch.empty_like(q, dtype=torch.float64)
    REF.paged_attention(want, q, kv, table, rows, scale, window, sinks)
    out = torch.full_like(q, float("nan"), device=DEV)
    K.paged_attention(out, q.to(DEV), kv.to(DEV), table.to(DEV), on_device(rows), scale, window, sinks.to(DEV) if sink else None)
    assert (out.cpu() - want).abs().max().item() <= 2e-5


@pytest.mark.parametrize("window", [0, 50])
def test_attention_float32_does_not_depend_on_the_cut(K, window):
    """The last 70 of 230 tokens computed at once, behind 160 and behind 193 others: the same bits for the tokens they share."""
    heads, kv_heads, head_dim, page = 4, 2, 128, 16
    q, kv, table, rows = paged_case(heads, kv_heads, head_dim, page, [(160, 70)], torch.float32, seed=3)
    outs = []
    for skip in (0, 33):
        from holon_b200.engine.batch import Rows
        n = 70 - skip
        qs = torch.tensor([0, n], dtype=torch.int32)
        part = Rows(rows.row_slot, qs, rows.kv_len, 1, n, 0, n, 230)
        out = torch.empty(n, heads, head_dim, device=DEV)
        K.paged_attention(out, q[skip:].contiguous().to(DEV), kv.to(DEV), table.to(DEV), on_device(part), 0.09, window)
        outs.append(out)
    assert torch.equal(outs[0][33:], outs[1])


@pytest.mark.parametrize("window", [0, 50])
def test_attention_float32_of_a_portion_of_one_token(K, window):
    """It runs as a one-token row does, with the keys in another order: the same up to rounding."""
    from holon_b200.engine.batch import Rows
    q, kv, table, rows = paged_case(4, 2, 128, 16, [(160, 70)], torch.float32, seed=3)
    outs = []
    for n in (70, 1):
        part = Rows(rows.row_slot, torch.tensor([0, n], dtype=torch.int32), rows.kv_len, 1, n, int(n == 1), n, 230)
        out = torch.empty(n, 4, 128, device=DEV)
        K.paged_attention(out, q[70 - n:].contiguous().to(DEV), kv.to(DEV), table.to(DEV), on_device(part), 0.09, window)
        outs.append(out)
    assert (outs[0][69] - outs[1][0]).abs().max().item() <= 2e-6


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_attention_float32_leaves_out_what_is_not_seen(K, bad):
    """Values of the last key that are no numbers reach the query that sees it and none before it."""
    heads, kv_heads, head_dim, page = 4, 2, 64, 16
    q, kv, table, rows = paged_case(heads, kv_heads, head_dim, page, [(20, 90), (0, 40)], torch.float32, seed=5)
    out = []
    for plant in (False, True):
        if plant:
            kv[table[rows.row_slot[0], 109 // page], 1, :, 109 % page] = bad
        o = torch.empty_like(q, device=DEV)
        K.paged_attention(o, q.to(DEV), kv.to(DEV), table.to(DEV), on_device(rows), 0.125, 0)
        out.append(o)
    assert torch.equal(out[0][:89], out[1][:89]) and torch.equal(out[0][90:], out[1][90:])
    assert not out[1][89].isfinite().any()


def plain_attention(q, kv, table, rows, scale, window):
    """In 64 bits, except that a score that overflows in 32 bits is minus infinity."""
    out = torch.zeros_like(q, dtype=torch.float64)
    group = q.shape[1] // kv.shape[2]
    for b in range(rows.n_rows):
        t0, n = int(rows.query_start[b]), int(rows.kv_len[b])
        j = torch.arange(n)
        k, v = (kv[table[rows.row_slot[b], j // kv.shape[3]].long(), i, :, j % kv.shape[3]].double() for i in (0, 1))
        for t in range(t0, int(rows.query_start[b + 1])):
            pos = n - int(rows.query_start[b + 1]) + t
            lo = max(0, pos - window + 1) if window else 0
            for h in range(q.shape[1]):
                s = k[lo:pos + 1, h // group] @ (q[t, h].double() * scale)
                out[t, h] = torch.softmax(s.float().double(), 0) @ v[lo:pos + 1, h // group]
    return out


@pytest.mark.parametrize("window", [0, 1, 2, 70])
def test_attention_float32_scores_of_minus_infinity(K, window):
    """Keys whose product with the query overflows weigh nothing, wherever they stand among a tile's or a group's keys; a query that
    sees no other key has no answer. (In 64 bits as in 32: the weights of the rest are not touched.)"""
    heads, kv_heads, head_dim, page = 4, 2, 64, 16
    spec = [(332, 1), (40, 1), (0, 200), (63, 5)]
    q, kv, table, rows = paged_case(heads, kv_heads, head_dim, page, spec, torch.float32, seed=11)
    q[..., 0] = 8.0
    for b, (before, new) in enumerate(spec):
        for j in (0, 5, 63, 64, 127, 199, 331, 332):
            if j < before + new:
                kv[table[rows.row_slot[b], j // page], 0, :, j % page, 0] = -3e38
    want = plain_attention(q, kv, table, rows, 1.0, window)
    assert window != 1 or want.isnan().any()
    out = torch.full_like(q, float("nan"), device=DEV)
    K.paged_attention(out, q.to(DEV), kv.to(DEV), table.to(DEV), on_device(rows), 1.0, window)
    assert torch.equal(out.isnan().cpu(), want.isnan())
    # scores of up to 30 in size are off by up to 2^-24 of that times a few roundings, and so are the weights
    assert (out.cpu() - want).nan_to_num().abs().max().item() <= 1e-4
