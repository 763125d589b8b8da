"""Which form of latent attention a step's portions take, and which kernel the experts' gated units, without a GPU (see test_kernel_choice_cpu)."""
import types

import pytest
import torch

from holon_b200.engine.batch import Rows
from test_kernel_choice_cpu import Noted

BF16 = torch.bfloat16


def table(**more):
    k = Noted()
    k.lib = types.SimpleNamespace(hb_latent_prompt_takes=lambda dim, rot, vdim, rank: int((dim, rot, vdim) in ((128, 64, 128), (64, 32, 64)) and rank % 16 == 0))
    k.expert_products, k.expert_tile_rows = "fast", 0
    for name, value in more.items():
        setattr(k, name, value)
    return k


def rows(new, lens, host=True):
    qs = [0]
    for n in new:
        qs.append(qs[-1] + n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32)                                # noqa: E731
    return Rows(i32(list(range(len(new)))), i32(qs), i32(lens), len(new), qs[-1], new.count(1), max(new), max(lens), qs if host else None, lens if host else None)


def expands(k, r, heads=16, dim=128, rot=64, vdim=128, rank=512, window=0, scale=0.1, tensors=()):
    return k.latent_expands(r, heads, dim, rot, vdim, rank, window, scale, *tensors)


def test_portions_whose_lengths_are_known():
    assert expands(table(), rows([2048], [2048])) and expands(table(), rows([1, 17, 300], [900, 17, 300]))
    assert not expands(table(), rows([1, 1], [40, 50]))                               # one-token rows alone
    assert not expands(table(), rows([2048], [2048], host=False))
    r = rows([2048], [2048])
    r.plan["any cut"] = True                                                           # a recorded step's rows may be cut otherwise
    assert not expands(table(), r)
    for other in (dict(prefill_attention="mma"), dict(attention_bf16="generic")):
        assert not expands(table(**other), rows([2048], [2048]))
    assert not expands(table(), rows([2048], [2048]), scale=-0.1)


@pytest.mark.parametrize("dim,rot,vdim,rank,takes", [(128, 64, 128, 512, True), (64, 32, 64, 80, True), (128, 64, 64, 512, False), (128, 32, 128, 512, False), (64, 32, 64, 72, False)])
def test_sizes(dim, rot, vdim, rank, takes):
    assert expands(table(), rows([300], [300]), dim=dim, rot=rot, vdim=vdim, rank=rank) == takes


def test_rows_seen_and_scratch():
    """Eight cache rows a new token (and a tile a request), of a window's only those from its first tile on, up to 512 MB of scratch."""
    assert expands(table(), rows([512], [4096])) and not expands(table(), rows([500], [4097 + 64]))
    assert expands(table(), rows([100], [100_000]), window=700) and not expands(table(), rows([100], [100_000]))
    k = table()
    assert k._latent_rows(rows([1, 100, 64], [500, 1000, 64]), 65) == 192 + 64        # keys 836 .. 999 in tiles from 832 on; 0 .. 63
    assert k._latent_rows(rows([1, 100, 63], [500, 1000, 63]), 0) == 1024 + 64
    assert expands(table(), rows([30_000], [30_000])) and not expands(table(), rows([70_000], [70_000]), heads=32)


def test_the_account_covers_what_portions_may_take():
    """Whatever portions of a step's tokens see: where they take the form that makes keys and values, its scratch is in the account."""
    import random
    k, rng, most = table(), random.Random(7), 0
    heads, dim, rot, vdim, rank = 16, 128, 64, 128, 512
    for _ in range(400):
        tokens, seqs, longest = rng.choice([64, 512, 4096]), rng.choice([1, 3, 16]), rng.choice([300, 2048, 8192])
        new, left = [], tokens
        while left > 1 and len(new) < seqs:
            new.append(min(left, longest, max(2, left if rng.random() < 0.3 else rng.randrange(2, left + 1))))
            left -= new[-1]
        lens = [min(longest, n + int(rng.choice([0, 1, 7, 9]) * n * rng.random() * 1.2)) for n in new]
        r, window = rows(new, lens), rng.choice([0, 0, 100])
        if expands(k, r, window=window):
            taken = 2 * k._latent_rows(r, window) * (heads * (dim + vdim) + rank + rot)
            bound = k.latent_scratch(tokens, seqs, longest, heads, dim, rot, vdim, rank)
            assert taken <= bound <= k.LATENT_SCRATCH
            most = max(most, taken / bound)
    assert most > 0.9
    assert k.latent_scratch(512, 2, 4096, heads, dim, 32, vdim, rank) == 0            # (sizes that keep the folded form)


def test_tensors_that_do_not_fit_sixteen_bytes():
    wide = torch.zeros(64, 40, dtype=BF16)
    assert expands(table(), rows([300], [300]), tensors=(wide, wide[:, :16]))
    for other in (wide.float(), wide[:, 1:], torch.zeros(64, 36, dtype=BF16)):
        assert not expands(table(), rows([300], [300]), tensors=(wide, other))


@pytest.mark.parametrize("per,products,experts,inter,kernel", [
    (96, "fast", 4, 16, "hb_expert_swiglu_tcgen05"), (95, "fast", 4, 16, None), (1, "tcgen05", 4, 16, "hb_expert_swiglu_tcgen05"), (200, "mma", 4, 16, None),
    (200, "generic", 4, 16, None), (200, "fast", 4, 12, None), (96, "fast", 1024, 8, "hb_expert_swiglu_tcgen05"), (96, "fast", 1025, 8, None)])
def test_gated_units_of_experts(per, products, experts, inter, kernel):
    k, n = table(expert_products=products), per * experts
    k._check = lambda *tensors: None
    i32, wide = torch.zeros(experts + 1, dtype=torch.int32), lambda *s: torch.zeros(1, dtype=BF16).expand(*s)     # noqa: E731
    k.expert_swiglu(torch.empty(n, inter, dtype=BF16), wide(n, 16), None, wide(experts, 2 * inter, 16), i32)
    assert (k.called[0] == kernel) if kernel else ("hb_expert_swiglu_tcgen05" not in k.called and k.called[-1] == "hb_silu_mul")
