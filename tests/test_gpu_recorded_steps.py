"""`Runner.step` records steps of one-token rows that come again: the same logits as when they ran kernel by kernel, whatever changes
between the steps of a kind, and no recording where a part cannot be captured."""
import pytest
import torch

from holon_b200.engine import StepEntry, build
from holon_b200.weights import RandomSource

pytestmark = pytest.mark.gpu
CONFIG = dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=2, hidden_size=128, num_attention_heads=4, num_key_value_heads=2, head_dim=32,
              intermediate_size=192, vocab_size=331, rope_theta=10000.0, rms_norm_eps=1e-6, tie_word_embeddings=False)


def made(dtype="bfloat16", graphs=True):
    with torch.inference_mode():
        return build(RandomSource(CONFIG, seed=5, device="cuda:0", dtype=getattr(torch, dtype)), dtype=dtype, device="cuda:0", page_size=16, max_seqs=4,
                     max_model_len=1024, max_step_tokens=1024, pages=160, cuda_graphs=graphs)


def trace(built, lengths, steps, seed=1, between=None):
    g = torch.Generator().manual_seed(seed)
    ids = [torch.randint(0, 331, (n + steps,), generator=g).tolist() for n in lengths]
    out, cache = [], built.cache
    with torch.inference_mode():
        slots = [cache.admit() for _ in ids]
        for s in range(steps + 1):
            entries = []
            for slot, tokens, n in zip(slots, ids, lengths):
                new, at = (tokens[:n], 0) if s == 0 else (tokens[n + s - 1:n + s], n + s - 1)
                assert cache.reserve(slot, at + len(new))
                entries.append(StepEntry(slot, new, at, [len(new) - 1]))
            out.append(built.runner.step(entries))
            if between:
                between(s)
        for slot in slots:
            cache.release(slot)
    return out


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_the_same_logits_as_kernel_by_kernel(dtype):
    """Rows that pass 512 keys change the plan and so the recording; results that were handed out stay as they were."""
    built = made(dtype)
    first = trace(built, [509, 3, 40], 7)
    kept = [x.clone() for x in first]
    again = trace(built, [509, 3, 40], 7)
    assert 0 < sum(r is not None for r in built.runner._recorded.values()) <= 2
    other = trace(built, [20, 77, 5], 4, seed=2)
    assert all(torch.equal(a, b) for a, b in zip(first, kept)) and all(torch.equal(a, b) for a, b in zip(first, again))
    plain = made(dtype, graphs=False)
    assert not plain.runner._use_graphs
    # (keys are cut for the longest row's power of two in place of its length: another order of summation)
    for a, b in zip(first + other, trace(plain, [509, 3, 40], 7) + trace(plain, [20, 77, 5], 4, seed=2)):
        assert torch.linalg.norm(a - b) <= (1e-5 if dtype == "float32" else 2e-2) * torch.linalg.norm(b)


def test_what_changes_between_steps_is_seen():
    """Another weight, another switch of the kernel table: a recording of their own."""
    built, plain = made(), made(graphs=False)
    trace(built, [9, 30], 5)
    for b in (built, plain):
        p = next(p for n, p in b.model.params() if "down_proj" in n)
        p.tensor = p.tensor * 3.0
    b = trace(plain, [9, 30], 5)
    for a in (trace(built, [9, 30], 5), trace(built, [9, 30], 5)):
        assert all(torch.linalg.norm(x - y) <= 2e-2 * torch.linalg.norm(y) for x, y in zip(a, b))
    built.ctx.kernels.fused_norm = False
    a = trace(built, [9, 30], 5)
    built.ctx.kernels.fused_norm = True
    assert all(torch.linalg.norm(x - y) <= 2e-2 * torch.linalg.norm(y) for x, y in zip(a, b))
    assert len(built.runner._recorded) >= 3


def test_few_recordings_are_kept_and_other_steps_run_as_they_are():
    built = made()
    built.runner.GRAPHS = 2
    for rows in (1, 2, 3, 4):
        trace(built, [5] * rows, 3)
    assert len(built.runner._recorded) <= 2
    cache = built.cache
    with torch.inference_mode():
        slot = cache.admit()
        cache.reserve(slot, 40)
        before = dict(built.runner._recorded)
        assert built.runner.step([StepEntry(slot, [3], 0, [])]) is None              # nothing wanted
        assert built.runner.step([StepEntry(slot, [4, 5, 6], 1, [0, 2])]).shape == (2, 331)
        cache.release(slot)
    assert built.runner._recorded == before


def test_a_part_that_cannot_be_captured():
    """A part that reads a result on the host runs as it always did."""
    built, plain = made(), made(graphs=False)
    forward, seen = built.model.head.forward, []
    built.model.head.forward = lambda rows: (seen.append(float(rows.float().sum().item())), forward(rows))[1]
    a, b = trace(built, [9, 30], 6), trace(plain, [9, 30], 6)
    assert not built.runner._use_graphs and len(seen) >= 7
    assert all(torch.linalg.norm(x - y) <= 2e-2 * torch.linalg.norm(y) for x, y in zip(a, b))
