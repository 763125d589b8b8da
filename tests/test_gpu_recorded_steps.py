"""`Runner.step` records steps of one-token rows that come again: the same logits as when they ran kernel by kernel, whatever changes
between the steps of a kind, and no recording where a part cannot be captured."""
import pytest
import torch

from rulorax_tools import CONFIGS as RULORAX

from holon_b200.engine import StepEntry, build
from holon_b200.weights import RandomSource, load_weights

pytestmark = pytest.mark.gpu
CONFIG = dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=2, hidden_size=128, num_attention_heads=4, num_key_value_heads=2, head_dim=32,
              intermediate_size=192, vocab_size=331, rope_theta=10000.0, rms_norm_eps=1e-6, tie_word_embeddings=False)


def made(dtype="bfloat16", graphs=True):
    with torch.inference_mode():
        return build(RandomSource(CONFIG, seed=5, device="cuda:0", dtype=getattr(torch, dtype)), dtype=dtype, device="cuda:0", page_size=16, max_seqs=4,
                     max_model_len=1024, max_step_tokens=1024, pages=160, cuda_graphs=graphs)


def trace(built, lengths, steps, seed=1, between=None):
    g = torch.Generator().manual_seed(seed)
    ids = [torch.randint(0, built.model.spec.vocab, (n + steps,), generator=g).tolist() for n in lengths]
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


def latent(graphs=True, seed=5):
    with torch.inference_mode():
        return build(RandomSource(RULORAX["a"], seed=seed, device="cuda:0", dtype=torch.float32), dtype="float32", device="cuda:0", page_size=16, max_seqs=4,
                     max_model_len=256, max_step_tokens=256, pages=64, cuda_graphs=graphs)


def replayed(built):
    return sum(key[0] == built.runner._generation for key in built.runner._recorded)


def close(a, b):
    return all(torch.linalg.norm(x - y) <= 1e-5 * torch.linalg.norm(y) for x, y in zip(a, b, strict=True))


def test_weights_that_are_loaded_again():
    """The same tensors with other numbers: what latent attention derives from them is another tensor."""
    built, plain = latent(), latent(graphs=False, seed=6)
    trace(built, [9, 30], 5)
    assert replayed(built) == 1
    with torch.inference_mode():
        load_weights(built.model, built.model.spec, RandomSource(RULORAX["a"], seed=6, device="cuda:0", dtype=torch.float32).tensors(), torch.float32, "cuda:0")
        torch.cuda.empty_cache()
    want = trace(plain, [9, 30], 6)
    assert close(trace(built, [9, 30], 6), want) and close(trace(built, [9, 30], 6), want) and replayed(built) == 1


def test_weights_swapped_and_swapped_back():
    built, plain = latent(), latent(graphs=False)
    want = trace(plain, [9, 30], 6)
    assert close(trace(built, [9, 30], 6), want)
    own = {n: p.tensor for n, p in built.model.params()}
    for other in (True, False):
        for n, p in built.model.params():
            p.tensor = own[n] * 0.5 if other and own[n].is_floating_point() else own[n]
        with torch.inference_mode():
            built.model.finalize()
        got = [trace(built, [9, 30], 6) for _ in range(3)]
        assert all(close(x, want) != other for x in got) and all(torch.equal(a, b) for x in got for a, b in zip(x, got[0]))


def test_storage_behind_a_parameter_and_a_number_of_a_part():
    built, plain = latent(), latent(graphs=False)
    trace(built, [9, 30], 4)
    for b in (built, plain):
        with torch.inference_mode():
            p = next(p for n, p in b.model.params() if n.endswith("out.weight"))
            p.tensor.data = p.tensor.data * 3.0
    want = trace(plain, [9, 30], 6)
    assert close(trace(built, [9, 30], 6), want) and close(trace(built, [9, 30], 6), want)
    for b in (built, plain):
        b.model.layers[0].mixer.scale *= 2.0
    other = trace(plain, [9, 30], 6)
    assert not close(other, want) and close(trace(built, [9, 30], 6), other) and close(trace(built, [9, 30], 6), other) and replayed(built)


def test_a_part_with_python_of_its_own_runs_in_every_step():
    """A wrapped `forward`, set before or after steps were recorded, and a part of a class that does not declare itself."""
    built, plain = made("float32"), made("float32", graphs=False)
    want = trace(plain, [9, 30], 6)
    trace(built, [9, 30], 4)
    assert replayed(built) == 1
    forward, kept = built.model.head.forward, []

    def watching(rows):
        kept.append(rows.clone())
        return forward(rows)

    built.model.head.forward = watching
    assert close(trace(built, [9, 30], 6), want) and len(kept) == 7 and all(len(x) for x in kept) and len({x.data_ptr() for x in kept}) == 7
    del built.model.head.forward
    other = made("float32")
    seen = []

    class Head(type(other.model.head)):
        def forward(self, rows):
            seen.append(rows.shape[0])
            return super().forward(rows)

    other.model.head.__class__ = Head
    assert close(trace(other, [9, 30], 6), want) and close(trace(other, [9, 30], 6), want) and seen == [2] * 14 and not other.runner._recorded


def test_kinds_that_come_once_take_no_recordings_place():
    built = made()
    built.runner.GRAPHS = 2
    trace(built, [5], 3)
    graph = next(iter(built.runner._recorded.values()))
    for rows in (2, 3, 4):
        trace(built, [5] * rows, 1)
    assert list(built.runner._recorded.values()) == [graph] and len(built.runner._seen) == 3
    trace(built, [5] * 2, 1)
    assert replayed(built) == 2 and built.runner._use_graphs and len(built.runner._seen) == 2
    built.runner.SEEN = 1
    trace(built, [500] * 2, 1)
    trace(built, [600] * 1, 1)
    assert len(built.runner._seen) == 1


def declared(built, before):
    """`before()` in every pass of a head that says it may be recorded."""
    class Head(type(built.model.head)):
        recordable = True

        def forward(self, rows):
            before(rows)
            return super().forward(rows)

    built.model.head.__class__ = Head


def test_a_capture_without_memory_is_tried_again():
    built, plain = made("float32"), made("float32", graphs=False)
    failed = []

    def before(rows):
        if torch.cuda.is_current_stream_capturing() and len(failed) < 2:
            failed.append(rows.shape)
            raise torch.OutOfMemoryError("CUDA out of memory")

    declared(built, before)
    assert close(trace(built, [9, 30], 12), trace(plain, [9, 30], 12))
    assert len(failed) == 2 and replayed(built) == 1 and built.runner._use_graphs
    assert close(trace(built, [9, 30], 3), trace(plain, [9, 30], 3))


def test_a_part_that_says_so_and_cannot_be_captured():
    built, plain = made("float32"), made("float32", graphs=False)
    seen = []
    declared(built, lambda rows: seen.append(float(rows.float().sum().item())))
    with pytest.warns(UserWarning, match="kernel by kernel"):
        a = trace(built, [9, 30], 8)
    assert close(a, trace(plain, [9, 30], 8)) and not built.runner._use_graphs and not built.runner._recorded and built.runner._pool is None
    assert len(seen) == 9                                  # (the capture ended ahead of its number)


def test_an_error_of_a_part_stays_its_own():
    built = made("float32")

    def before(rows):
        if torch.cuda.is_current_stream_capturing():
            raise RuntimeError("a fault of its own")

    declared(built, before)
    with pytest.raises(RuntimeError, match="a fault of its own"):
        trace(built, [9, 30], 8)
    assert built.runner._use_graphs and torch.cuda.current_stream().query() in (True, False)
