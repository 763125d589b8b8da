"""The step function: a batch of (request, its next tokens) in, logits at the wanted places out.

It runs only the tokens it is given, as one batch, reading everything earlier from the cache
(core/holon/core/executor.py:357-430, 497-564). The caller (the scheduler's engine, or the replay tool) has
admitted the requests and reserved their pages; the step checks that and fails before it touches the device.
"""
from __future__ import annotations

import warnings
from collections.abc import Sequence

import numpy as np
import torch
from torch.utils._device import DeviceContext

from .batch import GroupStep, Rows, StepContext, StepEntry, Uploader
from .recorded import Reads


class StepError(ValueError):
    """A batch that cannot run: tokens out of order, pages not reserved, too many tokens."""


class _Recorded:
    """A step of one-token rows as a CUDA graph that leaves its logits in `logits`, and the kernels it launches."""

    __slots__ = ("graph", "logits", "launches")

    def __init__(self, graph, logits, launches: int) -> None:
        self.graph, self.logits, self.launches = graph, logits, launches


def _watched() -> bool:
    """Whether a mode of the caller's (torch's dispatch and function modes, but for a default device) sees each torch call of a step."""
    modes = range(torch._C._len_torch_function_stack())
    return torch._C._len_torch_dispatch_stack() > 0 or any(type(torch._C._get_function_stack_at(i)) is not DeviceContext for i in modes)


class Runner:
    GRAPHS = 8                                        # recorded steps a runner keeps, the last used ones
    SEEN = 64                                         # kinds of steps it remembers to have run once

    def __init__(self, model, cache, build_ctx, max_step_tokens: int, cuda_graphs: bool = False) -> None:
        """`cuda_graphs`: `step` records steps of one-token rows that come again and replays them, where all that such a step
        reads is understood (engine/recorded.py)."""
        self.model, self.cache, self.ctx = model, cache, build_ctx
        self._graphs = cuda_graphs and build_ctx.device.type == "cuda"
        self._recorded: dict[tuple, _Recorded] = {}                # by shape and plan
        self._seen: dict[tuple, None] = {}                         # kinds that came once
        self._pool = self._stream = None                           # the recordings' memory (None: there are none)
        self._logits = None                                        # [max_seqs, vocab]: where all of them leave their logits
        self.device, self.max_step_tokens = build_ctx.device, max_step_tokens
        s, t, g = cache.max_seqs + 1, max_step_tokens, len(cache.groups)
        tables = sum(s * (group.max_pages + 1) + 8 for group in cache.groups)     # every block-table row changed at once
        self.uploader = Uploader(t * (3 + g) + 16 * s + 64 + tables, self.device)
        self.vocab = model.spec.vocab
        self._reads = None                                        # what recorded steps read (None: not looked at)
        self._use_graphs = self._graphs and Reads.declared(model) # whether steps may be recorded, as far as known
        self._generation = self._wait = self._backoff = 0

    # ------------------------------------------------------------------ host half
    def check(self, entries: Sequence[StepEntry]) -> None:
        c, seen, total = self.cache, set(), 0
        if not entries:
            raise StepError("a step needs at least one entry")
        for e in entries:
            n = len(e.tokens)
            if n == 0:
                raise StepError(f"slot {e.slot}: an entry brings no tokens")
            if e.slot not in c.live:
                raise StepError(f"slot {e.slot} is not admitted")
            if e.slot in seen:
                raise StepError(f"slot {e.slot} appears twice in one step")
            seen.add(e.slot)
            if e.start != int(c.computed[e.slot]):
                raise StepError(f"slot {e.slot}: tokens start at {e.start}, the cache holds {int(c.computed[e.slot])}")
            if e.start + n > c.capacity(e.slot):
                raise StepError(f"slot {e.slot}: pages for {e.start + n} tokens are not reserved "
                                f"(capacity {c.capacity(e.slot)})")
            if any(not 0 <= w < n for w in e.want):
                raise StepError(f"slot {e.slot}: wanted places {list(e.want)} are outside its {n} tokens")
            if e.from_last and n != 1:
                raise StepError(f"slot {e.slot}: only a single token can be fed from the device")
            if any(not 0 <= t < self.vocab for t in e.tokens):
                raise StepError(f"slot {e.slot}: a token id is outside the vocabulary of {self.vocab}")
            total += n
        if total > self.max_step_tokens:
            raise StepError(f"{total} tokens in one step; max_step_tokens is {self.max_step_tokens}")

    def context(self, entries: Sequence[StepEntry], pad_rows: int | None = None, extra=None) -> StepContext:
        """Lays the batch out (rows of one token first), uploads it in one copy and returns the device-side view.
        `pad_rows` (not None: the step runs as a CUDA graph): so many rows of one token each for the padding slot
        follow the entries' one-token rows, and logits are taken at the last token of every row, padding included,
        so that the layout and the work depend on the counts alone (one-token rows with padding, rows of several
        tokens, tokens), not on the entries.
        `extra`: {name: int32 array} uploaded alongside; the device views land in `StepContext.extra`."""
        c = self.cache
        order = sorted(range(len(entries)), key=lambda i: len(entries[i].tokens) != 1)       # stable
        counts = [len(entries[i].tokens) for i in order]
        n_decode = sum(1 for n in counts if n == 1)
        bucket = pad_rows is not None
        pad_rows = pad_rows or 0
        if pad_rows:
            counts[n_decode:n_decode] = [1] * pad_rows
        b = len(counts)
        query_start = np.zeros(b + 1, dtype=np.int32)
        np.cumsum(counts, out=query_start[1:])
        t = int(query_start[-1])
        token_ids, positions = np.zeros(t, dtype=np.int32), np.zeros(t, dtype=np.int32)
        row_slot, kv_len = np.full(b, c.padding_slot, dtype=np.int32), np.ones(b, dtype=np.int32)
        token_slot = np.full(t, c.padding_slot, dtype=np.int32)
        from_last = np.zeros(b, dtype=np.int32)
        offset_of = {}
        rows = list(range(n_decode)) + list(range(n_decode + pad_rows, b))
        for r, i in zip(rows, order):
            e, a, n = entries[i], int(query_start[r]), counts[r]
            token_ids[a:a + n] = e.tokens
            positions[a:a + n] = np.arange(e.start, e.start + n)
            token_slot[a:a + n] = e.slot
            row_slot[r], kv_len[r] = e.slot, e.start + n
            from_last[r] = int(e.from_last)
            offset_of[i] = a
        if bucket:
            logits_index = query_start[1:] - 1
        else:
            logits_index = np.array([offset_of[i] + w for i, e in enumerate(entries) for w in e.want], dtype=np.int32)
        up = self.uploader
        up.begin()
        up.put("token_ids", token_ids)
        up.put("positions", positions)
        up.put("query_start", query_start)
        up.put("row_slot", row_slot)
        up.put("kv_len", kv_len)
        up.put("logits_index", logits_index)
        up.put("from_last", from_last)
        for g in c.groups:
            up.put(f"write_index.{g.index}", g.write_index(token_slot, positions).astype(np.int32))
        for name, array in (extra or {}).items():
            up.put(name, array)
        changed = []
        for g in c.groups:                            # block-table rows that changed, behind everything a graph reads
            slots, table_rows = g.take_dirty()        # (copies: the host table may change before the upload is read)
            if len(slots):
                up.put(f"table_slots.{g.index}", slots)
                up.put(f"table_rows.{g.index}", table_rows.reshape(-1))
                changed.append(g)
        dev = up.end()
        for g in changed:
            self.ctx.kernels.scatter_rows(g.table_device, dev[f"table_slots.{g.index}"], dev[f"table_rows.{g.index}"])
        rows_ = Rows(dev["row_slot"], dev["query_start"], dev["kv_len"], b, t, n_decode + pad_rows,
                     max(counts), int(kv_len.max()), query_start, kv_len)
        if bucket:
            rows_.plan["any cut"] = True              # (a graph's launches serve every cut of its tokens into its rows)
        groups = [GroupStep(g.table_device, dev[f"write_index.{g.index}"], g.page_size) for g in c.groups]
        step = StepContext(dev["token_ids"], dev["positions"], dev["logits_index"], rows_, groups, c)
        step.extra = {name: dev[name] for name in (extra or {})}
        step.from_last = dev["from_last"]
        step.offset_of = offset_of                    # entry index -> where its tokens start among the step's
        return step

    # ------------------------------------------------------------------ the step
    def step(self, entries: Sequence[StepEntry]) -> torch.Tensor | None:
        """Logits [wanted, vocab] in 32-bit, in the order of the entries and of each entry's `want`; None when
        nothing is wanted. Afterwards the cache holds the step's tokens."""
        self.check(entries)
        if self._graphs and all(len(e.tokens) == 1 and tuple(e.want) == (0,) and not e.from_last for e in entries) \
                and not torch.cuda.is_current_stream_capturing() and not _watched() and self._settled():
            logits = self._single(entries)
        else:
            logits = self.model.forward(self.context(entries))
        self.commit(entries)
        return logits

    def _read(self) -> tuple:
        """What a step reads beside its own arrays."""
        c = self.cache
        return (self.model, c.kv_of_entry, c.slot_states, self.uploader.dev, *(g.table_device for g in c.groups))

    def _settled(self) -> bool:
        """Whether a step of this model may be recorded at all, as far as known. Where something that steps read has been replaced, what was
        recorded before is of an earlier generation and is not replayed again. What the model reads now is looked at
        a step later, and after ever more steps where it may not be recorded or where every step finds something else replaced (the
        look takes as long as a step of few layers)."""
        if self._reads is not None and not self._reads.same(*self._read()):
            self._reads, self._generation = None, self._generation + 1
            self._rest()
        elif self._wait:
            self._wait -= 1
        elif not self._use_graphs:
            self._look()
        return self._use_graphs

    def _look(self) -> None:
        self._reads = Reads.of(*self._read())
        self._use_graphs = self._reads is not None
        if self._reads is None:
            self._rest()

    def _rest(self) -> None:
        self._wait = self._backoff = min(1023, 2 * self._backoff + 1)

    def _single(self, entries: Sequence[StepEntry]) -> torch.Tensor:
        """A step of one-token rows whose logits are all wanted. Enqueued kernel by kernel it is bound by the host (28 layers of
        width 1,024, five rows: 3.1 ms a step, 0.9 ms of it kernels; a trace of 2,200 tokens and six such steps takes 10.3 ms in place of 20.8), so a step whose
        shape and plan have come before is recorded and from then on replayed, until anything that it reads is replaced
        (`_settled`). The first of a kind runs as it is: a
        capture takes the host's time once more, which a step that never comes again would not earn back, and what
        kernels do for their first launch must not be captured. Both run with the plan that serves every step of the kind, so a
        step's logits do not depend on how it was run."""
        step = self.context(entries, pad_rows=0)
        kind = (len(entries), self.model.capture_plan(step, self.ctx.max_positions),
                torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction)
        key = (self._generation, *kind)
        found = self._recorded.get(key)
        if found is None and kind not in self._seen:
            self._keep(self._seen, kind, None, self.SEEN)
        elif found is None:
            if self._reads is None and not self._wait:
                self._look()
            if self._reads is not None:
                del self._seen[kind]
                found = self._record(step)
        if found is None:
            return self.model.forward(step)
        self._keep(self._recorded, key, found, self.GRAPHS)
        self._backoff = 0
        found.graph.replay()
        if found.launches:
            self.ctx.kernels.launches += found.launches
        return found.logits.clone()                    # (the place is the next replay's, too)

    @staticmethod
    def _keep(kept: dict, key, value, most: int) -> None:
        kept.pop(key, None)
        kept[key] = value
        while len(kept) > most:
            del kept[next(iter(kept))]

    def _record(self, step) -> _Recorded | None:
        """None where it did not work: for want of memory (the step is recorded another time), or, and then nothing is recorded from then on,
        where a part does what a capture refuses (reads results on the host, say) although it says that it may be recorded."""
        kernels = self.ctx.kernels
        before = getattr(kernels, "launches", None)
        graph, main = torch.cuda.CUDAGraph(), torch.cuda.current_stream(self.device)
        if self._stream is None:
            self._stream = torch.cuda.Stream(self.device)
        self._stream.wait_stream(main)
        error = None
        try:
            if self._logits is None:
                with torch.inference_mode(False):      # (steps in and out of that mode write it)
                    self._logits = torch.empty(self.cache.max_seqs, self.vocab, dtype=torch.float32, device=self.device)
        except torch.OutOfMemoryError:
            return None
        logits = self._logits[:len(step.logits_index)]
        with torch.cuda.stream(self._stream):
            try:
                graph.capture_begin(pool=self._pool, capture_error_mode="thread_local")
                try:
                    logits.copy_(self.model.forward(step))      # (a step's own logits are the pool's, as all it makes)
                finally:
                    graph.capture_end()
            except RuntimeError as e:
                error = e.__context__ or e             # (the capture's end fails, too, once something in it has failed)
        main.wait_stream(self._stream)
        launches = 0
        if before is not None:
            launches, kernels.launches = kernels.launches - before, before
        if error is None:
            self._pool = graph.pool()
            return _Recorded(graph, logits, launches)
        if getattr(kernels, "_pending", None):         # (queued for a launch that was to be recorded)
            kernels._pending.clear()
        if isinstance(error, torch.OutOfMemoryError):
            return None
        if "captur" not in str(error):
            raise error
        warnings.warn(f"steps of one-token rows run kernel by kernel from here on: {error}")
        self._graphs = self._use_graphs = False
        self._recorded.clear()
        self._pool = None                              # (a pool without a graph is given back: its name stands for nothing)
        return None

    def commit(self, entries: Sequence[StepEntry]) -> None:
        for e in entries:
            self.cache.advance(e.slot, e.start + len(e.tokens))
