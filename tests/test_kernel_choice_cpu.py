"""Which function of the compiled library a call of the kernel table goes to, without a GPU: the table's methods on CPU tensors
with a library that only writes down what it is asked for."""
import types

import pytest
import torch

from holon_b200.engine.batch import Rows
from holon_b200.kernels.cuda import CudaKernels

F32 = torch.float32


class Noted(CudaKernels):
    def __init__(self):
        self.device, self.called, self.scan_parts, self._pending, self._splits = torch.device("cpu"), [], True, [], {}
        self.gemm, self.gemm_pair, self.attention_bf16, self.prefill_attention, self.skinny32 = "auto", True, "fast", "tcgen05", True
        self.lib = types.SimpleNamespace(hb_recurrent_blocks_floats=lambda general, dim: 1 if dim in (64, 128, 256) else 0,
                                         hb_latent_tcgen05_takes=lambda *sizes: 1)

    def _check(self, *tensors):
        assert all(t is None or t.is_contiguous() for t in tensors)

    def _call(self, name, *args):
        self.called.append(name)

    def linear_tcgen05(self, out, x, weight, swiglu=False, pair=None):
        self.called.append("linear_tcgen05")


def rows_of(counts, host=False):
    counts = sorted(counts, key=lambda n: n != 1)
    starts = [sum(counts[:i]) for i in range(len(counts) + 1)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32)                                # noqa: E731
    return Rows(i32(list(range(len(counts)))), i32(starts), i32(counts), len(counts), starts[-1], counts.count(1), max(counts), max(counts),
                starts if host else None, counts if host else None)


def scan(counts, *, heads=2, kv_heads=2, dim=64, vdim=8, host=False, **given):
    """The calls of a scan over `counts`; given: decay, head, token, beta, rate, take, skip."""
    k, rows = Noted(), rows_of(counts, host)
    t = rows.n_tokens
    shapes = dict(decay=(t, heads, dim), head=(heads,), token=(t, heads), beta=(t, heads), rate=(t, heads, dim), take=(t, heads), skip=(heads,))
    x = {name: torch.zeros(shape) if given.get(name) else None for name, shape in shapes.items()}
    k.recurrent_scan(torch.zeros(t, heads, vdim), torch.zeros(t, 2, kv_heads, dim), torch.zeros(t, heads, vdim), x["decay"], x["head"], x["beta"],
                     torch.zeros(len(counts), heads, vdim, dim), rows, token_decay=x["token"], rate=x["rate"], take=x["take"], skip=x["skip"])
    return k.called


@pytest.mark.parametrize("given", [dict(head=True), dict(token=True), dict(decay=True, beta=True), dict(head=True, beta=True), dict(decay=True, rate=True)])
@pytest.mark.parametrize("more", [dict(take=True), dict(skip=True), dict(take=True, skip=True)])
def test_factors_and_skips_go_to_the_scan(given, more):
    """What the token-by-token scan refuses (all of these but a decay per token with both) is not run without them."""
    assert scan([300], **given, **more) == ["hb_recurrent_scan"]


def test_sizes_that_the_scan_refuses_are_refused():
    for given in (dict(head=True), dict(token=True)):
        assert scan([300], **given) == ["hb_recurrent_chunks"]
        assert scan([300], dim=1028, **given) == ["hb_recurrent_scan"]               # (a key size above 1024)
        assert scan([300], heads=1, kv_heads=1, dim=1024, vdim=4200, **given) == ["hb_recurrent_scan"]   # (states that the chunks refuse)


BLOCKS = dict(decay=True, beta=True)


def test_a_row_goes_in_parts_by_its_own_tokens(monkeypatch):
    """Long rows in parts and short ones by the scan, whatever the average; no launch for rows that the host knows not to be there."""
    monkeypatch.setattr(CudaKernels, "CHUNK_TOKENS", 192)
    monkeypatch.setattr(CudaKernels, "BLOCK_TOKENS", 48)
    parts, short, scanned = "hb_recurrent_chunks", "hb_recurrent_scan_below", "hb_recurrent_scan"
    for host, counts, want in ((True, [191], [scanned]), (True, [192], [parts]), (True, [1, 192], [parts, scanned]),
                               (True, [191, 191, 1], [scanned]), (True, [2048, *[16] * 11], [parts, short]), (True, [300, 192], [parts]),
                               (False, [191], [scanned]), (False, [192], [parts]), (False, [96, 96], [parts, short]), (False, [96, 95], [scanned]),
                               (True, [1] * 300, [scanned])):
        assert scan(counts, host=host, head=True) == want, counts
        assert scan(counts, host=host, token=True) == want, counts
    for host, counts, want in ((True, [47], [scanned]), (True, [48, 100], ["hb_recurrent_blocks"]), (True, [47, 48], ["hb_recurrent_blocks", short])):
        assert scan(counts, host=host, **BLOCKS) == want, counts
    assert scan([100], dim=96, host=True, **BLOCKS) == [scanned]


def test_parts_of_any_cut():
    """For a captured launch the parts of every cut of so many tokens into so many rows fit what is launched."""
    import random
    rng = random.Random(1)
    for _ in range(300):
        portions, least, size = rng.randint(1, 6), rng.choice([48, 192]), rng.choice([8, 64])
        counts = [rng.randint(2, 400) for _ in range(portions)]
        exact = CudaKernels._long_rows(rows_of(counts, host=True), least, size)
        captured = rows_of(counts, host=True)
        captured.plan["any cut"] = True
        most = CudaKernels._long_rows(captured, least, size)
        assert exact[0] <= most[0] and exact[1] <= most[1] and exact[2] <= most[2]
        assert exact[:2] == (sum(n >= least for n in counts), sum(-(-n // size) for n in counts if n >= least))


def product(m, n, k=256, out=F32, gemm="auto"):
    table = Noted()
    table.gemm = gemm
    mm = []
    real, torch.mm = torch.mm, lambda *a, **kw: mm.append("library")
    try:
        table.linear(torch.zeros(m, n, dtype=out), torch.zeros(m, k, dtype=torch.bfloat16), torch.zeros(n, k, dtype=torch.bfloat16))
    finally:
        torch.mm = real
    return table.called + mm


@pytest.mark.parametrize("n,rows", [(1, None), (15, None), (17, 1536), (33, 768), (63, 768), (65, 512), (97, 384), (129, 308), (162, 640), (255, 640)])
def test_products_of_an_odd_number_of_32_bit_columns(n, rows):
    """The library's up to `rows` rows (None: always), and at any number of them where it is asked for."""
    for m in (17, 64, 256, 307, 383, 511, 639, 767, 1535, 1536, 4096):
        tcgen05 = rows is not None and m >= rows
        assert product(m, n) == ["linear_tcgen05" if tcgen05 else "library"], m
        assert product(m, n, gemm="cublas") == product(m, n, out=torch.bfloat16) == product(m, n, k=252) == ["library"]
    assert product(2048, 64) == product(2048, 257) == ["library"]
    assert product(16, n) == ["hb_gemm_bf16_skinny"]


@pytest.mark.parametrize("heads,tokens,ones,rows,kernel", [
    (16, 2048, 0, 1, "hb_latent_attention_tcgen05"), (1, 65534 * 128, 0, 1, "hb_latent_attention_tcgen05"),
    (1, 65534 * 128 + 1, 0, 1, "hb_latent_attention_bf16"), (1, 65535 * 128, 0, 1, "hb_latent_attention_bf16"),
    (1, 65532 * 128 + 3, 1, 3, "hb_latent_attention_tcgen05"), (1, 65533 * 128 + 130, 1, 3, "hb_latent_attention_bf16"),
    (128, 1 << 24, (1 << 24) - 2, (1 << 24) - 1, "hb_latent_attention_bf16")])
def test_latent_prompts_of_more_tiles_than_a_launch_has(heads, tokens, ones, rows, kernel):
    """What the tcgen05 kernel refuses (more than 65,535 tiles, or 2^31 queries and heads in a step) stays with the other one."""
    k, rank = Noted(), 64
    k._check = lambda *tensors: None
    k.latent_split = 1
    k.sms = 148
    wide = lambda *shape: torch.zeros(1, dtype=torch.bfloat16).expand(*shape)         # noqa: E731
    i32 = torch.zeros(1, dtype=torch.int32)
    k.latent_attention(wide(tokens, heads, rank), wide(tokens, heads, rank + 16), wide(2, 64, rank + 16), i32.view(1, 1),
                       Rows(i32, i32, i32, rows, tokens, ones, 1, 1), 0.1, rank, 0)
    assert k.called[-1] == kernel


def test_cuts_of_a_step():
    """Every cut holds the step's tokens in rows that can be; no other cut needs noticeably more parts than the measured ones."""
    import random
    from holon_b200.engine.build import _cuts
    rng = random.Random(2)
    for _ in range(300):
        rows, longest = rng.randint(1, 70), rng.choice([40, 200, 5000])
        tokens = rng.randint(1, min(4096, rows * longest))
        lengths = [n for n in (CudaKernels.CHUNK_TOKENS + 1, CudaKernels.BLOCK_TOKENS + 1)]
        cuts = _cuts(tokens, rows, longest, lengths)
        assert all(sum(c) == tokens and len(c) <= rows and 1 <= min(c) and max(c) <= longest for c in cuts)
        for least, size in ((CudaKernels.CHUNK_TOKENS, 64), (CudaKernels.BLOCK_TOKENS, 8)):
            parts = lambda c: sum(-(-n // size) for n in c if n >= least)             # noqa: E731
            for _ in range(5):
                ends = sorted(rng.randint(0, tokens) for _ in range(rng.randint(1, rows) - 1))
                counts = [b - a for a, b in zip([0, *ends], [*ends, tokens])]
                if max(counts) <= longest:
                    assert parts(counts) <= 1.03 * max(map(parts, cuts)) + 2, (tokens, rows, longest, counts, cuts)
