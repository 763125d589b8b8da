"""The recurrences in parts of several tokens against the token-by-token formula in 64 bits and against the token-by-token
kernel: rows whose last part is short, one-token rows beside them, every form of decay, decays of zero and below, value sizes
that leave a tile of columns half empty."""
import pytest
import torch

from holon_b200.engine.batch import Rows

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
FORMS = ["fixed", "token", "channel", "fixed delta", "delta", "general"]


@pytest.fixture(scope="module")
def K():
    from holon_b200.kernels import load_kernels
    return load_kernels(torch.device(DEV))


def plain(qk, v, state, counts, slots, decay, beta, rate):
    """decay [tokens, heads, dim] in 64 bits; state [slots, heads, vdim, dim]."""
    qk, v, state, decay = (x.double() for x in (qk, v, state, decay))
    group, out, t = v.shape[1] // qk.shape[2], torch.empty_like(v), 0
    for n, slot in zip(counts, slots):
        s = state[slot].transpose(1, 2).clone()                                       # [head, key, value]
        for t in range(t, t + n):
            q, k = (qk[t, i].repeat_interleave(group, 0) for i in (0, 1))
            a = torch.einsum("hkv,hk->hv", s if rate is not None else s * decay[t][..., None], k)
            u = v[t] if beta is None else beta[t].double()[:, None] * (v[t] - a)
            s = s * decay[t][..., None] + k[..., None] * u[:, None]
            if rate is not None:
                s = s - (rate[t].double() * k)[..., None] * a[:, None]
            out[t] = torch.einsum("hkv,hk->hv", s, q)
        t += 1
        state[slot] = s.transpose(1, 2)
    return out, state


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 2, 64, 64), (3, 3, 128, 129), (5, 5, 256, 20), (6, 2, 128, 128), (2, 1, 64, 7),
                                                     (40, 8, 64, 70), (3, 1, 36, 10), (10, 5, 256, 70)])
def test_against_the_formula(K, form, heads, kv_heads, dim, vdim, monkeypatch):
    for name in ("CHUNK_TOKENS", "BLOCK_TOKENS"):                                      # (short rows too)
        monkeypatch.setattr(type(K), name, 2, raising=False)
    g = torch.Generator().manual_seed(dim + vdim)
    counts, slots = [1, 1, 8, 3, 200, 9, 7, 64, 65, 127], [6, 0, 3, 1, 2, 8, 5, 7, 9, 10]
    t = sum(counts)
    qk = torch.nn.functional.normalize(torch.randn(t, 2, kv_heads, dim, generator=g), dim=-1)
    v, state = torch.randn(t, heads, vdim, generator=g), torch.randn(11, heads, vdim, dim, generator=g) * 0.2
    decay = 1 - torch.rand(t, heads, dim, generator=g) ** 3 * 0.3
    decay[5:40:7] = 0.0                                                               # what went before is gone
    decay[60:64, :, ::3] = 1e-30
    decay[70:74] *= -1
    beta = torch.rand(t, heads, generator=g) if "delta" in form else None
    rate = torch.rand(t, heads, dim, generator=g) if form == "general" else None
    head = 1 - 2.0 ** -(3 + torch.arange(heads, dtype=torch.float32)) if "fixed" in form else None
    if head is not None:
        head[-1] *= -1
    token = decay[:, :, 0].contiguous() if form == "token" else None
    if head is not None:
        decay = head[None, :, None].expand(t, heads, dim)
    if token is not None:
        decay = token[:, :, None].expand(t, heads, dim)
    want, want_state = plain(qk, v, state, counts, slots, decay, beta, rate)
    starts = torch.tensor([0] + counts, dtype=torch.int32).cumsum(0).to(torch.int32)
    rows = Rows(torch.tensor(slots, dtype=torch.int32, device=DEV), starts.to(DEV), starts[1:].to(DEV), len(counts), t, 2, max(counts), 0)
    dev = lambda x: None if x is None else x.contiguous().to(DEV)                     # noqa: E731
    errors = {}
    for parts in (False, True):
        monkeypatch.setattr(K, "scan_parts", parts)
        s, out = dev(state), torch.full((t, heads, vdim), float("nan"), device=DEV)
        before = K.launches
        K.recurrent_scan(out, dev(qk), dev(v), dev(decay) if head is None and token is None else None, dev(head), dev(beta), s, rows,
                         token_decay=dev(token), rate=dev(rate))
        taken = form in ("fixed", "token") or form != "channel" and dim in (64, 128, 256)
        assert K.launches - before == (2 if parts and taken else 1)
        errors[parts] = [float(torch.linalg.norm(x.cpu() - w) / torch.linalg.norm(w)) for x, w in ((out, want), (s, want_state))]
        # 32-bit sums over up to 256 channels, and over the tokens that a decay near one lets through
        assert max(errors[parts]) < 2e-6, errors
        assert torch.equal(s[4].cpu(), state[4])                                      # a slot of no row
    assert errors[True][0] < 1.25 * errors[False][0] + 1e-8 and errors[True][1] < 2 * errors[False][1], errors


@pytest.mark.parametrize("form", ["fixed", "token", "delta", "general"])
def test_what_is_no_number_reaches_no_earlier_token(K, form):
    """An infinity among token 37's values, and then among its keys: the outputs before it keep their bits, those from it on are no numbers."""
    t, heads, dim, vdim = 220, 2, 64, 64
    g = torch.Generator().manual_seed(1)
    qk = torch.nn.functional.normalize(torch.randn(t, 2, heads, dim, generator=g), dim=-1).to(DEV)
    v, decay = torch.randn(t, heads, vdim, generator=g).to(DEV), (1 - torch.rand(t, heads, dim, generator=g) * 0.1).to(DEV)
    beta, rate = torch.rand(t, heads, generator=g).to(DEV), torch.rand(t, heads, dim, generator=g).to(DEV)
    rows = Rows(torch.zeros(1, dtype=torch.int32, device=DEV), torch.tensor([0, t], dtype=torch.int32, device=DEV),
                torch.tensor([t], dtype=torch.int32, device=DEV), 1, t, 0, t, t)

    def run(qk, v):
        out, state = torch.empty_like(v), torch.zeros(2, heads, vdim, dim, device=DEV)
        K.recurrent_scan(out, qk, v, decay if form in ("delta", "general") else None, decay[0, :, 0].contiguous() if form == "fixed" else None,
                         beta if form == "delta" else None, state, rows, token_decay=decay[:, :, 0].contiguous() if form == "token" else None,
                         rate=rate if form == "general" else None)
        return out, state

    clean, _ = run(qk, v)
    bad_v, bad_k = v.clone(), qk.clone()
    bad_v[37, 1, 5] = float("inf")
    bad_k[37, 1, 1, 7] = float("inf")
    for out, state, where in ((*run(qk, bad_v), (slice(37, None), 1, 5)), (*run(bad_k, v), (slice(38, None), 1))):
        assert torch.equal(out[:37], clean[:37]) and torch.equal(out[:, 0], clean[:, 0])
        assert not out[where].isfinite().any() and not state[0, 1].isfinite().all()


def test_a_state_space_value_that_is_no_number_reaches_no_earlier_token(K):
    t, heads, groups, n, vdim = 220, 4, 2, 64, 64
    g = torch.Generator(device=DEV).manual_seed(1)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)                           # noqa: E731
    cb, v, dt, rate, skip = r(t, 2, groups, n), r(t, heads, vdim), torch.rand(t, heads, generator=g, device=DEV), r(heads), r(heads)
    decay, starts = torch.exp(-rate.exp() * dt), torch.tensor([0, t], dtype=torch.int32, device=DEV)
    rows = Rows(starts[:1], starts, starts[1:], 1, t, 0, t, t, [0, t], [t])
    outs = []
    for bad in (None, float("inf"), float("nan")):
        if bad is not None:
            v[37, 1, 5] = bad
        out, state = torch.empty_like(v), torch.zeros(2, heads, vdim, n, device=DEV)
        K.state_space_scan(out, cb, v, dt, decay, rate, skip, state, rows)
        outs.append(out)
    for out in outs[1:]:
        assert torch.equal(out[:37], outs[0][:37]) and not out[37:, 1, 5].isfinite().any()
        kept = torch.ones_like(out, dtype=torch.bool)
        kept[37:, 1, 5] = False
        assert torch.equal(out[kept], outs[0][kept])


def off_by(x, floats):
    """x at an address that many floats behind a 16-byte boundary."""
    y = torch.empty(x.numel() + floats, device=x.device)[floats:].view(x.shape)
    assert y.data_ptr() % 16 == 4 * floats and y.is_contiguous()
    return y.copy_(x)


@pytest.mark.parametrize("form", ["fixed", "token", "delta", "general", "state space"])
@pytest.mark.parametrize("vdim", [64, 7])
def test_values_anywhere_in_memory(K, form, vdim):
    """v (and a state space's C and B) need no 16-byte boundary: the same bits as on one."""
    t, heads, dim = 220, 4, 64
    g = torch.Generator(device=DEV).manual_seed(2)
    qk = torch.nn.functional.normalize(torch.randn(t, 2, heads, dim, generator=g, device=DEV), dim=-1)
    v, decay = torch.randn(t, heads, vdim, generator=g, device=DEV), 1 - torch.rand(t, heads, dim, generator=g, device=DEV) * 0.1
    beta, rate = torch.rand(t, heads, generator=g, device=DEV), torch.rand(t, heads, dim, generator=g, device=DEV)
    starts = torch.tensor([0, t], dtype=torch.int32, device=DEV)
    rows = Rows(starts[:1], starts, starts[1:], 1, t, 0, t, t, [0, t], [t])
    outs = []
    for floats in (0, 1, 2):
        out, state, values = torch.empty_like(v), torch.zeros(2, heads, vdim, dim, device=DEV), off_by(v, floats)
        if form == "state space":
            K.state_space_scan(out, off_by(qk, floats), values, beta, torch.exp(-beta), torch.zeros(heads, device=DEV), beta[0].clone(), state, rows)
        else:
            K.recurrent_scan(out, qk, values, decay if form in ("delta", "general") else None, decay[0, :, 0].contiguous() if form == "fixed" else None,
                             beta if form == "delta" else None, state, rows, token_decay=decay[:, :, 0].contiguous() if form == "token" else None,
                             rate=rate if form == "general" else None)
        outs.append((out, state))
    for out, state in outs[1:]:
        assert torch.equal(out, outs[0][0]) and torch.equal(state, outs[0][1])


@pytest.mark.parametrize("form", ["fixed", "token", "delta", "general"])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 2, 128, 64), (8, 8, 256, 128)])
def test_a_row_does_not_depend_on_the_rows_beside_it(K, form, heads, kv_heads, dim, vdim):
    """Rows below, at and above the lengths from which a row goes in parts: the same bits alone and together."""
    counts = [1, 1, 15, 47, 16, 127, 128, 300, 2, 449]
    g = torch.Generator(device=DEV).manual_seed(dim)
    t, slots = sum(counts), [9, 0, 3, 1, 2, 8, 5, 7, 4, 6]
    qk = torch.nn.functional.normalize(torch.randn(t, 2, kv_heads, dim, generator=g, device=DEV), dim=-1)
    v = torch.randn(t, heads, vdim, generator=g, device=DEV)
    decay = 1 - torch.rand(t, heads, dim, generator=g, device=DEV) * 0.1
    beta, rate = torch.rand(t, heads, generator=g, device=DEV), torch.rand(t, heads, dim, generator=g, device=DEV)
    begin = torch.randn(10, heads, vdim, dim, generator=g, device=DEV) * 0.1

    def run(first, counts, slots, host):
        i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)                # noqa: E731
        starts, at = [sum(counts[:i]) for i in range(len(counts) + 1)], slice(first, first + sum(counts))
        rows = Rows(i32(slots), i32(starts), i32(counts), len(counts), starts[-1], counts.count(1), max(counts), 0, starts if host else None)
        state, out = begin.clone(), torch.empty_like(v[at])
        K.recurrent_scan(out, qk[at].contiguous(), v[at].contiguous(), decay[at].contiguous() if form in ("delta", "general") else None,
                         decay[0, :, 0].contiguous() if form == "fixed" else None, beta[at].contiguous() if form == "delta" else None, state, rows,
                         token_decay=decay[at, :, 0].contiguous() if form == "token" else None,
                         rate=rate[at].contiguous() if form == "general" else None)
        return out, state

    for host in (False, True):
        together, states = run(0, counts, slots, host)
        for i, n in enumerate(counts):
            first = sum(counts[:i])
            alone, state = run(first, [n], [slots[i]], host)
            assert torch.equal(alone, together[first:first + n]) and torch.equal(state[slots[i]], states[slots[i]]), (n, host)
