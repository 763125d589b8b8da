"""Kernels that take several neighbouring numbers a thread, and products with a gated unit in their epilogue, at the sizes where such a
form begins and ends: whole pieces, one piece over, sizes and views that stay with the general form."""
import pytest
import torch

from ref_kernels import RefKernels
from test_gpu_kernels import close, rand

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
REF = RefKernels()
BF16 = torch.bfloat16


@pytest.fixture(scope="module")
def K():
    from holon_b200.kernels import load_kernels
    return load_kernels(torch.device(DEV))


@pytest.mark.parametrize("tokens", [1, 33])
@pytest.mark.parametrize("n,at,wide", [(8, 0, 8), (520, 8, 640), (2048, 16, 4096), (4104, 0, 4104), (100, 0, 100), (64, 3, 72), (64, 8, 77)])
@pytest.mark.parametrize("dtype", [torch.float32, BF16])
def test_sigmoid_gate(K, tokens, n, at, wide, dtype):
    o, g = rand(tokens, n, dtype=dtype, seed=1), rand(tokens, wide, dtype=dtype, seed=2, scale=4.0)
    got = o.clone().to(DEV)
    K.sigmoid_gate(got, g.to(DEV)[:, at:at + n])
    REF.sigmoid_gate(o, g[:, at:at + n])
    close(got, o, dtype)


@pytest.mark.parametrize("heads,dim,vdim", [(8, 128, 256), (4, 4, 6), (3, 4, 3), (2, 8, 5), (3, 5, 7), (1, 12, 2)])
@pytest.mark.parametrize("more", [0, 3, 8])
@pytest.mark.parametrize("dtype", [torch.float32, BF16])
def test_mlstm_prepare(K, heads, dim, vdim, more, dtype):
    t = 5
    first, take = rand(t, 2 * heads * dim + heads * vdim + more, dtype=dtype, seed=1), rand(t, heads, seed=2)
    out = []
    for kernels, dev in ((K, DEV), (REF, "cpu")):
        qk, v1 = torch.full((t, 2, heads, dim), 7.0, device=dev), torch.full((t, heads, vdim + 1), 7.0, device=dev)
        kernels.mlstm_prepare(qk, v1, take.to(dev), first.to(dev), 0.3)
        out.append((qk.cpu(), v1.cpu()))
    assert torch.equal(out[0][1], out[1][1])
    close(out[0][0], out[1][0], torch.float32)


@pytest.mark.parametrize("heads,kv_heads,vd", [(16, 4, 128), (8, 8, 20), (8, 4, 6), (16, 2, 64), (9, 3, 8), (12, 4, 30), (4, 4, 3), (1, 1, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, BF16])
def test_talking_mix(K, heads, kv_heads, vd, dtype):
    tokens, skip = 7, 2
    wide, talk = rand(tokens, heads, kv_heads, vd, dtype=dtype, seed=1), rand(heads, heads, seed=2)
    out = torch.full((tokens, heads, vd), 7.0, dtype=dtype, device=DEV)
    w, m = wide.to(DEV), talk.to(DEV)
    K._call("hb_talking_mix", K._p(out), K._p(w), int(dtype == BF16), skip, tokens - skip, heads, kv_heads, vd, K._p(m))
    own = torch.arange(heads) // (heads // kv_heads)
    want = torch.einsum("hg,tghd->thd", talk.double(), wide.double()[:, :, own])
    assert (out[:skip] == 7.0).all()
    # sums of up to 16 numbers of size 1 by such, rounded once (2^-9 of up to about 16)
    close(out[skip:], want[skip:], dtype, scale=8.0)


@pytest.mark.parametrize("dim", [4, 508, 1024, 1028, 2048, 2052, 4100, 8192, 8196, 30])
@pytest.mark.parametrize("kept", [0, 1, 2, 5, 6, 9])
@pytest.mark.parametrize("y_dtype,cast_dtype", [(BF16, BF16), (torch.float32, BF16), (BF16, torch.float32), (None, BF16)])
def test_out_norm_add(K, dim, kept, y_dtype, cast_dtype):
    rows = 3
    y = rand(rows, dim, seed=1).to(y_dtype) if y_dtype else None
    bias, w = rand(dim, seed=2).to(BF16), rand(dim, seed=3)
    src, hist, coef = rand(rows, dim, seed=4), rand(max(kept, 1), rows, dim, seed=5), rand(max(kept, 1), seed=6)
    out = []
    for kernels, dev in ((K, DEV), (REF, "cpu")):
        mv = lambda a: a.to(dev) if a is not None else None      # noqa: E731
        h, avg, cast = hist.clone().to(dev), torch.zeros(rows, dim, device=dev), torch.zeros(rows, dim, dtype=cast_dtype, device=dev)
        dst = h[kept - 1] if kept else torch.zeros(rows, dim, device=dev)
        more = dict(hist=h, n_hist=kept, coef=coef.to(dev), avg=avg) if kept else {}
        kernels.out_norm_add(dst, src.to(dev), mv(y), mv(bias) if y is not None else None, mv(w) if y is not None else None, 1e-6, 1.0, cast=cast, **more)
        out.append([a.float().cpu() for a in (dst, avg, cast)])
    close(out[0][0], out[1][0], torch.float32, scale=4.0)
    close(out[0][1], out[1][1], torch.float32, scale=8.0)
    close(out[0][2], out[1][2], cast_dtype, scale=8.0)


@pytest.mark.parametrize("rows,experts,inter,k", [(900, 5, 264, 136), (400, 3, 8, 64), (2000, 6, 512, 72)])
@pytest.mark.parametrize("products", ["tcgen05", "mma"])
def test_swiglu_of_experts(K, rows, experts, inter, k, products, monkeypatch):
    monkeypatch.setattr(K, "expert_products", products)
    g = torch.Generator().manual_seed(rows)
    starts = torch.tensor([0, *torch.sort(torch.randint(0, rows + 1, (experts - 1,), generator=g)).values.tolist(), rows], dtype=torch.int32)
    tokens = rows // 2
    x, w = rand(tokens, k, dtype=BF16, seed=1), rand(experts, 2 * inter, k, dtype=BF16, seed=2, scale=k ** -0.5)
    token_of = torch.randint(0, tokens, (rows,), generator=g).to(torch.int32)
    out, both = torch.full((rows, inter), 7.0, dtype=BF16, device=DEV), torch.empty(rows, 2 * inter)
    K.expert_swiglu(out, x.to(DEV), token_of.to(DEV), w.to(DEV), starts.to(DEV))
    REF.expert_linear(both, x.float(), token_of, w.float(), starts, 0)
    want = torch.nn.functional.silu(both[:, :inter]) * both[:, inter:]
    assert K.tcgen05_status() == 0
    close(out, want, BF16, scale=4.0)                            # (products of up to about 8, the library's form rounds twice)
