"""Query/key preparation in 16-byte pieces and the batched few-rows product, at the edges of what they take, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def K():
    from serve_b200.kernels import load_kernels

    return load_kernels(DEV)


@pytest.mark.parametrize("m", [1, 8, 9, 16, 17])
@pytest.mark.parametrize("b,n,k", [(1, 8, 16), (16, 192, 128), (3, 40, 256), (5, 136, 48), (2, 64, 272)])
def test_batched_few_rows(K, m, b, n, k):
    """Views of wider buffers on both sides; 17 rows and k = 272 are the library's."""
    wide_a = torch.randn(m, b, k + 8, device=DEV).bfloat16()
    w = (torch.randn(b, n, k, device=DEV) / k ** 0.5).bfloat16()
    wide_o = torch.full((m, b, n + 24), 7.0, device=DEV, dtype=torch.bfloat16)
    K.linear_batched(wide_a[:, :, 4: 4 + k], w, wide_o[:, :, 16: 16 + n])
    want = torch.einsum("mbk,bnk->mbn", wide_a[:, :, 4: 4 + k].double(), w.double())
    most = torch.einsum("mbk,bnk->mbn", wide_a[:, :, 4: 4 + k].double().abs(), w.double().abs())
    # one rounding to bfloat16 (2^-8 of the value at most) and float sums of k terms
    assert ((wide_o[:, :, 16: 16 + n].double() - want).abs() <= 2.0 ** -8 * want.abs() + (k + 8) * 2.0 ** -23 * most).all()
    assert (wide_o[:, :, :16] == 7.0).all() and (wide_o[:, :, 16 + n:] == 7.0).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens", [1, 7, 400])
@pytest.mark.parametrize("heads,kv,d,dim,rot,norm,bias,shared", [
    (16, 4, 128, 128, 64, True, True, False),
    (3, 1, 64, 50, 48, True, False, False),                # padded heads, nearly wholly rotated
    (40, 8, 128, 120, 0, False, True, False),              # no rotation, no norm; more than 512 items
    (64, 8, 256, 256, 128, True, True, False),             # many items a thread
    (6, 2, 80, 80, 16, True, True, True),                  # the values are the keys as projected
    (4, 0, 64, 64, 32, True, False, False),                # queries only
    (2, 1, 24, 20, 12, True, True, False),                 # pieces that do not fit: the other kernel
])
def test_query_key_preparation(K, dtype, tokens, heads, kv, d, dim, rot, norm, bias, shared):
    g = torch.Generator(device=DEV).manual_seed(tokens + d)
    rn = lambda *s: torch.randn(s, generator=g, device=DEV)
    page, n_pages = 16, -(-tokens // 16) + 3
    cols = (heads + (1 if shared else 2) * kv) * d
    live = torch.zeros(cols // d, d, device=DEV)
    live[:, :dim] = 1.0
    live = live.view(-1)
    sums = (rn(tokens, cols + 8) * torch.cat([live, live.new_ones(8)]))[:, :cols]
    b = rn(cols) * live if bias else None
    qw, kw = (rn(heads * d), rn(kv * d) if kv else None) if norm else (None, None)
    pos = torch.arange(tokens, device=DEV, dtype=torch.int32) + 3
    table = torch.randperm(n_pages, generator=g, device=DEV).to(torch.int32)[None].contiguous()
    inv = 1.0 / 10000.0 ** (torch.arange(max(rot // 2, 1), device=DEV).float() / max(rot // 2, 1))
    q = torch.full((tokens, heads * d), float("nan"), device=DEV, dtype=dtype)
    kc, vc = (torch.zeros(n_pages, max(kv, 1), page, d, device=DEV, dtype=dtype) for _ in range(2))
    K.qk_prepare(sums, b, pos, torch.zeros(tokens, dtype=torch.int32, device=DEV), heads, kv, d, dim, qw, kw, 1e-5, inv, rot, q, kc, vc, table, page,
                 keys_are_values=shared)
    K.check_errors()
    x = sums.double() + (b.double() if bias else 0.0)
    nq, nk = heads * d, kv * d
    ang = (pos.float()[:, None] * inv[None]).double()[:, None]

    def turned(z, w, n):
        if w is not None:
            z = z / torch.sqrt(z.square().sum(-1, keepdim=True) / (n * dim) + 1e-5) * w.double()
        z = z.view(tokens, n, d)
        h = rot // 2
        u, v = z[..., :h], z[..., h:rot]
        c, s = ang[..., :h].cos(), ang[..., :h].sin()
        return torch.cat([u * c - v * s, v * c + u * s, z[..., rot:]], -1)

    # float arithmetic throughout (a sum of squares, a root, a turn: below 2^-20 of the row's largest value), one rounding at the end
    tol = lambda want: dict(atol=float(want.abs().max()) * 2.0 ** -20 + 1e-6, rtol=2.0 ** -8 if dtype == torch.bfloat16 else 1e-6)
    want = turned(x[:, :nq], qw, heads)
    torch.testing.assert_close(q.double().view(tokens, heads, d), want, **tol(want))
    if kv:
        keys, values = turned(x[:, nq: nq + nk], kw, kv), x[:, nq + (0 if shared else nk):][:, :nk].view(tokens, kv, d)
        cell = table[0].long()[pos.long() // page]
        torch.testing.assert_close(kc[cell, :, pos.long() % page].double(), keys, **tol(keys))
        torch.testing.assert_close(vc[cell, :, pos.long() % page].double(), values, **tol(values))
