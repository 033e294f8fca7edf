"""The experts' tensor-core products at the edges of their tiles: runs of 1 to more than 256 tokens an expert, counts that are no
multiple of 16, 64 or 128, outputs that end inside a unit, k that ends inside a stage, experts without tokens, every epilogue. The widest two:
long rows of few tokens an expert have two accumulators that fill tensor memory, and blocks that hand them over to a second unit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

E, TOP = 5, 2


def _reference(x, logits, w_gu, w_down, kind):
    x, w_gu, w_down = x.double(), w_gu.double(), w_down.double()
    ff = w_down.shape[2]
    score = torch.softmax(logits.double(), -1) if kind == "swiglu" else torch.sigmoid(logits.double())
    w, idx = score.sort(dim=-1, descending=True, stable=True)
    out = torch.zeros((x.shape[0], w_down.shape[1]), dtype=torch.float64, device=x.device)
    most = torch.zeros_like(out)                            # the same sums of absolute values
    for j in range(TOP):
        for e in range(E):
            t = (idx[:, j] == e).nonzero()[:, 0]
            wt = w[t, j][:, None]
            h = x[t] * wt if kind == "clamped_swish" else x[t]
            g, u = h @ w_gu[e, :ff].T, h @ w_gu[e, ff:].T
            if kind == "clamped_swish":
                g = g.clamp(max=1.5)
                a = g * torch.sigmoid(1.702 * g) * (u.clamp(-1.5, 1.5) + 1)
            else:
                a = g * torch.sigmoid(g) * u
            wt = 1.0 if kind == "clamped_swish" else wt
            out.index_add_(0, t, (a @ w_down[e].T) * wt)
            most.index_add_(0, t, (a.abs() @ w_down[e].abs().T) * wt)
    return out, most


def _bound(want, most):
    """Two roundings to bfloat16 (8 significant bits: by at most 2^-8 of the value): of the activations, so a sum moves by 2^-8 of its
    absolute terms, and of the output; the float sums add less than 2^-15 of the absolute terms."""
    first = (2.0 ** -8 + 2.0 ** -15) * most
    return first + 2.0 ** -8 * (want.abs() + first) + 1e-30


@pytest.mark.parametrize("kind", ["swiglu", "clamped_swish"])
@pytest.mark.parametrize("tokens,k,ff,n", [(1, 64, 32, 40), (7, 96, 160, 64), (16, 2080, 96, 200), (17, 64, 128, 136), (33, 160, 64, 129), (65, 128, 416, 128),
                                           (129, 32, 96, 257), (200, 64, 64, 64), (257, 96, 32, 72), (700, 128, 224, 300),
                                           (200, 3104, 4832, 64), (249, 3136, 4768, 40)])
def test_expert_products(tokens, k, ff, n, kind):
    from serve_b200.kernels import load_kernels

    kernels = load_kernels("cuda:0")
    g = torch.Generator(device="cuda").manual_seed(tokens * 1000 + ff)
    draw = lambda *s: torch.randn(s, generator=g, device="cuda")
    x = draw(tokens, k).bfloat16()
    logits = draw(tokens, E)
    logits[:, 0] += 2.0                                     # a crowded expert
    logits[:, 3] -= 50.0                                    # and one that nobody chooses
    w_gu, w_down = (draw(E, 2 * ff, k) / k ** 0.5).bfloat16(), (draw(E, n, ff) / ff ** 0.5).bfloat16()
    out = torch.full((tokens, n), float("nan"), device="cuda", dtype=torch.bfloat16)
    kernels.routed_experts(x, logits, w_gu, w_down, TOP, out, score="softmax" if kind == "swiglu" else "sigmoid", scale_input=kind != "swiglu",
                           activation=kind, limit=1.5, alpha=1.702)
    kernels.check_errors()
    want, most = _reference(x, logits, w_gu, w_down, kind)
    assert ((out.double() - want).abs() <= _bound(want, most)).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens,k,ff", [(1, 64, 32), (19, 256, 96), (300, 96, 64)])
@pytest.mark.parametrize("gated,identity", [(True, 0), (False, 2)])
def test_one_choice_beside_a_shared_expert(tokens, k, ff, gated, identity, dtype):
    """A single choice a token has no sums of its own to add up, but its output still meets the shared expert's (or is the token itself)."""
    from serve_b200.kernels import load_kernels

    kernels = load_kernels("cuda:0")
    g = torch.Generator(device="cuda").manual_seed(tokens + ff)
    draw = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, shared = draw(tokens, k).to(dtype), draw(tokens, k).to(dtype)
    outputs = E + identity
    logits = draw(tokens, 8)                                # columns beyond the outputs and the gate are not read
    w_gu, w_down = (draw(E, 2 * ff, k) / k ** 0.5).to(dtype), (draw(E, k, ff) / ff ** 0.5).to(dtype)
    bias = draw(outputs) * 0.1
    out = torch.full((tokens, k), float("nan"), device="cuda", dtype=dtype)
    kernels.routed_experts(x, logits, w_gu, w_down, 1, out, score="sigmoid", scale_input=False, activation="swiglu", outputs=outputs,
                           choice_bias=bias, shared=shared, shared_gated=gated)
    kernels.check_errors()
    score = torch.sigmoid(logits[:, :outputs].double())
    idx = (score + bias.double()).argmax(-1)
    want = shared.double() * (torch.sigmoid(logits[:, outputs].double())[:, None] if gated else 1.0)
    most = want.abs()
    for t in range(tokens):
        e, w = int(idx[t]), score[t, idx[t]]
        if e >= E:
            want[t] += w * x[t].double()
            most[t] += w * x[t].double().abs()
        else:
            a = x[t].double() @ w_gu[e, :ff].double().T
            a = a * torch.sigmoid(a) * (x[t].double() @ w_gu[e, ff:].double().T)
            want[t] += w * (a @ w_down[e].double().T)
            most[t] += w * (a.abs() @ w_down[e].double().abs().T)
    # float: sums of k and ff terms, each off by at most 2^-24 of the absolute terms a step
    bound = _bound(want, most) if dtype == torch.bfloat16 else (k + ff + 8) * 2.0 ** -24 * (most + want.abs()) + 1e-30
    assert ((out.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("tokens,k,ff,n", [(3, 64, 32, 48), (20, 96, 160, 130), (300, 64, 96, 72)])
def test_ungated_expert_products(tokens, k, ff, n):
    from serve_b200.kernels import load_kernels

    kernels = load_kernels("cuda:0")
    g = torch.Generator(device="cuda").manual_seed(tokens)
    draw = lambda *s: torch.randn(s, generator=g, device="cuda")
    x = draw(tokens, k).bfloat16()
    w_up, w_down = (draw(E, ff, k) / k ** 0.5).bfloat16(), (draw(E, n, ff) / ff ** 0.5).bfloat16()
    ids = torch.arange(tokens, device="cuda", dtype=torch.int32)
    table = torch.stack([torch.zeros(tokens, device="cuda"), 1 + torch.arange(tokens, device="cuda") % 3], 1).to(torch.int32).contiguous()
    out = torch.full((tokens, n), float("nan"), device="cuda", dtype=torch.bfloat16)
    kernels.table_experts(x, ids, None, table, w_up, w_down, 2, out)
    kernels.check_errors()
    want, most = (torch.zeros((tokens, n), dtype=torch.float64, device="cuda") for _ in range(2))
    for t in range(tokens):
        for e in table[t].tolist():
            a = (x[t].double() @ w_up[e].double().T).clamp(min=0).square()
            want[t] += 0.5 * (a @ w_down[e].double().T)
            most[t] += 0.5 * (a @ w_down[e].double().abs().T)
    assert ((out.double() - want).abs() <= _bound(want, most)).all()


def test_grouped_tokens_take_no_room_of_their_own():
    from serve_b200.kernels import load_kernels

    kernels = load_kernels("cuda:0")
    tokens, k, ff, n = 600, 512, 64, 512
    draw = lambda *s: torch.randn(s, device="cuda")
    x, logits = draw(tokens, k).bfloat16(), draw(tokens, E)
    w_gu, w_down = draw(E, 2 * ff, k).bfloat16(), draw(E, n, ff).bfloat16()
    out = torch.empty((tokens, n), device="cuda", dtype=torch.bfloat16)
    run = lambda: kernels.routed_experts(x, logits, w_gu, w_down, TOP, out)
    run()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    run()
    # float sums and activations of every pair; choices, weights and the grouping's lists are a few dozen bytes a pair
    assert torch.cuda.max_memory_allocated() - before <= TOP * tokens * (4 * n + 2 * ff + 64) + 16384


@pytest.mark.parametrize("pairs,experts,rows", [(1, 1, 16), (32, 64, 16), (33, 5, 16), (1024, 64, 256), (8192, 64, 256), (8200, 64, 256), (40000, 96, 256),
                                                (700, 1500, 32), (9000, 3000, 256)])
def test_grouping_by_expert(pairs, experts, rows):
    """Every pair once at a place of its expert's run, the runs in the experts' order, a tile for every ``rows`` rows of a run; choices that
    name no expert have no place."""
    g = torch.Generator(device="cuda").manual_seed(pairs)
    idx = torch.randint(0, experts + 1, (pairs,), generator=g, device="cuda", dtype=torch.int32)        # ``experts`` itself: none
    ints = lambda n: torch.full((n,), -7, dtype=torch.int32, device="cuda")
    offsets, order, tiles, n_tiles = ints(experts + 1), ints(pairs), ints(2 * (pairs // rows + min(experts, pairs)) + 2), ints(1)
    import ctypes

    from serve_b200.kernels import load_kernels

    kernels = load_kernels("cuda:0")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    assert kernels._moe_lib().sb_moe_sort(p(idx), pairs, experts, rows, p(offsets), p(order), p(tiles), p(n_tiles), kernels._s()) == 0
    counts = torch.bincount(idx.long(), minlength=experts + 1)[:experts].tolist()
    want = [0]
    for n in counts:
        want.append(want[-1] + n)
    assert offsets.tolist() == want
    got, tile = order.tolist(), []
    for e, n in enumerate(counts):
        assert sorted(got[want[e]: want[e + 1]]) == (idx == e).nonzero().flatten().tolist()
        tile += [(e, want[e] + r) for r in range(0, n, rows)]
    assert n_tiles.item() == len(tile) and tiles[: 2 * len(tile)].view(-1, 2).tolist() == [list(t) for t in tile]
    assert got[want[-1]:] == [-7] * (pairs - want[-1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens,n,top", [(1, 4, 1), (33, 64, 3), (70, 1000, 5), (9, 924, 4), (7, 1100, 2), (5, 1024, 9), (3, 1924, 4), (4, 30, 2), (2, 2048, 3)])
def test_sum_over_a_tokens_choices(tokens, n, top, dtype):
    """Rows that fill the blocks a block takes a part of one in, rows that do not, rows of no whole pieces of four;
    choices that are the token itself, a gated shared expert, an input with a stride of its own."""
    import ctypes

    from serve_b200.kernels import load_kernels

    kernels = load_kernels("cuda:0")
    g = torch.Generator(device="cuda").manual_seed(n + top)
    draw = lambda *s: torch.randn(s, generator=g, device="cuda")
    parts, x = draw(tokens * top, n), draw(tokens, n + 4).to(dtype)[:, :n]
    shared, logits, weights = draw(tokens, n).to(dtype), draw(tokens, 3), draw(tokens * top)
    idx = torch.randint(0, 6, (tokens * top,), generator=g, device="cuda", dtype=torch.int32)
    room = torch.full((tokens * n + 8,), 7.0, device="cuda", dtype=dtype)
    out = room[: tokens * n].view(tokens, n)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    code = 1 if dtype == torch.bfloat16 else 0
    assert kernels._moe_lib().sb_moe_combine_more(p(parts), p(idx), p(weights), 4, p(x), x.stride(0), p(shared), ctypes.c_void_p(logits.data_ptr() + 8), 3,
                                                  top, tokens, n, p(out), code, kernels._s()) == 0
    rows = torch.where(idx[:, None] < 4, parts.double(), weights.double()[:, None] * x.double().repeat_interleave(top, 0)).view(tokens, top, n)
    want = rows.sum(1) + torch.sigmoid(logits[:, 2:].double()) * shared.double()
    most = rows.abs().sum(1) + shared.double().abs()
    # top + 1 float additions, the sigmoid's few roundings, and the output's own
    assert ((out.double() - want).abs() <= (top + 8) * 2.0 ** -24 * most + (2.0 ** -8 * want.abs() if code else 0.0)).all()
    assert (room[tokens * n:] == 7.0).all()
