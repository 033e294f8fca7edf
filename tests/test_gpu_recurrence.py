"""Prompt portions of the linear recurrences 32 tokens at a time (csrc/chunked_recurrence.cu): every mode against 64 bits, beside the
walking kernel, at the edges of chunks, states and value columns, mixed with short requests; decays that vanish; later tokens that
are not finite."""
import types

import pytest
import torch

from tests.emu_kernels import EmuKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
MODES = ["decay", "ssm", "delta", "delta_head", "wkv", "gla", "retention"]


@pytest.fixture(scope="module")
def K():
    from serve_b200.kernels import load_kernels

    return load_kernels(DEV)


def _case(mode, lengths, heads, qk_heads, dk, dv, dtype, seed, listed=True, slow=False):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rn = lambda *s: torch.randn(s, generator=g, device=DEV)
    ru = lambda *s: torch.rand(s, generator=g, device=DEV)
    if mode in ("wkv", "retention"):
        qk_heads = heads
    t, r = sum(lengths), len(lengths)
    wide = rn(t, 2 * qk_heads * dk + heads * dv).to(dtype)             # slices of one buffer, as projections are
    q, k, v = wide[:, : qk_heads * dk], wide[:, qk_heads * dk: 2 * qk_heads * dk], wide[:, 2 * qk_heads * dk:]
    kw = {}
    if mode in ("decay", "retention"):
        kw["decay"] = 1.0 - 2.0 ** (-1.0 - 8.0 * ru(heads))
    if mode == "retention":
        rot = dk // 2 // 8 * 8
        kw.update(inv_freq=1.0 / 10000.0 ** (torch.arange(max(rot // 2, 1), device=DEV).float() / max(rot // 2, 1)), rot_dims=rot, k_scale=dk ** -0.5)
    if mode == "ssm":
        kw.update(aux=rn(t, heads).to(dtype), a_log=(1 + 15 * ru(heads)).log(), dt_bias=rn(heads) - 3.0, d_skip=rn(heads))
    if mode.startswith("delta"):
        cols = heads if mode == "delta_head" else heads * dk
        kw.update(aux=rn(t, heads).to(dtype), rate=rn(t, cols).to(dtype), a_log=(1 + 15 * ru(heads)).log(), dt_bias=rn(cols) - (6.0 if slow else 2.0),
                  q_scale=dk ** -0.5)
        if mode == "delta_head":
            kw["rate_per_head"] = True
    if mode == "wkv":
        kw.update(rate=rn(t, heads * dk), dt_bias=rn(heads * dk) - 2.0, bonus=rn(heads * dk))
    if mode == "gla":
        kw.update(rate=rn(t, heads * dk), dt_bias=rn(heads * dk), q_scale=dk ** -0.5, rate_scale=1.0 / 16.0)
    cu = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32, device=DEV)
    order = sorted(range(r), key=lambda i: -lengths[i])
    shape = types.SimpleNamespace(rows=r, tokens=t, max_q=max(lengths), min_q=min(lengths), pure_decode=False,
                                  rows_by_q=torch.tensor(order, dtype=torch.int32, device=DEV) if listed else None,
                                  neg_q_sorted=tuple(-lengths[i] for i in order) if listed else None)
    rows = torch.repeat_interleave(torch.arange(r, device=DEV), torch.tensor(lengths, device=DEV))
    ctx = types.SimpleNamespace(shape=shape, cu_q=cu, slots=torch.randperm(r + 2, generator=g, device=DEV)[:r].to(torch.int32),
                                positions=(torch.arange(t, device=DEV) - cu[rows]).to(torch.int32) + 5, token_row=rows.to(torch.int32), memo={})
    pool = rn(r + 2, heads * dk * dv + 8) * 0.3                        # states are column slices of a wider tensor
    return types.SimpleNamespace(args=(q, k, v), pool=pool, ctx=ctx, kw=kw, dims=(heads, qk_heads, dk, dv), t=t,
                                 mode="delta" if mode.startswith("delta") else mode)


def _run(kernels, c, chunked=True, out_dtype=torch.float32):
    heads, qk_heads, dk, dv = c.dims
    pool = c.pool.clone()
    state = pool[:, 4: 4 + heads * dk * dv].view(-1, heads, dk, dv)
    out = torch.full((c.t, heads * dv), float("nan"), device=DEV, dtype=out_dtype)
    c.ctx.memo.clear()
    before = getattr(kernels, "use_chunked_recurrence", None)
    if before is not None:
        kernels.use_chunked_recurrence, kernels.use_chunked_retention, kernels.CHUNKS_FROM = chunked, False, 32
        kernels.use_chunk_rule = False
    try:
        kernels.linear_recurrence(c.mode, *c.args, state, c.ctx, out, heads, qk_heads, dk, dv, **c.kw)
    finally:
        if before is not None:
            kernels.use_chunked_recurrence, kernels.use_chunked_retention = before, True
            del kernels.CHUNKS_FROM, kernels.use_chunk_rule                       # (the class's again)
    return out, pool


def _exact(c):
    heads, qk_heads, dk, dv = c.dims
    pool = c.pool.double()
    state = pool[:, 4: 4 + heads * dk * dv].view(-1, heads, dk, dv)
    out = torch.empty((c.t, heads * dv), device=DEV, dtype=torch.float64)
    EmuKernels(DEV, torch.float64).linear_recurrence(c.mode, *c.args, state, c.ctx, out, heads, qk_heads, dk, dv, **c.kw)
    return out, pool


def _error(got, want):
    return float((got.double() - want).norm() / want.norm())


SIZES = [
    # lengths, heads, qk heads, dk, dv, dtype, listed
    ([33], 1, 1, 128, 128, torch.bfloat16, True),
    ([64, 32, 1, 95], 2, 1, 64, 40, torch.bfloat16, True),                 # a whole number of chunks, a walked one, a ragged one
    ([40, 100, 33], 4, 2, 72, 16, torch.float32, False),                    # no list: requests in order
    ([2, 161, 5, 34], 3, 3, 16, 72, torch.bfloat16, True),
    ([300, 128], 2, 2, 100, 130, torch.float32, True),
    ([161, 100, 170, 160], 26, 13, 16, 24, torch.bfloat16, True),          # many pairs
]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("size", SIZES, ids=[f"n{len(s[0])}dk{s[3]}dv{s[4]}" for s in SIZES])
def test_chunks_against_64_bits_and_the_walk(K, mode, size):
    lengths, heads, qk_heads, dk, dv, dtype, listed = size
    c = _case(mode, lengths, heads, qk_heads, dk, dv, dtype, seed=dk + dv, listed=listed)
    want, want_pool = _exact(c)
    out, pool = _run(K, c)
    walked, walked_pool = _run(K, c, chunked=False)
    K.check_errors()
    # a sum of n terms in float is off by at most n 2^-24 of its absolute terms; of the sums here (dk or 32 terms, chunk after chunk)
    # neighbouring ones cancel like random numbers, so a few times sqrt(dk) 2^-24 of the whole (2-norms) stays far above both kernels
    bound = 8 * dk ** 0.5 * 2.0 ** -24 + 2e-7
    for got, ref in ((out, want), (pool, want_pool), (walked, want), (walked_pool, want_pool)):
        assert _error(got, ref) < bound
    untouched = [i for i in range(pool.shape[0]) if i not in c.ctx.slots.tolist()]
    assert torch.equal(pool[untouched], c.pool[untouched])
    assert torch.equal(pool[:, :4], c.pool[:, :4]) and torch.equal(pool[:, -4:], c.pool[:, -4:])


@pytest.mark.parametrize("mode", MODES)
def test_a_later_token_does_not_reach_back(K, mode):
    c = _case(mode, [100], 2, 2, 64, 48, torch.bfloat16, seed=3)
    first, _ = _run(K, c)
    c.args[2][71, 5] = float("inf")                                        # a value inside the third chunk
    c.args[1][80, 7] = float("nan")
    out, _ = _run(K, c)
    assert torch.equal(out[:64], first[:64])
    # the chunk that meets such a number takes its sums in another order: both orders are within the bound above of the exact sums
    bound = 2 * (8 * 64 ** 0.5 * 2.0 ** -24 + 2e-7)
    assert _error(out[64:71], first[64:71]) < bound
    heads, _, _, dv = c.dims
    clean = [j for j in range(dv) if j != 5]
    assert _error(out[71:80][:, clean], first[71:80][:, clean]) < bound    # the columns of S never meet
    assert not torch.isfinite(out[71, 5]) and torch.isnan(out[81, :dv]).all()


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("dk,dv", [(128, 128), (100, 72), (100, 40), (64, 128), (40, 136)])
def test_many_pairs(K, mode, dk, dv):
    """So many (request, head) pairs that blocks walk 32 or 64 columns of S: ragged requests, part of a block's columns beyond the last, an
    infinity in the values of one request."""
    heads = 26
    c = _case(mode, [161, 33, 100, 64, 40, 5], heads, 13, dk, dv, torch.bfloat16, seed=dk + dv)
    want, want_pool = _exact(c)
    out, pool = _run(K, c)
    bound = 8 * dk ** 0.5 * 2.0 ** -24 + 2e-7              # as above
    assert _error(out, want) < bound and _error(pool, want_pool) < bound
    untouched = [i for i in range(pool.shape[0]) if i not in c.ctx.slots.tolist()]
    assert torch.equal(pool[untouched], c.pool[untouched])
    c.args[2][70, dv + 5] = float("inf")                   # the second head of the first request, inside its third chunk
    later, _ = _run(K, c)
    K.check_errors()
    hit = torch.zeros_like(out, dtype=torch.bool)
    hit[70:161, dv: 2 * dv] = True
    assert _error(later[~hit], out[~hit].double()) < 2 * bound and not torch.isfinite(later[70, dv + 5])
    others = [dv + j for j in range(dv) if j != 5]         # the columns of S never meet
    assert _error(later[:161][:, others], out[:161][:, others].double()) < 2 * bound


@pytest.mark.parametrize("mode", ["delta", "wkv", "gla"])
def test_decays_that_vanish(K, mode):
    """Rates so high that products of decays underflow inside a chunk, beside rows that hardly decay."""
    c = _case(mode, [150], 2, 2, 64, 32, torch.float32, seed=11)
    t, cols = c.kw["rate"].shape
    fast = torch.rand((t, cols), device=DEV) < 0.2
    c.kw["rate"] = torch.where(fast, -2000.0 if mode == "gla" else (6.0 if mode == "wkv" else 200.0), c.kw["rate"]).contiguous()
    want, want_pool = _exact(c)
    out, pool = _run(K, c)
    assert _error(out, want) < 1e-5 and _error(pool, want_pool) < 1e-5


@pytest.mark.parametrize("mode", ["ssm", "delta_head"])
@pytest.mark.parametrize("dk", [64, 128])
def test_first_decays_of_a_chunk(K, mode, dk):
    """Decays that differ from token to token, those of a chunk's first two tokens far from the chunk's product and from the others: a lane
    that read the product in the place of one of them would carry it into every later token."""
    c = _case(mode, [1024, 97], 4, 2, dk, 32, torch.float32, seed=17)
    rate = c.kw["aux" if mode == "ssm" else "rate"]
    start = torch.arange(c.t, device=DEV)
    start = torch.where(start < 1024, start, start - 1024) % 32
    rate[start == 0] = -9.0
    rate[start == 1] = 2.0
    want, want_pool = _exact(c)
    bound = 8 * dk ** 0.5 * 2.0 ** -24 + 2e-7              # as above
    for _ in range(5):
        out, pool = _run(K, c)
        assert _error(out, want) < bound and _error(pool, want_pool) < bound


@pytest.mark.parametrize("mode", ["decay", "delta"])
def test_a_device_without_room_for_the_chunks(K, mode, monkeypatch):
    """Pages and weights may fill the device: a step that cannot have the chunks' work space is walked."""
    c = _case(mode, [150, 20], 2, 2, 64, 32, torch.bfloat16, seed=5)
    want, want_pool = _run(K, c, chunked=False)
    empty, asked = torch.empty, []

    def full(*args, **kwargs):
        asked.append(args)
        if len(asked) == 2:                                                # (the first is the walk's own)
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*args, **kwargs)

    monkeypatch.setattr(torch, "empty", full)
    out, pool = _run(K, c)
    monkeypatch.undo()
    assert len(asked) == 2 and torch.equal(out, want) and torch.equal(pool, want_pool)


def _in_steps(kernels, c, row, cuts):
    """Request ``row`` of a case alone, its tokens brought in portions that end at ``cuts``."""
    heads, _, dk, dv = c.dims
    cu = c.ctx.cu_q.tolist()
    outs, state, begin = [], c.pool[int(c.ctx.slots[row])][None].clone(), cu[row]
    for end in [cu[row] + x for x in cuts] + [cu[row + 1]]:
        one = types.SimpleNamespace(**vars(c))
        n = end - begin
        ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        shape = types.SimpleNamespace(rows=1, tokens=n, max_q=n, min_q=n, pure_decode=False, rows_by_q=ints([0]), neg_q_sorted=(-n,))
        one.ctx = types.SimpleNamespace(shape=shape, cu_q=ints([0, n]), slots=ints([0]), positions=c.ctx.positions[begin:end].contiguous(),
                                        token_row=ints([0] * n), memo={})
        part = lambda x: x[begin:end] if torch.is_tensor(x) and x.dim() == 2 and x.shape[0] == c.t else x
        one.args, one.kw = tuple(part(x) for x in c.args), {k: part(v) for k, v in c.kw.items()}
        one.pool, one.t = state, n
        out, state = _run(kernels, one)
        outs.append(out)
        begin = end
    return torch.cat(outs), state


@pytest.mark.parametrize("mode", MODES)
def test_cuts_and_company_change_no_more_than_the_rounding(K, mode):
    """A prompt whole beside others, alone, and in portions (chunks of its own, then walked tokens, then chunks that begin elsewhere): the
    sums are added up in another order each time, so all of them are within the bound above of the exact ones, and no further."""
    c = _case(mode, [333, 40, 5], 3, 3, 64, 48, torch.float32, seed=23)
    n, bound = 333, 2 * (8 * 64 ** 0.5 * 2.0 ** -24 + 2e-7)
    out, pool = _run(K, c)
    state = pool[int(c.ctx.slots[0])][None]
    for cuts in ([], [100], [7, 170, 180]):
        alone, after = _in_steps(K, c, 0, cuts)
        assert _error(alone, out[:n].double()) < bound and _error(after, state.double()) < bound
