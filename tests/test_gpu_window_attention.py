"""Prompt portions on the tensor-memory attention behind a window (with kept first keys and a sink), and over one cached row for all
heads: against the mma.sync kernel's neighbourhood of the torch version, with given-back pages missing and unwritten rows poisoned."""
import math

import pytest
import torch

from tests.test_gpu_kernels import DEV, E, K, _paged_setup  # noqa: F401  (K: the fixture)

pytestmark = pytest.mark.gpu

CASES = [
    # heads, kv, page, q_lens, kv_lens, window, keep
    (4, 1, 64, [300], [300], 64, 0),                       # a window of one tile
    (4, 1, 64, [300], [300], 100, 4),
    (8, 2, 16, [130, 1, 40], [400, 700, 333], 50, 20),     # small pages: kept and passed ones in one tile
    (8, 8, 32, [65, 17], [600, 17], 129, 70),              # kept keys over two tiles
    (16, 4, 128, [257], [1000], 200, 4),                   # pages of two tiles
    (12, 3, 256, [70, 300], [900, 300], 65, 130),          # pages of four tiles
    (6, 2, 64, [200], [200], 1024, 4),                     # a window longer than the sequence
    (16, 1, 64, [70, 2, 1], [333, 500, 90], 90, 0),        # a portion of two tokens beside a decoded one
    (4, 2, 8, [33], [201], 1, 1),                          # a query that sees itself and the first key
]


@pytest.mark.parametrize("d,shared", [(64, False), (128, False), (128, True), (256, True)])
@pytest.mark.parametrize("case", CASES, ids=[f"h{c[0]}kv{c[1]}p{c[2]}w{c[5]}k{c[6]}" for c in CASES])
def test_window_on_the_tensor_memory_path(K, case, d, shared):  # noqa: F811
    heads, kv_heads, page, q_lens, kv_lens, window, keep = case
    if shared:
        kv_heads = 1
    s = _paged_setup("bfloat16", heads, kv_heads, d, page, q_lens, kv_lens)
    assert K._attention_lib(d).sb_attention_tc_supports(heads, kv_heads, page, 1 if shared else 0, s["qkv"].stride(0)) == 1
    if shared:
        s["vc"] = s["kc"]
    for r, (n, L) in enumerate(zip(q_lens, kv_lens)):
        b = (L - 1) // page
        if L % page:                                       # rows of the last page beyond the sequence
            s["kc"][int(s["bt"][r, b]), :, L % page:] = float("nan")
            s["vc"][int(s["bt"][r, b]), :, L % page:] = float("nan")
        for blk in range(-(-keep // page), max(0, L - n - window + 1) // page):      # pages the window has passed: given back, reused
            s["kc"][int(s["bt"][r, blk])] = float("nan")
            s["vc"][int(s["bt"][r, blk])] = float("nan")
            s["bt"][r, blk] = -1
    sinks = torch.randn(heads, device=DEV)
    scale = 1.0 / math.sqrt(d)
    t = sum(q_lens)
    out = torch.full((t, heads * d), float("nan"), device=DEV, dtype=torch.bfloat16)
    want = torch.empty_like(out)
    args = (s["kc"], s["vc"], s["bt"], s["cu"], s["kv"], s["row"], s["pos"], heads, kv_heads, d, page, scale, window)
    K.attention(s["qkv"], *args, out, s["shape"], sinks=sinks, keep_first=keep)
    K.check_errors()
    E.attention(s["qkv"], *args, want, s["shape"], sinks=sinks, keep_first=keep)
    assert bool(torch.isfinite(out).all()), "a row was not written, or NaN"
    # probabilities are rounded to bfloat16 (2^-8 of each): a sum of p v moves by 2^-8 of sum p |v|, at most 2^-8 max |v|; plus the output's
    # own rounding on both sides
    top = float(torch.nan_to_num(s["vc"].float(), 0.0).abs().max())
    torch.testing.assert_close(out.float(), want.float(), atol=2.0 ** -8 * top, rtol=2.0 ** -7)


@pytest.mark.parametrize("d,shared", [(64, False), (128, False), (256, True)])
@pytest.mark.parametrize("page", [16, 64, 128])
@pytest.mark.parametrize("keep", [0, 4])
def test_numbers_no_query_sees_do_not_matter(K, d, shared, page, keep):  # noqa: F811
    """Infinities and NaN at keys that lie behind every query's window and are not kept (beside the kept ones, and in the block of keys
    where the window begins): the result is the one with other numbers there, bit for bit."""
    heads, kv_heads, window = 8, 1 if shared else 2, 100
    s = _paged_setup("bfloat16", heads, kv_heads, d, page, [200], [600])       # queries 400 .. 599 see keys from 301 on
    if shared:
        s["vc"] = s["kc"]
    args = lambda: (s["kc"], s["vc"], s["bt"], s["cu"], s["kv"], s["row"], s["pos"], heads, kv_heads, d, page, 1.0 / math.sqrt(d), window)
    clean = torch.empty((200, heads * d), device=DEV, dtype=torch.bfloat16)
    K.attention(s["qkv"], *args(), clean, s["shape"], keep_first=keep)
    for key, number in ((4, float("nan")), (10, float("inf")), (63, float("-inf")), (256, float("nan")), (290, float("inf")), (300, float("nan"))):
        for cache in (s["kc"], s["vc"]):
            cache[int(s["bt"][0, key // page]), :, key % page] = number
    out = torch.empty_like(clean)
    K.attention(s["qkv"], *args(), out, s["shape"], keep_first=keep)
    K.check_errors()
    assert bool(torch.isfinite(clean).all()) and torch.equal(out, clean)


@pytest.mark.parametrize("d,shared,window", [(64, False, 200), (128, False, 200), (128, True, 200), (256, True, 0), (256, True, 200)])
@pytest.mark.parametrize("sharp", [1.0, 6.0])
def test_no_further_from_64_bits_than_the_mma_kernel(K, d, shared, window, sharp):  # noqa: F811
    """Scores of about unit size and so far apart that single keys have most of the weight: the error against 64 bits is at most that of the
    mma.sync kernel (the two round at different places, so a twentieth is allowed for)."""
    heads, kv_heads, page = 16, 1 if shared else 4, 64
    s = _paged_setup("bfloat16", heads, kv_heads, d, page, [700], [700])
    if shared:
        s["vc"] = s["kc"]
    scale = sharp / math.sqrt(d)
    args = (s["kc"], s["vc"], s["bt"], s["cu"], s["kv"], s["row"], s["pos"], heads, kv_heads, d, page, scale, window)
    q = s["qkv"][:, : heads * d].view(700, heads, d).double()
    gather = lambda cache: cache[s["bt"][0].long()].transpose(1, 2).reshape(-1, kv_heads, d)[:700].double().repeat_interleave(heads // kv_heads, 1)
    k, v = gather(s["kc"]), gather(s["vc"])
    at = torch.arange(700, device=DEV)
    seen = (at[None] <= at[:, None]) & ((at[None] > at[:, None] - window) if window else True)
    p = (torch.einsum("qhd,khd->hqk", q, k) * scale).masked_fill(~seen[None], -math.inf).softmax(-1)
    want = torch.einsum("hqk,khd->qhd", p, v).reshape(700, heads * d)
    errors = []
    for tensor_memory in (True, False):
        out = torch.empty((700, heads * d), device=DEV, dtype=torch.bfloat16)
        K.use_tcgen05_attention = tensor_memory
        try:
            K.attention(s["qkv"], *args, out, s["shape"])
        finally:
            K.use_tcgen05_attention = True
        errors.append(float((out.double() - want).norm() / want.norm()))
    K.check_errors()
    assert errors[0] <= 1.05 * errors[1], errors


@pytest.mark.parametrize("d,shared", [(64, False), (128, False), (128, True), (256, True)])
@pytest.mark.parametrize("page", [16, 64, 192, 256])
@pytest.mark.parametrize("window", [0, 333])
@pytest.mark.parametrize("q_lens,kv_lens", [([129, 40], [129, 400]), ([900, 850], [900, 1000])], ids=["few", "many"])
def test_references_that_move(K, d, shared, page, window, q_lens, kv_lens):  # noqa: F811
    """Keys that grow along the sequence, a stronger one in either half of a tile in turn: the reference of a row's exponentials moves in tile
    after tile, seen by one of the row's two threads only, and the accumulator is rescaled with it. With many tiles of rows the form
    of head size 128 that shares an SM is taken, with few the other one."""
    heads, kv_heads = (16, 1) if shared else (16, 8)
    s = _paged_setup("bfloat16", heads, kv_heads, d, page, q_lens, kv_lens)
    for r, L in enumerate(kv_lens):
        for key in range(0, L, 41):                        # 41 and the tile's 64 keys have no common divisor: every place of both halves
            s["kc"][int(s["bt"][r, key // page]), :, key % page] *= 1.0 + key / 100.0
    if shared:
        s["vc"] = s["kc"]
    scale, t = 1.0 / math.sqrt(d), sum(q_lens)
    out = torch.full((t, heads * d), float("nan"), device=DEV, dtype=torch.bfloat16)
    want = torch.empty_like(out)
    args = (s["kc"], s["vc"], s["bt"], s["cu"], s["kv"], s["row"], s["pos"], heads, kv_heads, d, page, scale, window)
    K.attention(s["qkv"], *args, out, s["shape"])
    K.check_errors()
    E.attention(s["qkv"], *args, want, s["shape"])
    assert bool(torch.isfinite(out).all()), "a row was not written, or NaN"
    # as above; the reference attention's scores and weights are 32-bit, so what differs is the weights' rounding (2^-8 of each) and both outputs'
    top = float(s["vc"].float().abs().max())
    torch.testing.assert_close(out.float(), want.float(), atol=2.0 ** -8 * top, rtol=2.0 ** -7)
