"""The kernels around the recurrences over prompt portions: the short convolution with a run of tokens a thread, and what the recurrences
read of queries, keys and decays in pieces of four, against the torch versions."""
import types

import pytest
import torch

from tests.emu_kernels import EmuKernels
from tests.test_gpu_recurrence import DEV, K, _case, _error, _exact, _run  # noqa: F401  (K: the fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("bias,activation,residual", [(True, "silu", False), (False, "none", True)])
@pytest.mark.parametrize("lengths,channels,runs", [([1, 9, 2, 1000, 3, 8, 16, 1, 1, 2007], 2048, None), ([1, 9, 2, 700, 3, 8, 16, 1, 1, 0], 2048, True),
                                                   ([1, 1, 13, 2, 0], 1032, True), ([4096], 1032, None), ([5, 6], 64, False)])
def test_convolution_over_runs_of_tokens(K, taps, bias, activation, residual, lengths, channels, runs):  # noqa: F811
    """Requests that begin inside a run of eight tokens, ones shorter than the filter, a count of tokens that is no multiple of a run; the state's
    inputs before the first tokens. Few tokens take a thread each. Whether a step is taken in runs depends on the GPU's size: a last request of 0
    tokens stands for as many as make it one that is, all but a token of a run."""
    wide, places = -(-channels // 1024), 4 * torch.cuda.get_device_properties(0).multi_processor_count
    if lengths[-1] == 0:
        lengths = lengths[:-1] + [8 * (places * 9 // 10 // wide) - 1 - sum(lengths)]
    blocks = -(-sum(lengths) // 8) * wide
    if runs is not None:                                                # (the rule of sb_causal_conv)
        assert (blocks * 10 >= -(-blocks // places) * places * 7) == runs
    g = torch.Generator(device=DEV).manual_seed(taps + channels)
    rn = lambda *s: torch.randn(s, generator=g, device=DEV)
    t, r = sum(lengths), len(lengths)
    wide = rn(t, channels + 24).to(torch.bfloat16)                      # columns of a wider buffer
    x, w = wide[:, 8: 8 + channels], rn(channels, taps).to(torch.bfloat16)
    b = rn(channels).to(torch.bfloat16) if bias else None
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    rows = [i for i, n in enumerate(lengths) for _ in range(n)]
    ctx = types.SimpleNamespace(shape=types.SimpleNamespace(rows=r, tokens=t, max_q=max(lengths), min_q=min(lengths), pure_decode=False),
                                cu_q=ints(cu), token_row=ints(rows), slots=torch.randperm(r + 1, generator=g, device=DEV)[:r].to(torch.int32))
    states = [rn(r + 1, taps - 1, channels)]
    states.append(states[0].clone())
    outs = [torch.full((t, channels), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    K.causal_conv(x, w, b, states[0], ctx, outs[0], activation=activation, residual=residual)
    EmuKernels(DEV, torch.float64).causal_conv(x, w, b, states[1], ctx, outs[1], activation=activation, residual=residual)
    # both round to bfloat16 once; the float sums of at most five terms may land on the other side of a rounding's edge
    torch.testing.assert_close(outs[0].float(), outs[1].float(), rtol=2.0 ** -7, atol=1e-5)
    assert torch.equal(states[0], states[1])


@pytest.mark.parametrize("mode", ["decay", "ssm", "delta", "delta_head", "gla"])
@pytest.mark.parametrize("dk,dtype", [(16, torch.float32), (132, torch.bfloat16), (256, torch.bfloat16), (388, torch.float32), (512, torch.bfloat16), (30, torch.bfloat16)])
def test_what_the_walk_reads(K, mode, dk, dtype):  # noqa: F811
    """States of one to four pieces of 128 rows, token counts that are no multiple of a warp's tokens; 30 rows are no whole pieces."""
    c = _case(mode, [3, 1, 6], 3, 3, dk, 40, dtype, seed=dk)
    want, want_pool = _exact(c)
    out, pool = _run(K, c, chunked=False)
    bound = 8 * dk ** 0.5 * 2.0 ** -24 + 2e-7              # (see the chunks' test)
    assert _error(out, want) < bound and _error(pool, want_pool) < bound


@pytest.mark.parametrize("mode", ["decay", "ssm", "delta", "delta_head", "gla"])
@pytest.mark.parametrize("dk", [16, 48, 100, 128])
def test_what_the_walk_reads_of_many_tokens(K, mode, dk):  # noqa: F811
    """From 8,192 (token, head) pairs on a warp takes four tokens of up to 128 rows: requests that begin inside such a run, a last run of one."""
    lengths = [100, 1, 150, 6]
    c = _case(mode, lengths, 32, 32, dk, 40, torch.bfloat16, seed=dk)
    assert sum(lengths) * 32 >= 8192 and sum(lengths) % 4 == 1
    want, want_pool = _exact(c)
    bound = 8 * dk ** 0.5 * 2.0 ** -24 + 2e-7              # (see the chunks' test)
    for chunked in (False, True):                          # walked; the two longer requests in chunks
        out, pool = _run(K, c, chunked=chunked)
        assert _error(out, want) < bound and _error(pool, want_pool) < bound
