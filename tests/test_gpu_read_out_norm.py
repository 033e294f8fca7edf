"""The norm and gate of recurrent read-outs (csrc/sequence_ops.cu) on the kernels that keep a group in registers and on the general one,
against 64 bits: sizes at the edges of a warp's and a block's share, gate first or last, weights that repeat, strided rows."""
import pytest
import torch

from tests.emu_kernels import EmuKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def K():
    from serve_b200.kernels import load_kernels

    return load_kernels(DEV)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("gate", [None, "sigmoid", "silu_first"])
@pytest.mark.parametrize("channels,groups,weight", [(512, 1, 512), (516, 1, 516), (1024, 2, 512), (2048, 1, 2048), (2044, 1, None),
                                                    (4096, 2, 4096), (2052, 1, 2052), (1032, 1, 1032), (96, 3, 32), (1026, 1, 1026),
                                                    (3072, 2, 512)])
def test_norm_and_gate(K, channels, groups, weight, gate, dtype):
    g = torch.Generator(device=DEV).manual_seed(channels + groups)
    rn = lambda *s: torch.randn(s, generator=g, device=DEV)
    t = 9
    y = rn(t, channels + 4)[:, :channels] * 3.0
    z = rn(t, channels + 8)[:, :channels].to(dtype) if gate else None
    w = rn(weight).to(dtype) if weight else None
    out = torch.full((t, channels + 8), 7.0, device=DEV, dtype=dtype)
    kw = dict(groups=groups, eps=1e-5, weight=w, gate=z, gate_act="silu" if gate == "silu_first" else "sigmoid", gate_first=gate == "silu_first", scale=0.5)
    K.gated_norm(y, out[:, :channels], **kw)
    want = torch.empty((t, channels), device=DEV, dtype=torch.float64)
    EmuKernels(DEV, torch.float64).gated_norm(y, want, **kw)
    # float: sums of at most 4,096 squares, all positive, in lanes (16 terms each, then 7 or fewer halvings and the square root halves the
    # error) plus eight roundings and the exponential: below 40 of 2^-24; then one rounding to the result's type
    bound = 40 * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
    assert bool(((out[:, :channels].double() - want).abs() <= bound * want.abs() + 1e-30).all())
    assert bool((out[:, channels:] == 7.0).all())
