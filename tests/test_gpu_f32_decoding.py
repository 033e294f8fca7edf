"""The float32 path's decoding kernels at their edges: keys shared out over blocks (with every option of the scores, short and long
requests side by side, several tokens a request) and the few-rows product (columns, rows and k beyond whole tiles), against 64 bits."""
import math

import pytest
import torch

from tests.emu_kernels import EmuKernels
from tests.test_gpu_kernels import DEV, K, _paged_setup  # noqa: F401  (K: the fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [{}, {"window": 100, "keep_first": 5}, {"softcap": 3.0, "sinks": True}, {"slopes": True, "chunk": 256}])
@pytest.mark.parametrize("heads,kv_heads,d,page,q_lens,kv_lens", [
    (8, 2, 64, 64, [1, 1, 1], [2000, 1, 129]),                 # a long request, one key, one key in the second share
    (6, 1, 48, 24, [2, 1], [700, 333]),                        # 12 rows in a tile, pages that are no power of two
    (4, 4, 256, 16, [1, 3], [1025, 140]),
    (16, 8, 128, 64, [1] * 40, [100 + 7 * i for i in range(40)]),      # too many pairs to share keys out
])
def test_decoding_attention_with_shared_out_keys(K, heads, kv_heads, d, page, q_lens, kv_lens, opts):  # noqa: F811
    s = _paged_setup("float32", heads, kv_heads, d, page, q_lens, kv_lens)
    o = dict(opts)
    window = o.pop("window", 0)
    if o.pop("sinks", False):
        o["sinks"] = torch.randn(heads, device=DEV)
    if o.pop("slopes", False):
        o["slopes"] = torch.rand(heads, device=DEV) * 0.05
    out = torch.full((sum(q_lens), heads * d), float("nan"), device=DEV)
    want = torch.empty_like(out, dtype=torch.float64)
    args = (s["qkv"], s["kc"], s["vc"], s["bt"], s["cu"], s["kv"], s["row"], s["pos"], heads, kv_heads, d, page, 1.0 / math.sqrt(d), window)
    K.attention(*args, out, s["shape"], **o)
    EmuKernels(DEV, torch.float64).attention(*args, want, s["shape"], **o)
    # scores of at most 6 are off by d 2^-24 of their absolute terms (about 3e-6), weights by as much of themselves, and the sums of up to
    # 2,000 weights and of weights times values (below 5) by 2^-24 of themselves a step, mostly cancelling
    torch.testing.assert_close(out.double(), want, atol=5e-5, rtol=0)


@pytest.mark.parametrize("m", [1, 8, 9, 32])
@pytest.mark.parametrize("n,k", [(1, 4), (7, 100), (130, 512), (2500, 516), (9472, 644), (2368, 2052)])
def test_few_rows_product(K, m, n, k):  # noqa: F811
    a, w = torch.randn(m, k, device=DEV), torch.randn(n, k, device=DEV)
    out = torch.full((m, n), float("nan"), device=DEV)
    K.linear(a, w, out)
    want = a.double() @ w.double().T
    # a sum of k products is off by at most k 2^-24 of its absolute terms
    assert ((out.double() - want).abs() <= (k + 8) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)).all()
