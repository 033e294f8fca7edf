"""Which steps of the linear recurrences run 32 tokens at a time: the rule against both kernels' times on a B200."""
import pytest

from serve_b200.kernels.cuda import chunks_pay

# mode, a decay a head, rows and columns of the state, heads, requests, tokens of each; us chunked, us walked
MEASURED = [
    ("decay", False, 128, 128, 16, 1, 1024, 82, 260), ("decay", False, 128, 128, 16, 8, 256, 164, 216), ("decay", False, 64, 64, 32, 16, 128, 142, 120),
    ("decay", False, 64, 64, 16, 16, 256, 136, 126), ("decay", False, 16, 64, 16, 16, 200, 116, 66), ("decay", False, 64, 64, 16, 4, 200, 36, 52),
    ("delta", True, 128, 128, 16, 1, 97, 28, 41), ("delta", True, 128, 128, 32, 16, 256, 835, 1247), ("delta", True, 64, 64, 32, 16, 200, 401, 278),
    ("delta", True, 16, 64, 16, 16, 256, 231, 104), ("delta", True, 64, 128, 16, 16, 161, 260, 202), ("delta", True, 64, 64, 8, 1, 161, 26, 54),
    ("delta", False, 64, 64, 32, 16, 256, 692, 366), ("delta", False, 16, 64, 16, 4, 1024, 345, 231), ("delta", False, 64, 128, 32, 4, 200, 190, 139),
    ("delta", False, 128, 128, 16, 1, 512, 76, 190), ("delta", False, 64, 64, 16, 1, 1024, 108, 314), ("delta", False, 128, 128, 32, 16, 256, 1114, 1282),
    ("wkv", False, 64, 64, 16, 1, 512, 41, 124), ("wkv", False, 64, 64, 16, 16, 161, 120, 106), ("wkv", False, 128, 128, 32, 16, 200, 661, 835),
    ("gla", False, 16, 64, 16, 16, 256, 139, 86), ("gla", False, 64, 64, 32, 16, 128, 171, 165), ("ssm", False, 64, 64, 32, 16, 161, 196, 152),
    ("ssm", False, 64, 128, 16, 4, 1024, 202, 289), ("retention", False, 64, 64, 32, 16, 200, 240, 194), ("retention", False, 128, 128, 32, 1, 512, 88, 157),
]


@pytest.mark.parametrize("m", MEASURED, ids=lambda m: "-".join(str(x) for x in m[:7]))
def test_the_faster_kernel_is_chosen(m):
    mode, per_head, dk, dv, heads, requests, tokens, chunked, walked = m
    assert chunks_pay(mode, per_head, dk, dv, heads, tokens, requests * tokens) == (chunked < walked)


def test_states_beyond_the_chunked_kernels():
    assert not chunks_pay("decay", False, 129, 64, 8, 4096, 4096)
