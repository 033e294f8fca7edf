"""Which steps of the linear recurrences run 32 tokens at a time: the rule against both kernels' times on a B200."""
import pytest

from serve_b200.kernels.cuda import chunks_pay

# mode, a decay a head, rows and columns of the state, heads, requests, tokens of each; us chunked, us walked
MEASURED = [
    ("decay", False, 128, 128, 16, 1, 1024, 80, 257), ("decay", False, 128, 128, 16, 8, 256, 126, 211),
    ("decay", False, 64, 64, 32, 16, 128, 130, 123), ("decay", False, 64, 64, 16, 16, 256, 124, 130),
    ("decay", False, 16, 64, 16, 16, 200, 105, 66), ("decay", False, 64, 64, 16, 4, 200, 37, 54), ("delta", True, 128, 128, 16, 1, 97, 28, 42),
    ("delta", True, 128, 128, 32, 16, 256, 670, 1220), ("delta", True, 64, 64, 32, 16, 200, 318, 257),
    ("delta", True, 16, 64, 16, 16, 256, 195, 92), ("delta", True, 64, 128, 16, 16, 161, 199, 194), ("delta", True, 64, 64, 8, 1, 161, 27, 55),
    ("delta", False, 64, 64, 32, 16, 256, 613, 351), ("delta", False, 16, 64, 16, 4, 1024, 315, 230),
    ("delta", False, 64, 128, 32, 4, 200, 166, 136), ("delta", False, 128, 128, 16, 1, 512, 74, 187),
    ("delta", False, 64, 64, 16, 1, 1024, 107, 311), ("delta", False, 128, 128, 32, 16, 256, 941, 1241),
    ("wkv", False, 64, 64, 16, 1, 512, 40, 124), ("wkv", False, 64, 64, 16, 16, 161, 109, 106), ("wkv", False, 128, 128, 32, 16, 200, 504, 835),
    ("gla", False, 16, 64, 16, 16, 256, 128, 88), ("gla", False, 64, 64, 32, 16, 128, 150, 159), ("ssm", False, 64, 64, 32, 16, 161, 160, 138),
    ("ssm", False, 64, 128, 16, 4, 1024, 144, 275), ("retention", False, 64, 64, 32, 16, 200, 203, 180),
    ("retention", False, 128, 128, 32, 1, 512, 68, 156),
]
# mode, a decay a head, rows and columns of the state, heads, tokens of the longest request, of all; us chunked, us walked: short, ragged requests
RAGGED = [
    ("delta", False, 48, 64, 24, 56, 551, 95, 50), ("wkv", False, 32, 64, 16, 47, 113, 22, 14), ("ssm", False, 64, 256, 4, 55, 476, 36, 24),
    ("decay", False, 100, 64, 16, 61, 396, 42, 35), ("retention", False, 32, 192, 24, 74, 586, 71, 40),
    ("delta", True, 96, 16, 12, 62, 268, 38, 30), ("gla", False, 24, 128, 8, 121, 404, 24, 31), ("ssm", False, 48, 64, 4, 93, 609, 19, 25),
    ("delta", False, 48, 192, 12, 122, 203, 40, 47), ("wkv", False, 32, 96, 6, 88, 285, 18, 21), ("decay", False, 100, 256, 20, 75, 221, 52, 64),
    ("gla", False, 32, 256, 6, 138, 1491, 52, 45), ("delta", True, 128, 192, 8, 94, 1049, 110, 143),
    ("retention", False, 32, 96, 6, 138, 464, 20, 30),
]
TIE = 1.08      # times this close are a tie: the rule's form (see RECURRENCE_COST) does not tell such steps apart


def _check(pays, chunked, walked):
    assert (chunked if pays else walked) <= TIE * min(chunked, walked)


@pytest.mark.parametrize("m", MEASURED, ids=lambda m: "-".join(str(x) for x in m[:7]))
def test_the_faster_kernel_is_chosen(m):
    mode, per_head, dk, dv, heads, requests, tokens, chunked, walked = m
    _check(chunks_pay(mode, per_head, dk, dv, heads, tokens, requests * tokens), chunked, walked)


@pytest.mark.parametrize("m", RAGGED, ids=lambda m: "-".join(str(x) for x in m[:7]))
def test_the_faster_kernel_is_chosen_for_short_requests(m):
    mode, per_head, dk, dv, heads, longest, tokens, chunked, walked = m
    _check(chunks_pay(mode, per_head, dk, dv, heads, longest, tokens), chunked, walked)


def test_states_beyond_the_chunked_kernels():
    assert not chunks_pay("decay", False, 129, 64, 8, 4096, 4096)
