"""Which short prompt portions behind a window leave the tensor-memory attention: the rule against both kernels' times on a B200."""
import pytest

from serve_b200.kernels.cuda import short_on_mma

# longest portion, query heads a kv head, keys a query sees, decoding requests too, (request, kv head) pairs, places; us tensor memory, mma.sync
MEASURED = [
    (16, 4, 16, False, 128, 148, 7.5, 9.1), (16, 4, 16, False, 160, 148, 13.2, 10.3), (6, 4, 6, False, 256, 148, 14.3, 9.4),
    (16, 4, 16, False, 512, 148, 27.5, 19.4), (24, 4, 24, False, 256, 148, 14.9, 18.5), (16, 4, 144, False, 160, 148, 17.7, 17.3),
    (16, 4, 144, False, 256, 148, 19.4, 17.7), (16, 4, 144, False, 320, 148, 27.2, 31.0), (16, 4, 144, False, 512, 148, 37.4, 32.9),
    (16, 4, 416, False, 256, 148, 26.4, 28.5), (16, 4, 1016, False, 512, 148, 88.1, 106.8), (6, 4, 6, False, 16, 148, 7.0, 7.9),
    (16, 4, 144, False, 296, 296, 11.2, 12.4), (16, 4, 144, False, 320, 296, 17.7, 13.6), (24, 4, 152, False, 320, 296, 18.0, 22.3),
    (6, 8, 6, False, 0, 148, 9.9, 11.6), (24, 8, 24, False, 0, 148, 10.0, 14.9),
]


@pytest.mark.parametrize("m", MEASURED, ids=lambda m: "-".join(str(x) for x in m[:6]))
def test_the_faster_kernel_is_chosen(m):
    assert short_on_mma(*m[:6]) == (m[7] < m[6])


def test_beside_decoding_requests():
    """One call from the host instead of two, while the keys are few."""
    assert short_on_mma(6, 4, 6, True, 16, 148) and short_on_mma(2, 8, 20, True, 0, 148)
    assert not short_on_mma(6, 4, 200, True, 16, 148) and not short_on_mma(17, 4, 17, True, 16, 148)
