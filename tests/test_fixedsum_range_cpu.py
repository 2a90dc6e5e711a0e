"""Fixed-point sums at the small end of the doubles (rocflu_gb300/csrc/fixedsum.h)."""
import pytest

from test_fixedsum_cpu import _run, prog  # noqa: F401


@pytest.mark.parametrize("weight", [-400, -410, -420, -430, -490])
def test_small_sums_stay_in_the_doubles(prog, weight):  # noqa: F811
    """The smallest values the sums take, 2^-499, and their differences down to
    one unit, with small weights: the exact sum, or the block is left to FP64
    where a sum's exponent could leave the normal doubles."""
    w, v = 2.0 ** weight, 2.0 ** -499
    up = v * (1 + 2.0 ** -52)
    for q, ws, want in (([2 * v, 3 * v], [1.0, 2.0], 5.0), ([up], [1.0], 2.0 ** -52),
                        ([v, up], [1.0, 2.0 ** -54], 2.0 ** -106)):
        got = _run(prog, [(v, q, [w * x for x in ws])])[0]
        if got == "bad":
            assert weight < -412
        else:
            assert float.fromhex(got) / w / v == want
