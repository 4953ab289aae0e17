"""The hard-leaf sieve of one query with blocks of levels crossed off at once:
sub-segments from the smallest (2^12 bits a warp: every block goes at once) to
the largest (2^18: none or only the last blocks do), 64- and 128-bit kernels,
against the oracle's hard leaves.  Whole numbers: tolerance zero."""
import pytest

pytestmark = pytest.mark.gpu

CASES = [(10**8 - 3, 2000), (10**10 + 19, 2155), (10**11, 46415 * 2), (10**12, 10**4), (2**40 + 15, 10**5 + 3),
         (10**13, 172354)]
_WANT = {}


@pytest.mark.parametrize("lbits,threads", [(14, 128), (15, 256), (16, 512), (16, 128), (18, 256), (20, 512), (20, 128)])
def test_blocks_of_levels_equal_oracle(ctx, cpx, orc, lbits, threads):
    for x, y in CASES:
        if (x, y) not in _WANT:
            _WANT[(x, y)] = orc.hard(x, y, 6)
        for wide in (False, True):
            t = cpx.terms_batch([x], [y], hard_log2_bits=lbits, hard_threads=threads, wide=wide, ctx=ctx)[0]
            assert t["hard"] == _WANT[(x, y)], (x, y, lbits, threads, wide)
