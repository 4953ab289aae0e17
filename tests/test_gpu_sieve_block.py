"""The block sieve of the prime counts, the pi tables and phi(x, a) where its
parts meet: the primes of the patterns (to 61), of a warp each (to 2053) and of
a thread each, the ends of a range inside a word, and blocks of 2^19, 2^20 and
2^21 numbers, against the oracle and published counts.  Tolerance zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a", [1, 2, 6, 7, 17, 18, 19, 20, 309, 310, 311, 312, 5000])
@pytest.mark.parametrize("x", [1, 61, 67 * 67, 2**19 - 1, 2**19, 2**21 + 1, 5_000_003])
def test_phi_at_the_bounds(ctx, cpx, orc, x, a):
    assert cpx.Phi(0, ctx=ctx).phi_std(x, a) == orc.phi(x, a)


def test_phi_in_blocks_of_2_20(ctx, cpx, orc):
    x = 3 * 148 * 2**20 + 12345
    for a in (5, 100):
        assert cpx.Phi(0, ctx=ctx).phi_std(x, a) == orc.phi(x, a)


@pytest.mark.parametrize("lo,hi", [(0, 3), (2, 68), (61, 67), (2053, 2064), (4_255_968, 4_255_970), (10**9 - 63, 10**9 + 1),
                                   (2**33 + 1, 2**33 + 2**19 + 2), (2**41 - 5, 2**41 + 70)])
def test_count_at_the_bounds(cpx, orc, lo, hi):
    own = cpx.Context(0)  # no resident table: counted block by block
    cpx.get_device_primes(2**41, 2**41 + 2, ctx=own)
    assert cpx.count_primes(lo, hi, ctx=own) == len(orc.primes(lo, hi))
    own.close()


def test_counts_in_large_blocks(cpx):
    own = cpx.Context(0)
    cpx.get_device_primes(2 * 10**10, 2 * 10**10 + 2, ctx=own)
    assert cpx.count_primes(10**10, 2 * 10**10, ctx=own) == 882206716 - 455052511  # pi(2e10) - pi(1e10)
    assert cpx.count_primes(0, 10**9, ctx=own) == 50847534
    own.close()


@pytest.mark.parametrize("base,rng", [(0, 6), (0, 2**19 + 2), (10**9, 30), (2**33 - 2, 2**20 + 6)])
def test_pi_window_four_outputs_a_thread(ctx, cpx, orc, base, rng):
    t = cpx.PiTable(base, 0, rng, ctx=ctx).getCurrent().to_host()
    ps = orc.primes(base, base + rng + 8)
    n = base - 1 + 2 * np.arange(rng // 2 + 2, dtype=np.int64)
    assert np.array_equal(t, np.searchsorted(ps, n, side="right"))
