"""The mu/lpf sieve in blocks of 4096, 8192 and 16384 odd numbers: the larger
ones against the oracle where it reaches, and against windows small enough for
the smallest blocks, cut at odd places of a block.  Tolerance zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,odd", [(0, 3 * 148 * 8192), (10**7 + 2, 3 * 148 * 8192 + 77)])
def test_blocks_of_8192_equal_oracle(ctx, cpx, orc, lo, odd):
    mu_o, lpf_o = orc.mu_lpf(lo, lo + 2 * odd)
    assert np.array_equal(cpx.gen_h_mu(lo, lo + 2 * odd, ctx=ctx), mu_o)
    assert np.array_equal(cpx.gen_h_lpf(lo, lo + 2 * odd, ctx=ctx), lpf_o)


@pytest.mark.parametrize("lo", [2**34 - 10**7, 2**34 + 2, 2063**2 * 4096 - 100, 10**13])
def test_large_blocks_equal_small_windows(ctx, cpx, lo):
    odd = 2 * 148 * 16384 + 1001
    mu, lpf = (a.to_host() for a in cpx.gen_d_mu_lpf(lo, lo + 2 * odd, ctx=ctx))
    for at, n in ((0, 5000), (16384 - 3, 20011), (odd // 2, 100_003), (odd - 7, 7)):
        m, p = (a.to_host() for a in cpx.gen_d_mu_lpf(lo + 2 * at, lo + 2 * (at + n), ctx=ctx))
        assert np.array_equal(m, mu[at:at + n]) and np.array_equal(p, lpf[at:at + n])
    # and by trial division
    for i in range(0, odd, odd // 40):
        n, k, m = lo + 2 * i + 1, lo + 2 * i + 1, 1
        p = int(lpf[i])
        assert n % p == 0 and all(n % d for d in range(3, min(p, 3000), 2))
        f = 3
        while f * f <= k and m:
            if k % f == 0:
                k //= f
                m = 0 if k % f == 0 else -m
            f += 2
        if m and k > 1:
            m = -m
        assert int(mu[i]) == m, n
