"""The easy leaves on both sides of their 32-bit quotients: at x = 10^19 the
smallest p have quotients above 2^31 and the others below, at 10^18 and below
every quotient is, and x/p lies on both sides of 2^40 and of 2^53 (the last with
the 128-bit kernels at 10^19 too).  Published pi(10^k); tolerance zero."""
import pytest

pytestmark = pytest.mark.gpu

PI = {16: 279238341033925, 17: 2623557157654233, 18: 24739954287740860, 19: 234057667276344607}


@pytest.mark.parametrize("k,alpha,wide", [(16, 12, True), (17, 16, False), (18, 20, False), (18, 48, True), (19, 40, False),
                                          (19, 90, False), (19, 60, True)])
def test_terms_sum_to_pi(ctx, cpx, k, alpha, wide):
    x = 10**k
    t = cpx.terms_batch([x], [cpx.default_y(x, alpha)], wide=wide, ctx=ctx)[0]
    assert t["pi"] == PI[k], (k, alpha, wide)
