"""The composite easy leaves of large y, whose m go through a list (more than
2^17 chunks of 1024 m over all levels) or come from the mu*lpf table (fewer):
the terms of published pi(10^k) sum to it, alone, in a batch of different y and
with the 128-bit kernels.  Tolerance zero."""
import pytest

pytestmark = pytest.mark.gpu

PI = {14: 3204941750802, 15: 29844570422669, 16: 279238341033925}


@pytest.mark.parametrize("k,alpha", [(14, 40), (14, 150), (15, 24), (15, 48), (15, 100), (16, 60)])
@pytest.mark.parametrize("wide", [False, True])
def test_terms_sum_to_pi(ctx, cpx, k, alpha, wide):
    x = 10**k
    t = cpx.terms_batch([x], [cpx.default_y(x, alpha)], wide=wide, ctx=ctx)[0]
    assert t["pi"] == PI[k], (k, alpha, wide)


def test_list_over_queries_of_different_y(ctx, cpx):
    xs = [10**15, 10**14, 10**15, 10**16]
    ys = [cpx.default_y(x, a) for x, a in zip(xs, (90, 30, 20, 40))]
    got = cpx.terms_batch(xs, ys, ctx=ctx)
    assert [t["pi"] for t in got] == [PI[15], PI[14], PI[15], PI[16]]
    for x, y, t in zip(xs, ys, got):  # as each alone
        assert t["easy"] == cpx.S2_easy(x, y, 6, ctx=ctx)
