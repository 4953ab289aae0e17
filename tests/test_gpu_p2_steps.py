"""P2 of batches whose warps take 128 primes a step: many queries whose prime
counts end anywhere in a step (from one prime to some 78 thousand), against the
same queries alone (one prime a lane a step) and, for a few, the oracle.
Tolerance zero."""
import math
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,wide", [(1, False), (2, False), (3, True)])
def test_batch_equals_each_alone(ctx, cpx, orc, seed, wide):
    r = random.Random(seed)
    xs, ys = [], []
    for k in range(72):
        x = r.randrange(10**11, 10**12)
        s, c = math.isqrt(x), round(x ** (1 / 3)) + 1
        # y close below sqrt(x): few primes, any remainder; else many
        y = s - r.randrange(20, 40000) if k % 3 == 0 else r.randrange(c, 4 * c)
        xs.append(x)
        ys.append(y)
    got = cpx.terms_batch(xs, ys, wide=wide, ctx=ctx)
    for k, (x, y, t) in enumerate(zip(xs, ys, got)):
        assert t["P2"] == cpx.P2(x, y, ctx=ctx), (x, y)
        if k % 24 < 2:
            assert t["P2"] == orc.P2(x, y), (x, y)
