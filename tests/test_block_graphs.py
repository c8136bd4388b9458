"""Products that run as graphs (a pair of buffers seen once, again, evicted) and blocks below, at and above
the smallest graph. Whole numbers, against GMP."""
import numpy as np
import pytest

from conftest import random_words

E = 86243


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 15, 16, 17, 300])
@pytest.mark.parametrize("ll,mul3", [(False, False), (True, False), (False, True)])
def test_block_counts(oracle, n, ll, mul3):
    import gpuowl_b200 as owl
    w = random_words(E, 5)
    want = oracle.gmp_square(E, w, n, ll=ll)
    if mul3:
        three = np.zeros_like(want)
        three[0] = 3
        want = oracle.gmp_mul(E, want, three)
    with owl.Plan(E) as p:
        a, b = p.alloc(), p.alloc()
        p.writeIn(a, w)
        for out in (b, b, a):  # the same graph for other buffers, then in place
            p.squareLoop(out, a, n, ll=ll, mul3=mul3, roe=False)
            assert np.array_equal(p.readOut(out), want)
        assert p.readROE().size == 0


@pytest.mark.gpu
def test_repeated_products(oracle):
    import gpuowl_b200 as owl
    ws = [random_words(E, s) for s in (1, 2, 3)]
    with owl.Plan(E) as p:
        bufs = [p.alloc() for _ in ws]
        for b, w in zip(bufs, ws):
            p.writeIn(b, w)
        have = list(ws)
        # pairs seen once, repeated and evicted; a square; a timeout changed in between
        order = [(0, 1)] * 3 + [(0, 2), (1, 0), (1, 2), (2, 0), (2, 1), (0, 1), (0, 1), (2, 2), (2, 2), (2, 2)]
        for i, (x, y) in enumerate(order):
            if i == 2:
                p.set_timeout(1_000_000_000)
            p.modMul(bufs[x], bufs[y], mul3=bool(i % 2))
            have[x] = oracle.gmp_mul(E, have[x], have[y], mul3=bool(i % 2))
            assert np.array_equal(p.readOut(bufs[x]), have[x]), (i, x, y)
        assert p.readROE().size == len(order)
