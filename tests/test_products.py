"""Products (the first runs directly, those after it with the same buffers as a graph) and powers, at shapes
whose passes start in different ways: column passes of several waves, passes that let the next one start
late (2048 points and more), radix-20 columns and the split-precision passes. Whole numbers, against GMP."""
import numpy as np
import pytest

from conftest import random_words

SHAPES = [(512, 512, 0), (4096, 64, 0), (64, 4096, 0), (64, 2560, 0), (2048, 1280, 0), (2048, 2048, 0),
          (64, 2048, 1), (64, 2560, 1), (2048, 64, 2)]


def power(oracle, E, a, h):
    r = a
    for bit in bin(h)[3:]:
        r = oracle.gmp_square(E, r, 1)
        if bit == "1":
            r = oracle.gmp_mul(E, r, a)
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,split", SHAPES)
def test_power_vs_gmp(oracle, W, H, split):
    import gpuowl_b200 as owl
    E = int(2 * W * H * 16.3) | 1
    wa, wb = random_words(E, 31), random_words(E, 32)
    # the large shapes take a short power (GMP needs 0.4 to 0.7 s a product there)
    h = 0b101 if W * H > 1 << 20 else 0xd6
    with owl.Plan(E, W=W, H=H, split=split) as p:
        a, b = p.alloc(), p.alloc()
        p.writeIn(a, wa)
        p.writeIn(b, wb)
        p.expMul(a, h, b)
        assert np.array_equal(p.readOut(a), oracle.gmp_mul(E, power(oracle, E, wa, h), wb))
        assert np.array_equal(p.readOut(b), wb)


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,split", SHAPES)
def test_repeated_products_vs_gmp(oracle, W, H, split):
    import gpuowl_b200 as owl
    E = int(2 * W * H * 16.3) | 1
    have, wb = random_words(E, 33), random_words(E, 34)
    with owl.Plan(E, W=W, H=H, split=split) as p:
        a, b = p.alloc(), p.alloc()
        p.writeIn(a, have)
        p.writeIn(b, wb)
        for i in range(3):  # direct, captured and launched, launched again
            p.modMul(a, b, mul3=(i == 1))
            have = oracle.gmp_mul(E, have, wb, mul3=(i == 1))
            assert np.array_equal(p.readOut(a), have), i
        assert np.array_equal(p.readOut(b), wb)
