"""The passes whose exchanges stay inside warps, at the widths and heights where their geometry changes:
CTAs below a warp, of one warp and of several, with and without paired lanes, with one and two middle
stages. Results are whole numbers and must equal GMP's."""
import numpy as np
import pytest

from conftest import random_words
from test_emulator import emu, run  # noqa: F401  (emu is a fixture)

EDGES = [(64, 64), (128, 64), (256, 64), (512, 64), (1024, 64), (2048, 64), (4096, 64),
         (64, 128), (64, 256), (64, 512), (64, 1024), (64, 2048), (64, 4096), (64, 640), (64, 1280), (64, 2560)]


def exponent(W, H, bpw=16.3):
    return int(2 * W * H * bpw) | 1


@pytest.mark.parametrize("W,H,n,flags", [(256, 64, 3, 0), (512, 64, 3, 2), (64, 512, 2, 0)])
def test_emulated_edges(emu, oracle, W, H, n, flags):  # noqa: F811
    E = exponent(W, H)
    _, got = run(emu, "square", E, W, H, n, flags, 9)
    assert np.array_equal(got, oracle.gmp_square(E, random_words(E, 9), n, ll=bool(flags & 2)))


@pytest.mark.parametrize("W", [64, 128, 256, 512, 1024, 2048, 4096])
def test_emulated_records_hold_what_lines_read(emu, oracle, W):  # noqa: F811
    """Making a plan computes only the entries of a line group's record that lines of its width read: with
    every other entry NaN the words are still GMP's."""
    E = exponent(W, 64)
    _, got = run(emu, "square", E, W, 64, 1, 0, 9, OWL_EMU_POISON="1")  # the entry and the exit line pass
    assert np.array_equal(got, oracle.gmp_square(E, random_words(E, 9), 1))


@pytest.mark.parametrize("H", [128, 256, 1024, 2048, 4096])
def test_emulated_column_heights(emu, oracle, H):  # noqa: F811
    """The plain column passes that no other emulated case runs at 16 values a thread."""
    E = exponent(64, H)
    _, got = run(emu, "square", E, 64, H, 1, 0, 9)
    assert np.array_equal(got, oracle.gmp_square(E, random_words(E, 9), 1))


@pytest.mark.gpu
@pytest.mark.parametrize("W,H", EDGES)
def test_edges_vs_gmp(oracle, W, H):
    import gpuowl_b200 as owl
    E = exponent(W, H)
    wa, wb = random_words(E, 21), random_words(E, 22)
    with owl.Plan(E, W=W, H=H) as p:
        a, b = p.alloc(), p.alloc()
        p.writeIn(a, wa)
        p.writeIn(b, wb)
        p.squareLoop(a, a, 18, roe=False)  # a graph: the tags of the carry words alternate
        p.squareLoop(a, a, 3, ll=True)
        p.modMul(a, b)
        want = oracle.gmp_square(E, oracle.gmp_square(E, wa, 18), 3, ll=True)
        assert np.array_equal(p.readOut(a), oracle.gmp_mul(E, want, wb))


@pytest.mark.gpu
@pytest.mark.parametrize("W,H", [(512, 128), (512, 256), (1024, 64), (1024, 128), (128, 1024), (256, 1024)])
def test_register_builds_vs_gmp(oracle, W, H):
    """Both builds of the 64- and 128-thread passes, at the sizes on either side of the lines between them, with
    and without the round-off measurement, and a product."""
    import gpuowl_b200 as owl
    E = exponent(W, H)
    wa, wb = random_words(E, 41), random_words(E, 42)
    with owl.Plan(E, W=W, H=H, column_variant=owl.COL_V16) as p:
        a, b = p.alloc(), p.alloc()
        p.writeIn(a, wa)
        p.writeIn(b, wb)
        p.squareLoop(a, a, 17, roe=False)
        p.squareLoop(a, a, 4)
        assert 0 < p.readROE().max() < 0.3
        p.modMul(a, b)
        assert np.array_equal(p.readOut(a), oracle.gmp_mul(E, oracle.gmp_square(E, wa, 21), wb))
