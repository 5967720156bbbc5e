"""The block fixed-point transforms: every line length, values at the ends of
a double's range, and non-finite right-hand sides."""
import numpy as np
import pytest

from oracle import ns_oracle as O
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


def _solve(n, pbc, rhs, pz=0):
    from ns_3d_staggered_dp_gb300 import Session, make_config

    bc = [1 if p == 1 else 2 for p in pbc]
    with Session(make_config(*n, lx=1.0, ly=1.0, lz=1.0, bc=bc, pbc=pbc, poisson_z=pz)) as s:
        return s.poisson(rhs)[1:-1, 1:-1, 1:-1]


def _oracle(n, pbc, rhs):
    return O.spectral_poisson(rhs, tuple(pbc), 1.0 / n[0], 1.0 / n[1], 1.0 / n[2])


CASES = [((m, 16, 16), (1, 1, 1), 0) for m in (16, 32, 64, 128, 256, 512)]
CASES += [((16, m, 32), (1, 1, 1), 0) for m in (16, 32, 64, 128, 256, 512)]
CASES += [((16, 16, m), (1, 1, 1), 1) for m in (32, 512)]
CASES += [((m, 18, 16), (b, b, b), 0) for m in (24, 32, 48, 64, 128, 256, 512) for b in (2, 3)]
CASES += [((16, m, 18), (b, b, b), 0) for m in (24, 32, 48, 64, 128, 256, 512) for b in (2, 3)]


@pytest.mark.parametrize("n,pbc,pz", CASES)
def test_line_lengths_and_spectra(n, pbc, pz):
    """White noise, and a field whose spectrum falls by 12 decades (blocks of
    very different magnitude meet in one line); the routine tolerance."""
    rng = np.random.default_rng(sum(n) + pbc[0])
    noise = rng.standard_normal(n)
    x = [(np.arange(m) + 0.5) / m for m in n]
    smooth = sum(10.0 ** (-2 * q) * np.cos(2 * np.pi * (q + 1) * x[0])[:, None, None]
                 * np.cos(2 * np.pi * (q % 3 + 1) * x[1])[None, :, None]
                 * np.cos(2 * np.pi * (q % 2 + 1) * x[2])[None, None, :] for q in range(7))
    for rhs in (noise - noise.mean(), smooth - smooth.mean()):
        assert rel_l2(_solve(n, pbc, rhs, pz), _oracle(n, pbc, rhs)) < 1e-12


@pytest.mark.parametrize("pbc", [(1, 1, 1), (3, 3, 3), (1, 3, 1)])
@pytest.mark.parametrize("scale", [1e-290, 1e-40, 1e40, 1e290])
def test_extreme_magnitudes(pbc, scale):
    """The solve is linear: a power-of-two scaling of the right-hand side scales the solution."""
    n = (32, 32, 32)
    rng = np.random.default_rng(9)
    rhs = rng.standard_normal(n)
    rhs -= rhs.mean()
    two = 2.0 ** np.round(np.log2(scale))
    assert rel_l2(_solve(n, pbc, rhs * two) / two, _oracle(n, pbc, rhs)) < 1e-12


def test_zero_right_hand_side():
    n = (32, 32, 32)
    for pbc in ((1, 1, 1), (3, 3, 3)):
        assert np.array_equal(_solve(n, pbc, np.zeros(n)), np.zeros(n))


@pytest.mark.parametrize("pbc", [(1, 1, 1), (3, 3, 3)])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_nonfinite_right_hand_side(pbc, bad):
    """One Inf or NaN reaches every value of the solution, as in the FP64 transforms."""
    n = (32, 32, 32)
    rhs = np.random.default_rng(3).standard_normal(n)
    rhs[7, 11, 5] = bad
    assert not np.isfinite(_solve(n, pbc, rhs)).any()
