"""Accuracy of the pressure solves beyond the routine tolerance: eigenvalues next to the Nyquist
mirror, and the allocation-free solve on flat boxes."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lam(n, L):
    """Eigenvalues of the discrete Laplacian, every mode by its smaller wavenumber."""
    out = 0.0
    for q, (m, l) in enumerate(zip(n, L)):
        k = np.minimum(np.arange(m), m - np.arange(m))
        out = out - (4.0 * np.sin(np.pi * k / m) ** 2 / (l / m) ** 2).reshape([-1 if d == q else 1 for d in range(3)])
    return out


@pytest.mark.parametrize("n", [(32, 32, 32), (64, 32, 16), (16, 128, 32)])
@pytest.mark.parametrize("mode", [(1, 1, 0), (0, 1, 0), (1, 0, 1)])
def test_lowest_modes(n, mode):
    """A right-hand side of one low mode is an eigenvector: the solution is it over the eigenvalue, to
    a few roundings of the transforms and line solves (4 units of 2^-52 in norm).  Both halves of the
    spectrum carry it, so an eigenvalue of wavenumber n - 1 that is off shows."""
    from ns_3d_staggered_dp_gb300 import Session, make_config

    x = [(np.arange(m) + 0.25) / m for m in n]
    rhs = np.ones(n)
    for q in range(3):
        if mode[q]:
            rhs = rhs * np.cos(2.0 * np.pi * x[q]).reshape([-1 if d == q else 1 for d in range(3)])
    want = rhs / _lam(n, (1.0, 1.0, 1.0))[mode]
    with Session(make_config(*n, lx=1.0, ly=1.0, lz=1.0)) as s:
        got = s.poisson(rhs)[1:-1, 1:-1, 1:-1]
    assert np.linalg.norm(got - want) <= 4.0 * 2.0 ** -52 * np.linalg.norm(want)


@pytest.mark.parametrize("n,lz", [((32, 32, 32), 1.0), ((32, 32, 32), 0.05), ((64, 32, 16), 0.01), ((16, 64, 64), 1e-3),
                                  ((32, 16, 64), 20.0)])
def test_allocation_free_solve_of_flat_boxes(n, lz):
    """The low modes of a flat box have rho next to 1 in the cyclic z solve, whose two recursions then
    add up their roundings: 4 units of 2^-52 in norm beside 4 of the transforms (and of this reference)."""
    import torch

    from ns_3d_staggered_dp_gb300 import _lib

    rhs = np.random.default_rng(n[0] + n[2]).standard_normal(n)
    rhs -= rhs.mean()
    lam = _lam(n, (1.0, 1.0, lz))
    lam[0, 0, 0] = np.inf
    want = np.fft.ifftn(np.fft.fftn(rhs) / lam).real
    r = torch.from_numpy(np.ascontiguousarray(rhs.transpose(2, 1, 0))).cuda()
    dp = torch.zeros(tuple(m + 2 for m in n[::-1]), device="cuda", dtype=torch.float64)
    st = torch.cuda.current_stream().cuda_stream
    rc = _lib.load().ns_poisson_fft_noalloc(ctypes.c_void_p(r.data_ptr()), ctypes.c_void_p(dp.data_ptr()), *n, 1.0, 1.0,
                                            lz, ctypes.c_void_p(st))
    assert rc == 0
    got = dp.cpu().numpy().transpose(2, 1, 0)[1:-1, 1:-1, 1:-1]
    assert np.linalg.norm(got - want) <= 8.0 * 2.0 ** -52 * np.linalg.norm(want)
