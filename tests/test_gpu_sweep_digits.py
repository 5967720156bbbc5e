"""The chunked sweeps cell by cell: small values next to large ones keep their digits."""
import numpy as np
import pytest

from oracle import ns_oracle as O

WALL = {1: 1, 2: 3}
LD = np.longdouble


def _cn_solve(x, axis, alpha, normal, bc, closure):
    """One sweep in long double over the unknowns along axis: cyclic lines (closure 0: row 1 of the normal
    component ties face 1 to itself), or walls of value zero (identity rows for the normal component, the
    mean of the two cells for the others)."""
    x = np.moveaxis(x, axis, 0).copy()
    m = x.shape[0]
    b, lo, up = np.full(m, 1 + 2 * LD(alpha)), np.full(m, -LD(alpha)), np.full(m, -LD(alpha))  # lo[0], up[m-1]: corners
    if bc == 1 and normal and closure == 0:
        b[0], lo[0] = b[0] + lo[0], 0
    if bc != 1:
        x[0] = x[-1] = 0
        b[0] = b[-1] = 1 if normal else LD(0.5)
        up[0] = lo[-1] = 0 if normal else LD(0.5)
        lo[0] = up[-1] = 0
    # elimination of a tridiagonal matrix with its two corners: col holds column m-1, row row m-1
    col, row = np.zeros(m, LD), np.zeros(m, LD)
    col[0], col[m - 2], col[m - 1] = lo[0], up[m - 2], b[m - 1]
    row[0], row[m - 2] = up[m - 1], lo[m - 1]
    for i in range(m - 1):
        if i < m - 2:
            f = lo[i + 1] / b[i]
            b[i + 1] -= f * up[i]
            col[i + 1] -= f * col[i]
            x[i + 1] -= f * x[i]
        f = row[i] / b[i]
        if i < m - 2:
            row[i + 1] -= f * up[i]
        col[m - 1] -= f * col[i]
        x[m - 1] -= f * x[i]
    x[m - 1] /= col[m - 1]
    for i in range(m - 2, -1, -1):
        x[i] = (x[i] - col[i] * x[m - 1] - (up[i] * x[i + 1] if i < m - 2 else 0)) / b[i]
    return np.moveaxis(x, 0, axis)


def _reference(f, c, alpha, bc, closure):
    """u*, v* or w* of a first step without convection, on the unknowns of component c (periodic axes: once)."""
    own = tuple(slice(0, -1) if q == c else slice(1, -1) for q in range(3))
    f = f.astype(LD)[tuple(own[q] if bc[q] == 1 else slice(None) for q in range(3))]
    r = f.copy()
    for q in range(3):
        up, dn = np.roll(f, -1, q), np.roll(f, 1, q)  # past a wall's end: rows that the sweeps replace
        r += LD(alpha) * (up + dn - 2 * f)
    for q in range(3):
        r = _cn_solve(r, q, alpha, q == c, bc[q], closure)
    return r[tuple(slice(None) if bc[q] == 1 or q == c else slice(1, -1) for q in range(3))]


@pytest.mark.parametrize("bc,closure", [(1, 0), (1, 1), (2, 0)])
@pytest.mark.parametrize("normal", [True, False])
def test_reference_solve(bc, closure, normal):
    """The long double elimination against a dense solve of the oracle's matrices."""
    n, alpha = 9, 0.07
    A = O.mat_cn(n, bc, 1.0, 2.0 * alpha, 1.0)[0 if normal else 1]
    m = n if bc == 1 else A.shape[0]
    x = np.random.default_rng(n).standard_normal((m, 4))
    if bc == 1:  # the unknowns once: the duplicates' columns folded in
        i0 = 0 if normal else 1
        B = np.zeros((n, n))
        for j in range(A.shape[0]):
            B[:, (j - i0) % n] += A[i0:i0 + n, j]
        if normal and closure:
            B[0, 0], B[0, n - 1] = B[0, 0] + alpha, -alpha
        A = B
    else:
        x[0] = x[-1] = 0.0
    got = _cn_solve(x.astype(LD), 0, alpha, normal, bc, closure)
    assert np.abs(A @ got.astype(float) - x).max() < 1e-14


@pytest.mark.gpu
@pytest.mark.parametrize("n,bc", [((64, 32, 128), (1, 1, 1)), ((512, 16, 16), (1, 1, 1)), ((64, 67, 16), (1, 2, 1)),
                                  ((38, 128, 61), (2, 2, 2)), ((300, 16, 18), (2, 2, 2))])
@pytest.mark.parametrize("alpha", [0.002, 0.012, 0.03, 0.07])
@pytest.mark.parametrize("quiet", [1e-6, 1e-14])
@pytest.mark.parametrize("closure", [0, 1])
def test_quiet_cells_keep_their_digits(n, bc, alpha, quiet, closure):
    """Velocities of 1e-30 (no convection to speak of) in a cell out of 500, quiet times that elsewhere, all
    positive, so that no sum of a sweep cancels: 4e-15 of the predictor's cells and 30 roundings a sweep."""
    from ns_3d_staggered_dp_gb300 import Session, make_config

    if closure and 1 not in bc:
        pytest.skip("no periodic axis")
    dt, h = 0.003, 0.125
    L = [h * m for m in n]
    nu = 2.0 * alpha * h ** 2 / dt
    rng = np.random.default_rng(sum(n))
    st = O.State.zeros(*n)
    for f in "uvw":
        a = getattr(st, f)
        setattr(st, f, 1e-30 * np.where(rng.random(a.shape) < 0.002, 1.0, quiet) * rng.uniform(0.5, 1.0, a.shape))
    O.vel_bc_staggered(st.u, st.v, st.w, O.Faces.zeros(*n), *bc)
    with Session(make_config(*n, lx=L[0], ly=L[1], lz=L[2], nu=nu, dt=dt, scheme=2, bc=bc, pbc=tuple(WALL[b] for b in bc),
                             cn_periodic_closure=closure)) as s:
        s.set_state(st.u, st.v, st.w, st.p)
        s.step(1)
        got = s.get_stage()
    a = 0.5 * dt * nu / h ** 2
    for c, k in enumerate("uvw"):
        ref = _reference(getattr(st, k), c, a, bc, closure)
        g = got[k + "s"][tuple((slice(0, -1) if bc[q] == 1 else slice(None)) if q == c else slice(1, -1) for q in range(3))]
        assert np.all(np.abs(g - ref) <= (4e-15 + 90 * 2.0 ** -53) * np.abs(ref)), k
