"""The predictor's block exponents: what may set them, and the accuracy of cells far below them."""
import numpy as np
import pytest

from oracle import ns_oracle as O
from tests.helpers import random_state

pytestmark = pytest.mark.gpu
WALLS = dict(bc=(2, 2, 2), pbc=(3, 3, 3))


def _step(cfg, st):
    from ns_3d_staggered_dp_gb300 import Session, make_config

    with Session(make_config(cfg.nx, cfg.ny, cfg.nz, lx=cfg.lx, ly=cfg.ly, lz=cfg.lz, nu=cfg.nu, dt=cfg.dt,
                             scheme=cfg.scheme, bc=cfg.bc, pbc=cfg.pbc, dp_flag=cfg.dp_flag)) as s:
        s.set_state(st.u, st.v, st.w, st.p, (st.px, st.py, st.pz))
        s.step(1)
        return s.get_state()


def _plant(st, value):
    """value into the edges of the box along each component's own axis, which no stencil reads."""
    for c, a in enumerate((st.u, st.v, st.w)):
        b, d = [q for q in range(3) if q != c]
        for x in (0, -1):
            for y in (0, -1):
                at = [slice(None)] * 3
                at[b], at[d] = x, y
                a[tuple(at)] = value


@pytest.mark.parametrize("n,kw", [((32, 16, 32), {}), ((34, 17, 21), WALLS), ((32, 20, 16), dict(bc=(1, 2, 1), pbc=(1, 3, 1)))])
@pytest.mark.parametrize("scheme", [O.AB2, O.AB2_CN])
@pytest.mark.parametrize("value", [1e30, np.inf, np.nan])
def test_unread_edges_change_nothing(n, kw, scheme, value):
    """A fill value in the edges of the caller's arrays: the same bits as without it."""
    cfg = O.Config(*n, nu=0.01, dt=0.003, scheme=scheme, **kw)
    st = random_state(cfg, sum(n), amp=0.1, history=True)
    _plant(st, 0.0)
    ref = _step(cfg, st)
    _plant(st, value)
    got = _step(cfg, st)
    for k in ("hx", "hy", "hz"):
        assert np.array_equal(got[k], ref[k]), k
    for k in "uvwp":
        inner = np.s_[1:-1, 1:-1, 1:-1]
        assert np.array_equal(got[k][inner], ref[k][inner]), k


# --- cells far below the largest velocity ---------------------------------------------------------
def _uneven(cfg, seed, kind, q):
    """Random components, q times as large outside a jet, or falling off from a point by up to q."""
    st = random_state(cfg, seed, history=True)
    for f, h in (("u", "px"), ("v", "py"), ("w", "pz")):
        a = getattr(st, f)
        x = [np.arange(m) for m in a.shape]
        if kind == "jet":
            m = np.full(a.shape, q)
            m[:, cfg.ny // 2 + 2:3 * cfg.ny // 4, :] = 1.0
            m[cfg.nx // 2 + 5:cfg.nx // 2 + 8, :, :] = 1.0
        else:
            r = sum((np.abs(x[c] - n / 2) / (n / 2)).reshape([-1 if d == c else 1 for d in range(3)])
                    for c, n in enumerate((cfg.nx, cfg.ny, cfg.nz)))
            m = q ** np.minimum(r / 2.0, 1.0)
        a *= m
        getattr(st, h)[...] = 0.0
    O.vel_bc_staggered(st.u, st.v, st.w, O.Faces.zeros(cfg.nx, cfg.ny, cfg.nz), *cfg.bc)
    return st


def _local(a):
    """Largest magnitude of the 3 x 3 x 3 neighbours."""
    b = np.pad(np.abs(a), 1, mode="edge")
    m = np.zeros(a.shape)
    for i in range(3):
        for j in range(3):
            for k in range(3):
                m = np.maximum(m, b[i:i + a.shape[0], j:j + a.shape[1], k:k + a.shape[2]])
    return m


@pytest.mark.parametrize("n,kw", [((64, 32, 32), {}), ((40, 33, 35), WALLS), ((32, 64, 16), dict(bc=(1, 2, 1), pbc=(1, 3, 1)))])
@pytest.mark.parametrize("scheme", [O.AB2, O.AB2_CN])
@pytest.mark.parametrize("kind,q", [("jet", 1e-2), ("jet", 1e-6), ("decay", 1e-12)])
def test_quiet_cells_keep_their_digits(n, kw, scheme, kind, q):
    """The history of every cell, as far from the oracle's as rounding of its own neighbourhood makes
    it: of products of the component and the largest velocity beside it.  A cell in fixed point has
    both no further below its block's largest than 2^-11 together, and the six products and three
    increments are off by 2^-58 of those: 2^-47 of the local ones; the FP64 sides' part is smaller."""
    cfg = O.Config(*n, lx=1.0 * n[0], ly=1.0 * n[1], lz=1.0 * n[2], nu=0.05, dt=0.01, scheme=scheme, **kw)
    st = _uneven(cfg, sum(n), kind, q)
    got, ref = _step(cfg, st), O.step(st.copy(), cfg)
    # slot arrays of the local magnitudes: the component's own axis has no slot 0 in its own array
    loc = [np.pad(_local(a), [(1, 0) if d == c else (0, 0) for d in range(3)], mode="edge")
           for c, a in enumerate((st.u, st.v, st.w))]
    big = np.maximum(np.maximum(loc[0], loc[1]), loc[2])
    for c, (k, r) in enumerate((("hx", "px"), ("hy", "py"), ("hz", "pz"))):
        err = np.abs(got[k] - getattr(ref, r))
        size = loc[c] * (3.0 * _local(big) + (12.0 * cfg.nu if scheme == O.AB2 else 0.0))
        size = size[(slice(None),) * c + (slice(1, None),)]
        assert (err <= 2.0 ** -47 * size).all(), (k, float((err / np.maximum(size, 1e-300)).max()))


# --- axes of very different spacing ---------------------------------------------------------------
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("aspect", [1.5, 3.0, 16.0, 100.0, 1000.0])
@pytest.mark.parametrize("scheme", [O.AB2, O.AB2_CN])
def test_terms_along_a_coarse_axis(axis, aspect, scheme):
    """Velocities that vary along the coarsest axis alone: the other axes' differences are exactly
    zero, so the history is the coarse terms.  Values of 1/2 to 1: at most 2^-4 of the block's largest
    square, three terms off by 2^-58 of that and the oracle's by a few 2^-53: 2^-49 in all."""
    n = [16, 16, 16]
    n[axis] = 32
    L = [1.0] * 3
    L[axis] = 2.0 * aspect
    h = L[axis] / n[axis]
    cfg = O.Config(*n, *L, nu=h, dt=1e-4, scheme=scheme)  # convection and viscous term of the same size
    st = O.State.zeros(*n)
    rng = np.random.default_rng(axis)
    for c, f in enumerate((st.u, st.v, st.w)):
        line = rng.uniform(0.5, 1.0, n[axis])
        at = np.arange(f.shape[axis]) - (0 if c == axis else 1)
        f[...] = line[at % n[axis]].reshape([-1 if d == axis else 1 for d in range(3)])
    got, ref = _step(cfg, st), O.step(st.copy(), cfg)
    size = 3.0 / h + (12.0 * cfg.nu / h ** 2 if scheme == O.AB2 else 0.0)
    for k, r in (("hx", "px"), ("hy", "py"), ("hz", "pz")):
        err = np.abs(got[k] - getattr(ref, r))
        assert err.max() <= 2.0 ** -49 * size, (k, float(err.max() / size))
