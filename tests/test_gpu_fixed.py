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


# --- the predictor's fixed-point stencils -------------------------------------------------------
def _layered(cfg, seed, mags=(1.0, 1.0, 1.0), zamp=0.0):
    """Random state with one magnitude per component, changing along z by 10^zamp over the box (the
    16-plane groups then have different exponents)."""
    from tests.helpers import random_state

    st = random_state(cfg, seed, history=True)
    for f, h, m in (("u", "px", mags[0]), ("v", "py", mags[1]), ("w", "pz", mags[2])):
        for name in (f, h):
            a = getattr(st, name)
            a *= m * 10.0 ** (zamp * np.cos(np.pi * np.arange(a.shape[2]) / cfg.nz))
    O.vel_bc_staggered(st.u, st.v, st.w, O.Faces.zeros(cfg.nx, cfg.ny, cfg.nz), *cfg.bc)
    return st


def _gpu_step(cfg, st, stage=False):
    from ns_3d_staggered_dp_gb300 import Session, make_config

    with Session(make_config(cfg.nx, cfg.ny, cfg.nz, lx=cfg.lx, ly=cfg.ly, lz=cfg.lz, nu=cfg.nu, dt=cfg.dt,
                             scheme=cfg.scheme, bc=cfg.bc, pbc=cfg.pbc, dp_flag=cfg.dp_flag)) as s:
        s.set_state(st.u, st.v, st.w, st.p, (st.px, st.py, st.pz))
        s.step(1)
        return s.get_state()


WALLS = dict(bc=(2, 2, 2), pbc=(3, 3, 3))
STENCILS = [((16, 16, 16), {}), ((32, 16, 64), dict(lz=3.0)), ((64, 32, 32), {})]
STENCILS += [((34, ny, nz), WALLS) for ny, nz in ((7, 15), (8, 16), (9, 17), (17, 33))]


@pytest.mark.parametrize("n,kw", STENCILS)
@pytest.mark.parametrize("scheme,dpf", [(O.EULER, 0), (O.AB2, 1), (O.AB2_CN, 0)])
@pytest.mark.parametrize("mags,zamp", [((1, 1, 1), 0.0), ((1, 1e-3, 1e-6), 0.0), ((1e-5, 1, 0), 2.0)])
def test_predictor_shapes_and_magnitudes(n, kw, scheme, dpf, mags, zamp):
    """Tile and group edges, unequal axes, components of very different size; the step's tolerance."""
    cfg = O.Config(*n, nu=0.01, dt=0.003, scheme=scheme, dp_flag=dpf, **kw)
    st = _layered(cfg, sum(n), mags, zamp)
    got, ref = _gpu_step(cfg, st), O.step(st.copy(), cfg)
    for k, a in (("u", "u"), ("v", "v"), ("w", "w"), ("p", "p"), ("hx", "px"), ("hy", "py"), ("hz", "pz")):
        assert rel_l2(got[k], getattr(ref, a)) < 1e-10, k


@pytest.mark.parametrize("amp", [1e-150, 1e-60, 1e60, 1e100])
def test_predictor_extreme_velocities(amp):
    """Velocities outside the fixed-point range take the FP64 stencils (large) or vanish against none
    (small); dt scaled so that the convection stays an increment."""
    cfg = O.Config(32, 16, 32, nu=0.01 * amp, dt=0.003 / amp, scheme=O.AB2)
    st = _layered(cfg, 5, (amp, amp, amp))
    for h in (st.px, st.py, st.pz):
        h *= amp  # a history of the size of u^2
    got, ref = _gpu_step(cfg, st), O.step(st.copy(), cfg)
    for k, a in (("u", "u"), ("v", "v"), ("w", "w")):
        assert rel_l2(got[k] / amp, getattr(ref, a) / amp) < 1e-10, k


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_predictor_nonfinite_velocity(bad):
    """A non-finite velocity spoils exactly the history entries that the reference's stencils spoil."""
    cfg = O.Config(32, 16, 64, nu=0.01, dt=0.003, scheme=O.AB2)
    st = _layered(cfg, 6)
    st.v[9, 7, 30] = bad
    with np.errstate(invalid="ignore", over="ignore"):
        got, ref = _gpu_step(cfg, st), O.step(st.copy(), cfg)
    for k, a in (("hx", "px"), ("hy", "py"), ("hz", "pz")):
        r = getattr(ref, a)
        fin = np.isfinite(r)
        assert np.array_equal(np.isfinite(got[k]), fin) and not fin.all(), k
        assert rel_l2(got[k][fin], r[fin]) < 1e-12, k


@pytest.mark.parametrize("n,kw", [((32, 16, 64), {}), ((34, 18, 49), WALLS)])
@pytest.mark.parametrize("scheme", [O.AB2, O.AB2_CN])
def test_slabs_of_different_exponents(n, kw, scheme):
    """ns_step_host predicts in z-slabs: the same bits as the whole-box step, with exponents that
    change from group to group."""
    from ns_3d_staggered_dp_gb300 import Session, make_config

    cfg = O.Config(*n, nu=0.01, dt=0.003, scheme=scheme, **kw)
    st = _layered(cfg, 11, (1, 1e-2, 1), 3.0)
    hist = (st.px, st.py, st.pz)
    with Session(make_config(*n, nu=0.01, dt=0.003, scheme=scheme, **kw)) as s:
        s.set_state(st.u, st.v, st.w, st.p, hist)
        s.step(1)
        dev = s.get_state()
        host = s.step_host(st.u, st.v, st.w, st.p, hist)
    for k in dev:
        assert np.array_equal(dev[k], host[k]), k


# --- the chunked ADI sweeps ---------------------------------------------------------------------
SWEEPS = [((16, 16, 16), (1, 1, 1)), ((64, 32, 128), (1, 1, 1)), ((32, 67, 16), (1, 2, 1)), ((64, 32, 34), (1, 1, 2)),
          ((38, 21, 35), (2, 2, 2)), ((66, 64, 17), (4, 2, 4))]


@pytest.mark.parametrize("n,bc", SWEEPS)
@pytest.mark.parametrize("alpha", [0.0, 1e-4, 0.004, 0.012, 0.03, 0.07, 0.3])
@pytest.mark.parametrize("closure", [0, 1])
def test_sweeps_for_every_halo(n, bc, alpha, closure):
    """u*, v*, w* after the sweeps, with viscous numbers on both sides of every halo's limit (and
    beyond the last, where the whole-line kernels run): a few roundings of values of order one."""
    from ns_3d_staggered_dp_gb300 import Session, make_config
    from tests.helpers import random_state

    if closure and 1 not in bc:
        pytest.skip("no periodic axis")
    wall = {1: 1, 2: 3, 4: 4}
    dt, L = 0.003, [2.0 * np.pi] * 3
    # the same viscous number on every axis: lengths in proportion to the cells
    L = [2.0 * np.pi * m / n[0] for m in n]
    nu = 2.0 * alpha * (L[0] / n[0]) ** 2 / dt
    cfg = O.Config(*n, *L, nu=nu, dt=dt, scheme=O.AB2_CN, bc=bc, pbc=tuple(wall[b] for b in bc))
    st = random_state(cfg, 3, amp=0.1, history=True)
    cnf = None
    if closure:  # the cyclic closure of the periodic normal component
        cnf = O.CNFactors(*n, cfg.bc, *(h * h for h in cfg.h), dt, nu)
        for ax, b in enumerate(bc):
            if b == 1:
                A = O.mat_cn(n[ax], 1, cfg.h[ax] ** 2, dt, nu)[0]
                A[0, n[ax] - 1], A[0, n[ax]] = A[0, n[ax]], 0.0
                cnf.lu[ax] = (O._lu(A), cnf.lu[ax][1])
    ref, parts = O.step(st.copy(), cfg, cnf=cnf, return_parts=True)
    with Session(make_config(*n, lx=L[0], ly=L[1], lz=L[2], nu=nu, dt=dt, scheme=2, bc=cfg.bc, pbc=cfg.pbc,
                             cn_periodic_closure=closure)) as s:
        s.set_state(st.u, st.v, st.w, st.p, (st.px, st.py, st.pz))
        s.step(1)
        g = s.get_stage()
        out = s.get_state()
    inner = {"us": (slice(None), slice(1, -1), slice(1, -1)), "vs": (slice(1, -1), slice(None), slice(1, -1)),
             "ws": (slice(1, -1), slice(1, -1), slice(None))}
    for k, sl in inner.items():
        assert rel_l2(g[k][sl], parts[k][sl]) < 1e-13, k
    for k in "uvw":
        assert rel_l2(out[k], getattr(ref, k)) < 1e-10, k


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("m", [14, 16, 30, 32, 34, 46, 64, 66, 126, 128, 130, 134, 254, 256, 270, 272, 300])
@pytest.mark.parametrize("bc", [1, 2, 4])
def test_sweeps_of_every_line_length(axis, m, bc):
    """Line lengths around every chunk count and past the longest line of one CTA."""
    from ns_3d_staggered_dp_gb300 import Session, make_config
    from tests.helpers import random_state

    if bc == 1 and m & (m - 1):
        pytest.skip("periodic lines are powers of two")
    if axis == 2 and m > 256:
        pytest.skip("the Poisson solve's line axis, 256 cells at most with a wall x")
    if bc == 1:
        m = max(m, 16) if m < 256 else 512
    n, code = [16, 8, 9] if bc != 1 else [16, 16, 16], [2, 2, 2] if bc != 1 else [1, 1, 1]
    n[axis], code[axis] = m, bc
    wall = {1: 1, 2: 3, 4: 4}
    dt, L = 0.003, [0.2 * q for q in n]
    for alpha in (0.004, 0.07):
        nu = 2.0 * alpha * 0.2 ** 2 / dt
        cfg = O.Config(*n, *L, nu=nu, dt=dt, scheme=O.AB2_CN, bc=tuple(code), pbc=tuple(wall[b] for b in code))
        st = random_state(cfg, m, amp=0.1, history=True)
        _, parts = O.step(st.copy(), cfg, return_parts=True)
        with Session(make_config(*n, lx=L[0], ly=L[1], lz=L[2], nu=nu, dt=dt, scheme=2, bc=cfg.bc, pbc=cfg.pbc)) as s:
            s.set_state(st.u, st.v, st.w, st.p, (st.px, st.py, st.pz))
            s.step(1)
            g = s.get_stage()
        for k, sl in (("us", np.s_[:, 1:-1, 1:-1]), ("vs", np.s_[1:-1, :, 1:-1]), ("ws", np.s_[1:-1, 1:-1, :])):
            assert rel_l2(g[k][sl], parts[k][sl]) < 1e-13, k


# --- the dense wall transforms ------------------------------------------------------------------
DENSE = [((16, m, 9), b) for m in (5, 8, 15, 16, 17, 31, 75, 100, 127, 129, 200, 257, 300) for b in (2, 3, 4)]
DENSE += [((m, 8, 9), b) for m in (6, 16, 18, 34, 90, 130, 256, 320) for b in (2, 3, 4)]


@pytest.mark.parametrize("n,pbc", DENSE)
def test_dense_lengths(n, pbc):
    """Odd and even lengths on both sides of the partial sums' length, every pressure code; the routine
    tolerance, and an extreme magnitude."""
    rng = np.random.default_rng(sum(n) + pbc)
    rhs = rng.standard_normal(n)
    rhs -= rhs.mean()
    ref = _oracle(n, (pbc,) * 3, rhs)
    assert rel_l2(_solve(n, (pbc,) * 3, rhs), ref) < 1e-12
    two = 2.0 ** 960
    assert rel_l2(_solve(n, (pbc,) * 3, rhs * two) / two, ref) < 1e-12


# --- the cyclic z solve and the one-launch fills ------------------------------------------------
@pytest.mark.parametrize("nz", [16, 32, 64, 128, 256, 512])
@pytest.mark.parametrize("lz", [0.05, 1.0, 40.0])
def test_cyclic_solve_lengths(nz, lz):
    """Every segment count; flat boxes (rho next to 1 in the low modes) and tall ones."""
    from ns_3d_staggered_dp_gb300 import Session, make_config

    n = (32, 16, nz)
    rhs = np.random.default_rng(nz).standard_normal(n)
    rhs -= rhs.mean()
    ref = O.spectral_poisson(rhs, (1, 1, 1), 1.0 / 32, 1.0 / 16, lz / nz)
    with Session(make_config(*n, lx=1.0, ly=1.0, lz=lz)) as s:
        assert rel_l2(s.poisson(rhs)[1:-1, 1:-1, 1:-1], ref) < 1e-11


@pytest.mark.parametrize("bc", [(1, 1, 1), (1, 2, 1), (1, 1, 4), (1, 4, 2), (2, 2, 2), (4, 2, 4), (4, 4, 4)])
def test_fills_of_every_code(bc):
    """vel_bc_staggered and the pressure ghosts with non-zero faces, edges and corners included."""
    from ns_3d_staggered_dp_gb300 import Session, make_config

    n = (32, 16, 16)
    rng = np.random.default_rng(sum(bc))
    for pw in (2, 3, 4):
        pbc = tuple(1 if b == 1 else pw for b in bc)
        cfg = O.Config(*n, 3.0, 1.0, 2.0, bc=bc, pbc=pbc)
        f = O.Faces.zeros(*n)
        for k in f.d:
            f.d[k] = rng.standard_normal(f.d[k].shape)
        sh = O.State.zeros(*n)
        us, vs, ws = (rng.standard_normal(a.shape) for a in (sh.u, sh.v, sh.w))
        ref = [us.copy(), vs.copy(), ws.copy()]
        O.vel_bc_staggered(*ref, f, *bc)
        rhs = rng.standard_normal(n)
        with Session(make_config(*n, lx=3.0, ly=1.0, lz=2.0, bc=bc, pbc=pbc)) as s:
            s.set_faces(f.d)
            got = s.vel_bc(us, vs, ws)
            dp = s.poisson(rhs)
        for a, b in zip(got, ref):
            assert np.array_equal(a, b)
        want = np.zeros(dp.shape)
        want[1:-1, 1:-1, 1:-1] = dp[1:-1, 1:-1, 1:-1]
        O.pr_bc_staggered(want, f, pbc, *cfg.h)
        np.testing.assert_allclose(dp, want, rtol=0, atol=4e-16 * max(1.0, np.abs(want).max()))


# --- states into page-locked arrays -----------------------------------------------------------------
@pytest.mark.parametrize("shift", [0, 1, 5])
@pytest.mark.parametrize("n,bc", [((16, 16, 16), (1, 1, 1)), ((18, 9, 13), (2, 2, 2)), ((64, 21, 32), (1, 2, 1))])
def test_state_into_page_locked_arrays(n, bc, shift):
    """The kernel that writes page-locked arrays against the staged copies, some fields left out."""
    import ctypes

    import torch

    from ns_3d_staggered_dp_gb300 import Session, make_config
    from tests.helpers import random_state

    cfg = O.Config(*n, 1.0, 1.0, 1.0, scheme=O.AB2, dt=1e-3, bc=bc, pbc=tuple(3 if b == 2 else 1 for b in bc))
    st = random_state(cfg, 7, history=True)
    with Session(make_config(*n, dt=1e-3, scheme=1, bc=bc, pbc=cfg.pbc)) as s:
        s.set_state(st.u, st.v, st.w, st.p, (st.px, st.py, st.pz))
        s.step(2)
        ref = s.get_state()
        keys = ("u", "v", "w", "p", "hx", "hy", "hz")
        for skip in ((), ("v", "hz"), ("u", "p", "hx", "hy")):
            buf, arg = {}, []
            for k in keys:
                buf[k] = torch.full((ref[k].size + shift + 3,), 7.0, dtype=torch.float64).pin_memory()
                p = ctypes.cast(buf[k].data_ptr() + 8 * shift, ctypes.POINTER(ctypes.c_double))
                arg.append(None if k in skip else p)
            s._check(s.lib.ns_get_state(s.h, *arg))
            for k in keys:
                got = buf[k].numpy()
                body = got[shift:shift + ref[k].size]
                assert (got[:shift] == 7.0).all() and (got[shift + ref[k].size:] == 7.0).all()
                assert (body == 7.0).all() if k in skip else np.array_equal(body, ref[k].ravel(order="F"))
