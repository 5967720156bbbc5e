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
