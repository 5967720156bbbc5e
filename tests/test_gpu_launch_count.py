"""ns_launch_count against the kernels that the device ran."""
import numpy as np
import pytest

from oracle import ns_oracle as O
from tests.helpers import random_state

pytestmark = pytest.mark.gpu


def _kernels(f):
    """Kernels of this library that f launches."""
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA]) as p:
        f()
    return sum(1 for e in p.events() if "ns::" in e.name)


@pytest.mark.parametrize("scheme", [O.AB2, O.AB2_CN])
def test_backward_step(scheme):
    """One step more of the backward pass and of its recomputed forward steps: the counter grows by
    what the device runs more (gathers of the results are the same for both)."""
    import torch

    from ns_3d_staggered_dp_gb300 import Session, make_config

    torch.zeros(1, device="cuda")
    cfg = O.Config(16, 16, 16, nu=0.01, dt=0.003, scheme=scheme)
    st = random_state(cfg, 1)
    seeds = [np.ones_like(a) for a in (st.u, st.v, st.w)]
    ran, counted = [], []
    for steps in (2, 3, 4):
        with Session(make_config(16, 16, 16, nu=0.01, dt=0.003, scheme=scheme)) as s:
            s.set_state(st.u, st.v, st.w, st.p)
            s.adj_forward(steps, 1)
            s.adj_backward(*seeds)  # what the first call sets up
            s.set_state(st.u, st.v, st.w, st.p)
            s.adj_forward(steps, 1)
            before = s.launch_count()
            ran.append(_kernels(lambda: s.adj_backward(*seeds)))
            counted.append(s.launch_count() - before)
    assert ran[2] - ran[1] == counted[2] - counted[1] > 0
