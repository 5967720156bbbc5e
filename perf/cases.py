"""Performance cases of the FP64 staggered Navier-Stokes step: the work a user has the library do,
through its public entry points (the Session, Batch and adjoint tiers of api.py and the C ABI with
pinned host buffers), from the smallest box to the 256^3 headline one.

Kinds of case
  session  a device-resident run: `steps` time steps, then the whole state read back (a driver that
           records a snapshot every few steps)
  host     one time step of a driver that keeps its state on the host (ns_step_host, pinned memory)
  poisson  the allocation-free periodic pressure solve on the caller's device buffers
  batch    the re-simulation of many sub-blocks of a parent run over `intervals` parent steps
  adjoint  a checkpointed forward run and the gradient of a function of its final velocity
Walls: "" triply periodic, "y" a channel, "xyz" a closed box (no slip, Neumann pressure).
"""
import ctypes
import math

import numpy as np
import torch

from ns_3d_staggered_dp_gb300 import _lib, api

PI = 3.1415926535897932
EULER, AB2, AB2_CN = 0, 1, 2
DEV = "cuda"


def listed():
    S = lambda name, n, walls, scheme, dpf, steps: {  # noqa: E731
        "name": name, "kind": "session", "nx": n[0], "ny": n[1], "nz": n[2], "walls": walls, "scheme": scheme,
        "dp_flag": dpf, "steps": steps}
    return [
        # one step of the smallest driver set-up (the 32^3 Taylor-Green size): launches and latency count
        S("periodic 32 one step", (32, 32, 32), "", AB2_CN, 0, 1),
        # a small production box with the explicit scheme and the incremental pressure
        S("periodic 64 ab2", (64, 64, 64), "", AB2, 1, 10),
        # the adjoint / parent-run size
        S("periodic 128 ab2cn", (128, 128, 128), "", AB2_CN, 0, 10),
        # the headline: 256^3 decaying turbulence
        S("periodic 256 ab2cn", (256, 256, 256), "", AB2_CN, 0, 16),
        # the wall-bounded channel configuration
        S("channel 256x128x256", (256, 128, 256), "y", AB2_CN, 0, 10),
        # a closed box of transform-friendly edges
        S("box 128", (128, 128, 128), "xyz", AB2_CN, 0, 10),
        # a closed box of ragged edges, incremental pressure
        S("box 90x75x61 ragged", (90, 75, 61), "xyz", AB2, 1, 10),
        # a host-resident driver: the state crosses the link both ways on every step
        {"name": "host 256 ab2cn", "kind": "host", "nx": 256, "ny": 256, "nz": 256, "walls": "", "scheme": AB2_CN,
         "dp_flag": 0},
        # a solver embedded in a host application that owns the device memory
        {"name": "poisson 64", "kind": "poisson", "nx": 64, "ny": 64, "nz": 64},
        # the re-simulation study: 64 sub-blocks, sub-step ratios 1, 2, 4 (explicit) and per-sweep faces (AB2-CN)
        {"name": "batch 64 ab2", "kind": "batch", "parent": 128, "count": 64, "subs_seed": 4096, "edge_max": 64,
         "scheme": AB2, "intervals": 8},
        {"name": "batch 64 ab2cn", "kind": "batch", "parent": 128, "count": 64, "subs_seed": 4096, "edge_max": 64,
         "scheme": AB2_CN, "intervals": 8},
        # a gradient for data assimilation
        {"name": "adjoint 128", "kind": "adjoint", "n": 128, "steps": 10, "ckpt_every": 5},
    ]


def draw(rng):
    kind = rng.choice(["session"] * 6 + ["host", "poisson", "batch", "adjoint"])
    pick = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    pow2 = lambda lo, hi: 1 << rng.randint(lo, hi)  # noqa: E731
    if kind in ("session", "host"):
        walls = rng.choice(["", "", "y", "xyz"])
        nx, ny, nz = pow2(4, 8), pow2(4, 8), pow2(4, 8)
        if walls:
            ny = pick(16, 200)
        if walls == "xyz":
            nx, nz = 2 * pick(8, 100), pick(16, 200)
        case = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "walls": walls, "scheme": rng.choice([EULER, AB2, AB2_CN]),
                "dp_flag": rng.choice([0, 1])}
        if kind == "session":
            case["steps"] = rng.randint(1, 12)
        return case
    if kind == "poisson":
        return {"kind": kind, "nx": pow2(4, 6), "ny": pow2(4, 6), "nz": pow2(4, 6)}
    if kind == "batch":
        return {"kind": kind, "parent": rng.choice([64, 128]), "count": pick(2, 64), "subs_seed": rng.randint(1, 9999),
                "edge_max": rng.choice([24, 32, 48]), "scheme": rng.choice([AB2, AB2_CN]),
                "intervals": rng.randint(2, 8)}
    return {"kind": kind, "n": pow2(4, 7), "steps": rng.randint(2, 10), "ckpt_every": rng.randint(1, 5)}


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _ext(case):
    return tuple(2.0 * PI if ax not in case["walls"] else 2.0 for ax in "xyz")


def _nu(n):
    return max(1.0 / 1600.0, 0.32 / n)  # resolved at the box's size


def _periodic_field(n, lengths, seed, k0=3.0):
    """A random solenoidal field of spectrum k^4 exp(-2 (k/k0)^2), unit rms, sampled at the staggered
    points of an (nx, ny, nz) box: slot arrays (n+2 per axis, slot m = cell m or its low face)."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    k = [torch.fft.fftfreq(m, 1.0 / m, device=DEV, dtype=torch.float64) for m in n]
    K = torch.meshgrid(*k, indexing="ij")
    K2 = K[0] ** 2 + K[1] ** 2 + K[2] ** 2
    amp = torch.sqrt(K2) * torch.exp(-K2 / k0 ** 2)
    a = [torch.randn(n, generator=g, device=DEV, dtype=torch.complex128) * amp for _ in range(3)]
    K2[0, 0, 0] = 1.0
    dot = (K[0] * a[0] + K[1] * a[1] + K[2] * a[2]) / K2
    out = []
    for c in range(3):
        ph = sum(K[q] * (0.0 if q == c else 0.5) * (2.0 * PI / n[q]) for q in range(3))
        out.append(torch.fft.ifftn((a[c] - K[c] * dot) * torch.exp(1j * ph)).real)
    rms = torch.sqrt(sum((f ** 2).mean() for f in out) / 3.0)
    return [torch.nn.functional.pad((f / rms)[None, None], (1, 1, 1, 1, 1, 1), mode="circular")[0, 0] for f in out]


def _wall_field(n, lengths, walls, seed):
    """A smooth shear profile between the walls plus seeded modes, all zero on the walls (slot arrays)."""
    r = np.random.default_rng(seed)
    out = []
    for c in range(3):
        x = [torch.arange(n[q] + 2, device=DEV, dtype=torch.float64).add(-1.0 if q == c else -0.5)
             * (lengths[q] / n[q]) for q in range(3)]
        f = torch.zeros(tuple(m + 2 for m in n), device=DEV, dtype=torch.float64)
        for _ in range(6):
            t = [torch.sin(int(r.integers(1, 4)) * (PI / 2.0) * x[q]) if ax in walls else
                 torch.sin(int(r.integers(1, 5)) * x[q] + r.uniform(0, 2 * PI)) for q, ax in enumerate("xyz")]
            f += float(r.standard_normal()) * 0.3 * t[0][:, None, None] * t[1][None, :, None] * t[2][None, None, :]
        if c == 0:
            prof = torch.ones((1, 1, 1), device=DEV, dtype=torch.float64)
            for q, ax in enumerate("xyz"):
                if ax in walls:
                    prof = prof * (x[q] * (2.0 - x[q])).reshape([-1 if d == q else 1 for d in range(3)])
            f += prof
        for q, ax in enumerate("xyz"):  # exact zeros on the walls, odd ghosts
            if ax not in walls:
                continue
            ix = [slice(None)] * 3
            at = lambda s: tuple(ix[:q] + [s] + ix[q + 1:])  # noqa: E731
            if q == c:
                f[at(0)] = 0.0
                f[at(1)] = 0.0
                f[at(n[q] + 1)] = 0.0
            else:
                f[at(0)] = -f[at(1)]
                f[at(n[q] + 1)] = -f[at(n[q])]
        out.append(f)
    return out


def _slots(case, seed):
    """u, v, w slot arrays on the GPU, the viscosity and the time step (CFL 0.3)."""
    n, L = (case["nx"], case["ny"], case["nz"]), _ext(case)
    f = _wall_field(n, L, case["walls"], seed) if case["walls"] else _periodic_field(n, L, seed)
    umax = max(float(q.abs().max()) for q in f)
    return f, _nu(max(n)), 0.3 * min(l / m for l, m in zip(L, n)) / umax


def _ref(f, c):
    """A slot array in the reference's padded shape (the component's own axis has no slot 0)."""
    return f[(slice(None),) * c + (slice(1, None),)] if c < 3 else f


def _host(f, c):
    """The same as a Fortran-ordered host array."""
    return _ref(f, c).permute(2, 1, 0).contiguous().cpu().numpy().transpose(2, 1, 0)


def _config(case, nu, dt, **kw):
    bc = [2 if ax in case["walls"] else 1 for ax in "xyz"]
    pbc = [3 if ax in case["walls"] else 1 for ax in "xyz"]
    L = _ext(case)
    return api.make_config(case["nx"], case["ny"], case["nz"], lx=L[0], ly=L[1], lz=L[2], nu=nu, dt=dt,
                           scheme=case["scheme"], dp_flag=case["dp_flag"], bc=bc, pbc=pbc, **kw)


def _pinned(count):
    return torch.empty(count, dtype=torch.float64, pin_memory=True)


def _ptr(t, offset=0):
    return ctypes.cast(t.data_ptr() + 8 * offset, ctypes.POINTER(ctypes.c_double))


KEYS = ("u", "v", "w", "p", "hx", "hy", "hz")


def _state_buffers(shapes):
    return {k: _pinned(int(np.prod(shapes[{"hx": "u", "hy": "v", "hz": "w"}.get(k, k)]))) for k in KEYS}


def _prepare_session(case, seed):
    f, nu, dt = _slots(case, seed)
    s = api.Session(_config(case, nu, dt))
    u, v, w = (_host(q, c) for c, q in enumerate(f))
    s.set_state(u, v, w, np.zeros(s.shapes["p"], order="F"))
    return {"session": s, "out": _state_buffers(s.shapes)}


def _prepare_host(case, seed):
    """A driver in mid-run: the state and the AB2 history after two steps, in pinned memory."""
    st = _prepare_session(case, seed)
    s = st["session"]
    s.step(2)
    st["in"] = _state_buffers(s.shapes)
    s._check(s.lib.ns_get_state(s.h, *[_ptr(st["in"][k]) for k in KEYS]))
    return st


def _prepare_poisson(case, seed):
    n = (case["nx"], case["ny"], case["nz"])
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = torch.randn(n[::-1], generator=g, device=DEV, dtype=torch.float64)
    return {"rhs": r - r.mean(), "n": n, "lib": _lib.load(),
            "dp": torch.zeros(tuple(m + 2 for m in n[::-1]), device=DEV, dtype=torch.float64)}


def _subs(case):
    r = np.random.default_rng(case["subs_seed"])
    edges = np.array([e for e in (16, 24, 32, 48, 64) if e <= case["edge_max"]])
    out = []
    for _ in range(case["count"]):
        n = [int(e) for e in r.choice(edges, 3)]
        ratio = 1 if case["scheme"] == AB2_CN else int(r.choice([1, 2, 4]))
        out.append((*[int(r.integers(1, case["parent"] + 2 - e)) for e in n], *n, ratio))
    return out


def _prepare_batch(case, seed):
    """The parent run up to the last snapshot that the intervals need, captured on the device; the
    parent then stands at the start of the re-simulated window again."""
    n, n0, T = case["parent"], 3, case["intervals"]
    par = {"nx": n, "ny": n, "nz": n, "walls": "", "scheme": case["scheme"], "dp_flag": 1}
    f, nu, dt = _slots(par, seed)
    s = api.Session(_config(par, nu, dt, keep_sweeps=int(case["scheme"] == AB2_CN)))
    s.set_state(*[_host(q, c) for c, q in enumerate(f)], np.zeros(s.shapes["p"], order="F"))
    subs, h = _subs(case), 2.0 * PI / n
    b = api.Batch(subs, scheme=case["scheme"], bc=2, pbc=3, nu=nu, dt0=dt, dx=h, dy=h, dz=h, n_slots=T + n0 + 8,
                  use_graph=1, restart=1)
    for k in range(1, T + n0 + 7):
        s.step(1)
        b.capture(s, k, k * dt)
        if k == n0:
            start = s.get_state()
    s.set_state(*[start[k] for k in ("u", "v", "w", "p")], [start[k] for k in ("hx", "hy", "hz")])
    s.synchronize()
    sizes = {k: [int(np.prod(b.shapes(i)[{"hx": "u", "hy": "v", "hz": "w"}.get(k, k)])) for i in range(len(subs))]
             for k in KEYS}
    at = {k: np.concatenate([[0], np.cumsum(v)]) for k, v in sizes.items()}
    return {"parent": s, "batch": b, "out": {k: _pinned(int(at[k][-1])) for k in KEYS}, "at": at, "t0": n0 * dt,
            "dt": dt, "T": T}


def _prepare_adjoint(case, seed):
    n = case["n"]
    box = {"nx": n, "ny": n, "nz": n, "walls": "", "scheme": AB2_CN, "dp_flag": 0}
    f, nu, dt = _slots(box, seed)
    s = api.Session(_config(box, nu, dt))
    s.set_state(*[_host(q, c) for c, q in enumerate(f)], np.zeros(s.shapes["p"], order="F"))
    g = _periodic_field((n, n, n), None, seed + 7919)
    pin = lambda shape: _pinned(int(np.prod(shape))).numpy().reshape(shape, order="F")  # noqa: E731
    seeds = []
    for c, k in enumerate("uvw"):
        a = pin(s.shapes[k])
        a[...] = _host(g[c], c)
        seeds.append(a)
    return {"session": s, "seeds": seeds, "out": {k: pin(s.shapes[k]) for k in "uvw"}}


def prepare(case, seed):
    st = {"session": _prepare_session, "host": _prepare_host, "poisson": _prepare_poisson, "batch": _prepare_batch,
          "adjoint": _prepare_adjoint}[case["kind"]](case, seed)
    st["case"] = case
    return st


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "session":
        s = st["session"]
        s.step(case["steps"])
        s._check(s.lib.ns_get_state(s.h, *[_ptr(st["out"][k]) for k in KEYS]))
        return st["out"]
    if kind == "host":
        s = st["session"]
        s._check(s.lib.ns_step_host(s.h, *[_ptr(st["in"][k]) for k in KEYS], *[_ptr(st["out"][k]) for k in KEYS]))
        return st["out"]
    if kind == "poisson":
        n = st["n"]
        rc = st["lib"].ns_poisson_fft_noalloc(
            ctypes.c_void_p(st["rhs"].data_ptr()), ctypes.c_void_p(st["dp"].data_ptr()), *n, 2.0 * PI, 2.0 * PI,
            2.0 * PI, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError("ns_poisson_fft_noalloc: %d" % rc)
        return st["dp"]
    if kind == "batch":
        b = st["batch"]
        b.init_from_parent(st["parent"])
        for q in range(st["T"]):
            b.advance(st["t0"] + q * st["dt"])
        for i in range(case["count"]):
            b._check(b.lib.ns_batch_get_state(b.h, i, *[_ptr(st["out"][k], int(st["at"][k][i])) for k in KEYS]))
        return st["out"]
    s = st["session"]
    s.adj_forward(case["steps"], case["ckpt_every"])
    return s.adj_backward(*st["seeds"], out=st["out"])


def work(case):
    """Per step the state is read and written once (u, v, w, the history, p), and about 60 operations a
    cell are the stencils, 45 the line solves, the rest the transforms; a snapshot is written once."""
    kind = case["kind"]
    if kind == "poisson":
        m = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 16.0 * m, "flops": m * (5.0 * math.log2(m) + 2.0)}
    if kind == "batch":
        cells = [(a * b * c, r) for _, _, _, a, b, c, r in _subs(case)]
        m = sum(c * (r + case["intervals"] - 1) for c, r in cells)
        once = sum(c for c, _ in cells)
        return {"bytes": 13 * 8.0 * m + 14 * 8.0 * once, "flops": m * (75.0 + 5.0 * 15.0)}
    if kind == "adjoint":
        m = case["n"] ** 3
        steps = case["steps"] * 3.0  # forward, recomputed, backward
        return {"bytes": 13 * 8.0 * m * steps + 6 * 8.0 * m, "flops": m * steps * (120.0 + 5.0 * math.log2(m))}
    m = case["nx"] * case["ny"] * case["nz"]
    steps = case.get("steps", 1)
    ops = 75.0 + (45.0 if case["scheme"] == AB2_CN else 0.0) + 5.0 * math.log2(m)
    return {"bytes": 13 * 8.0 * m * steps + 14 * 8.0 * m * (kind == "host") + 7 * 8.0 * m * (kind == "session"),
            "flops": m * steps * ops}


# ---------------------------------------------------------------------------------------------
# the same in plain 64-bit torch
# ---------------------------------------------------------------------------------------------
def _sh(a, q, d):
    """Interior slots of a slot array, shifted by d along axis q (d may be a list of (axis, shift))."""
    off = [0, 0, 0]
    for ax, s in ([(q, d)] if q is not None else d):
        off[ax] += s
    return a[tuple(slice(1 + o, a.shape[i] - 1 + o) for i, o in enumerate(off))]


def _poisson_slots(R, n, h, walls):
    """The interior solution of the discrete Poisson problem of zero mean (periodic / Neumann axes)."""
    F, lam, Q = R.to(torch.complex128), torch.zeros((1, 1, 1), device=R.device, dtype=torch.float64), {}
    for q, ax in enumerate("xyz"):
        m = torch.arange(n[q], device=R.device, dtype=torch.float64)
        if ax in walls:
            C = torch.cos(PI / (2 * n[q]) * m[:, None] * (2 * m[None, :] + 1)) * math.sqrt(2.0 / n[q])
            C[0] /= math.sqrt(2.0)
            Q[q] = C.to(torch.complex128)
            F = torch.tensordot(Q[q], F, dims=([1], [q])).movedim(0, q)
            e = -4.0 * torch.sin(PI * m / (2 * n[q])) ** 2 / h[q] ** 2
        else:
            F = torch.fft.fft(F, dim=q)
            e = -4.0 * torch.sin(PI * m / n[q]) ** 2 / h[q] ** 2
        lam = lam + e.reshape([-1 if d == q else 1 for d in range(3)])
    lam[0, 0, 0] = math.inf
    F = F / lam
    for q in range(3):
        F = torch.tensordot(Q[q].T, F, dims=([1], [q])).movedim(0, q) if q in Q else torch.fft.ifft(F, dim=q)
    return F.real


def _cn_matrix(n, a, normal, wall):
    """The Crank-Nicolson rows of one axis on the slots they solve for, and the first of those slots.
    The periodic normal component closes its first row on its own duplicate face."""
    dg, of = 1.0 + 2.0 * a, -a
    m = n if not wall else (n + 1 if normal else n + 2)
    A = torch.zeros((m, m), dtype=torch.float64)
    for d, val in ((0, dg), (1, of), (-1, of)):
        A.diagonal(d).fill_(val)
    if not wall:
        A[m - 1, 0] += of
        A[0, 0 if normal else m - 1] += of
        return A, 1
    A[0] = 0.0
    A[m - 1] = 0.0
    if normal:
        A[0, 0] = A[m - 1, m - 1] = 1.0
        return A, 1
    A[0, 0] = A[0, 1] = A[m - 1, m - 1] = A[m - 1, m - 2] = 0.5
    return A, 0


def _at(q, s):
    return tuple(s if d == q else slice(None) for d in range(3))


def _exact_steps(case, f, nu, dt, steps):
    n, L, walls = (case["nx"], case["ny"], case["nz"]), _ext(case), case["walls"]
    h = [l / m for l, m in zip(L, n)]
    per = [ax not in walls for ax in "xyz"]
    scheme, dpf = case["scheme"], case["dp_flag"]
    U = [q.clone() for q in f]
    p = torch.zeros_like(U[0])
    H = [torch.zeros_like(U[0]) for _ in range(3)]
    act = []
    for c in range(3):
        a = torch.zeros_like(U[0], dtype=torch.bool)
        a[tuple(slice(1 if per[c] or q != c else 2, n[q] + 1) for q in range(3))] = True
        act.append(a)
    lus = {}
    if scheme == AB2_CN:
        for q in range(3):
            for normal in (True, False):
                A, s0 = _cn_matrix(n[q], 0.5 * dt * nu / h[q] ** 2, normal, not per[q])
                lus[q, normal] = (*torch.linalg.lu_factor(A.to(DEV)), s0, A.shape[0])
    for it in range(steps):
        S = []
        for c in range(3):
            conv, lap = 0.0, 0.0
            for q in range(3):
                if q == c:
                    hi, lo = _sh(U[c], c, 0) + _sh(U[c], c, 1), _sh(U[c], c, -1) + _sh(U[c], c, 0)
                    conv = conv + (hi * hi - lo * lo) / (4.0 * h[c])
                else:
                    hi = (_sh(U[c], q, 0) + _sh(U[c], q, 1)) * (
                        _sh(U[q], None, [(c, -1), (q, 1)]) + _sh(U[q], q, 1))
                    lo = (_sh(U[c], q, -1) + _sh(U[c], q, 0)) * (_sh(U[q], c, -1) + _sh(U[q], c, 0))
                    conv = conv + (hi - lo) / (4.0 * h[q])
                lap = lap + (_sh(U[c], q, -1) - 2.0 * _sh(U[c], q, 0) + _sh(U[c], q, 1)) / h[q] ** 2
            gp = (_sh(p, c, 0) - _sh(p, c, -1)) / h[c]
            first = it == 0
            prev = _sh(H[c], c, 0)
            if scheme == AB2_CN:
                new = -conv
                r = 0.5 * nu * lap - (1.0 if first else 1.5) * conv - (0.0 if first else 0.5) * prev
            else:
                new = nu * lap - conv
                r = new if first or scheme == EULER else 1.5 * new - 0.5 * prev
            a = _sh(act[c], c, 0)
            X = U[c].clone()
            _sh(X, c, 0)[a] = (_sh(U[c], c, 0) + dt * (r - dpf * gp))[a]
            _sh(H[c], c, 0)[a] = new[a] if scheme != EULER else 0.0
            S.append(X)
        for q in range(3):  # boundary values, or the line solves with their boundary rows
            for c in range(3):
                X = S[c]
                if scheme == AB2_CN:
                    lu, piv, s0, m = lus[q, c == q]
                    B = X.movedim(q, 0)[s0:s0 + m].clone()
                    if not per[q]:
                        B[0] = 0.0
                        B[-1] = 0.0
                    Y = torch.linalg.lu_solve(lu, piv, B.reshape(m, -1)).reshape(B.shape)
                    X.movedim(q, 0)[s0:s0 + m] = Y
                elif not per[q]:
                    if c == q:
                        X[_at(q, 1)] = 0.0
                        X[_at(q, n[q] + 1)] = 0.0
                    else:
                        X[_at(q, 0)] = -X[_at(q, 1)]
                        X[_at(q, n[q] + 1)] = -X[_at(q, n[q])]
                if per[q]:
                    X[_at(q, 0)] = X[_at(q, n[q])]
                    X[_at(q, n[q] + 1)] = X[_at(q, 1)]
        R = sum((_sh(S[c], c, 1) - _sh(S[c], c, 0)) / h[c] for c in range(3)) / dt
        dp = torch.zeros_like(p)
        dp[1:-1, 1:-1, 1:-1] = _poisson_slots(R, n, h, walls)
        for q in range(3):
            dp[_at(q, 0)] = dp[_at(q, n[q] if per[q] else 1)]
            dp[_at(q, n[q] + 1)] = dp[_at(q, 1 if per[q] else n[q])]
        dp = dp - dp[0, 0, 0].clone()
        for c in range(3):
            U[c] = S[c].clone()
            U[c][_at(c, slice(1, None))] -= dt * torch.diff(dp, dim=c) / h[c]
            if per[c]:
                U[c][_at(c, 0)] = U[c][_at(c, n[c])]
        p = dpf * p + dp
    return U, p, H


def _flat(f, c):
    return _ref(f, c).permute(2, 1, 0).reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        n = (case["nx"], case["ny"], case["nz"])
        R = _prepare_poisson(case, seed)["rhs"].permute(2, 1, 0)
        x = _poisson_slots(R, n, [2.0 * PI / m for m in n], "")
        return torch.nn.functional.pad(x[None, None], (1, 1, 1, 1, 1, 1), mode="circular")[0, 0].permute(
            2, 1, 0).contiguous()
    if kind not in ("session", "host"):
        return None  # an independent restatement of these takes far longer than the call
    f, nu, dt = _slots(case, seed)
    U, p, H = _exact_steps(case, f, nu, dt, case["steps"] if kind == "session" else 3)
    return {"u": _flat(U[0], 0), "v": _flat(U[1], 1), "w": _flat(U[2], 2), "p": _flat(p, 3),
            "hx": _flat(H[0], 0), "hy": _flat(H[1], 1), "hz": _flat(H[2], 2)}
