"""The work whose time on the GPU is measured: cycles of the ladder on every field solver, from the smallest grid to the
largest, the batched sweep, the accelerator hook with the state on the host, and the separable inverse alone.

A pass of a cycle case is one protocol cycle (lMax = 40 steps) of a run under way: `prepare` builds the context, takes
the state up and steps one cycle, as every cycle of a ladder but its first finds it.  Outputs are the state the pass
left, on the device where the program keeps it there (views of the library's buffers, no copy), and what the voltmeter
read.  Sizes are those of the benchmark, the sweep and the tests, or odd ones between them.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

import juliatdgl_b200 as T
from juliatdgl_b200 import abi, gpu, protocol, sweep, workloads
from juliatdgl_b200.grid import sculpt, with_materials

LMAX = 40
RAMP_TURN = 20000          # the current ramp goes up for this many steps, then down again
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # the smallest run: every cycle is launches and latency (two KWT bands, the 12×8×4 parity size)
        dict(name="cycle_kwt_12x8x4", kind="kwt", nx=12, ny=8, nz=4, buf=1),
        # one run of the onset sweep alone: its smallest grid and its largest
        dict(name="cycle_plain_64x32x8", kind="plain", nx=64, ny=32, nz=8, buf=1),
        dict(name="cycle_plain_192x64x16", kind="plain", nx=192, ny=64, nz=16, buf=1),
        # thermal noise on an odd grid (KWT: SK-ROCK stages, the smoothed rotating frame)
        dict(name="cycle_noise_101x37x9", kind="noise", nx=101, ny=37, nz=9, buf=1),
        # the heat model with the Joule term
        dict(name="cycle_heat_96x48x8", kind="heat", nx=96, ny=48, nz=8, buf=1),
        # a sculpted sample with two normal fluids and the insulating padding (two conjugate-gradient solves a step)
        dict(name="cycle_fluids_40x20x8", kind="fluids", nx=40, ny=20, nz=8, buf=2),
        # the three-band ramp with padding and the open boundary: the parity tests' size, and the benchmark's
        dict(name="cycle_ramp_64x32x8", kind="ramp", nx=64, ny=32, nz=8, buf=2),
        dict(name="cycle_ramp_256x128x32", kind="ramp", nx=256, ny=128, nz=32, buf=8),
        # materials, noise on bands and field, the open boundary, and y-z planes of the large bilayer
        dict(name="cycle_bilayer_64x256x64", kind="bilayer", nx=64, ny=256, nz=64, buf=16),
        # the sweep's runs as one batch
        dict(name="batch_16", kind="batch", runs=16, mix=2),
        # the accelerator hook: state and carry go up and come back around the cycle
        dict(name="hook_ramp_128x64x16", kind="hook", nx=128, ny=64, nz=16, buf=4),
        # the separable inverse for callers with their own device memory (its largest grid in the tests)
        dict(name="sep_192x64x16", kind="sep", nx=192, ny=64, nz=16, buf=1),
    ]


def draw(rng):
    kind = rng.choice(["kwt", "plain", "plain", "noise", "heat", "fluids", "ramp", "ramp", "bilayer", "batch", "hook",
                       "sep"])
    lu = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    if kind == "batch":
        return dict(kind=kind, runs=rng.randint(4, 24), mix=rng.randint(3, 999))
    if kind in ("ramp", "hook"):
        big = kind == "ramp"
        return dict(kind=kind, nx=lu(24, 256 if big else 128), ny=lu(12, 128 if big else 64), nz=lu(4, 32 if big else 16),
                    buf=rng.randint(2, 8 if big else 4))
    if kind == "bilayer":
        return dict(kind=kind, nx=lu(24, 64), ny=lu(48, 240), nz=lu(16, 60), buf=rng.randint(4, 16))
    if kind == "fluids":
        return dict(kind=kind, nx=lu(20, 48), ny=lu(8, 24), nz=lu(4, 10), buf=rng.randint(2, 3))
    if kind == "sep":
        return dict(kind=kind, nx=lu(12, 192), ny=lu(8, 64), nz=lu(4, 16), buf=rng.randint(1, 2))
    return dict(kind=kind, nx=lu(12, 192), ny=lu(8, 64), nz=lu(4, 16), buf=rng.randint(1, 2))


# ------------------------------------------------------------------------------------------------ the host's plans
def _bilayer(gr):
    """Two layers and a thin barrier of a third material, band 3 absent from the upper one."""
    ax = lambda m: (m, m, 4 * m)

    def bands(sm, sg, third):
        return (T.Band.make(m_axes=ax(1.0 * sm), Γ=1.0 * sg, a=1.0),
                T.Band.make(m_axes=ax(sm / (16 * 0.59)), Γ=1.0 * sg, a=0.59),
                T.Band.make(m_axes=ax(2.0 * sm), Γ=1.2 * sg, a=third))

    lower = T.Model.make(bands(1.1, 0.9, 0.8), [[0.0, 1e-3, -0.02], [1e-3, 0.0, -0.02], [-0.02, -0.02, 0.0]],
                         κ=25.0, σn=1.05, T=0.5)
    upper = T.Model.make(bands(0.95, 1.1, 0.4), [[0.0, 1e-3, 0.0], [1e-3, 0.0, 0.0], [0.0, 0.0, 0.0]],
                         κ=25.0, σn=0.9, T=0.5)
    barrier = T.Model.make(lower.bands, lower.γ, κ=25.0, σn=1.15, T=0.5)
    kmid = gr.z1 + (gr.z2 - gr.z1) // 2
    k = np.arange(1, gr.Nz + 2)
    layer = np.where(k <= kmid, 1, np.where(k <= kmid + 2, 3, 2)).astype(np.uint8)
    mk = with_materials(T.box_masks(gr), gr, np.asfortranarray(np.broadcast_to(layer[None, None, :], gr.node)))
    st = T.Stepper.make(lower, gr, mk, materials=[upper, barrier], absent=[[], [3], []],
                        transparency=[[1.0, 1.0, 0.3], [1.0, 1.0, 0.3], [0.3, 0.3, 1.0]], σvac=0.01,
                        selffield_bc="open", pcg_tol=1e-10, noise=0.005, noise_seed=4, noise_field=True)
    return st, T.initial_state(lower, gr, mk, 0.03, materials=st.mt.models), 0.03


@functools.lru_cache(maxsize=4)
def _plan(kind, nx, ny, nz, buf):
    """(Stepper, seed state, H): what a program computes once per sample."""
    if kind in ("ramp", "hook"):
        return workloads.ramp(nx, ny, nz, buf)
    gr = T.Grid.make(nx, ny, nz, dx=0.5, buf=buf)
    if kind == "bilayer":
        return _bilayer(gr)
    wedge = T.build_masks(T.GeomSpec(GEOM_MODE="WEDGE", wedge_depth=0.3), gr)
    kw = {}
    if kind == "kwt":                      # the two-band parity model
        b = (T.Band.make(γkwt=10.0), T.Band.make(g=0.6, Γ=1.5, a=0.8, γkwt=5.0))
        md, H, kw = T.Model.make(b, [[0.0, -0.05], [-0.05, 0.0]], κ=25.0), 0.3, dict(dt=0.01)
    elif kind == "plain":                  # the sweep's model
        md, H = T.two_band(xi_ratio=4.0, κ=25.0), 0.2
    elif kind == "noise":
        md, H, kw = T.two_band(xi_ratio=4.0, κ=25.0, gamma_kwt=10.0), 0.2, dict(noise=1e-3, noise_seed=8)
    elif kind == "heat":
        md, H = T.two_band(xi_ratio=4.0, κ=25.0, gamma_kwt=3.0), 0.2
        kw = dict(heat=T.Heat(eta=0.5, joule=True, margin=2))
    elif kind == "fluids":                 # a vacuum slot from the y1 face, and an exchange rate of 1
        md, H = T.two_band(xi_ratio=4.0, κ=2.0, gamma_kwt=10.0), 0.03
        v = np.zeros(gr.node, dtype=bool)
        x0 = gr.x1 + nx // 4
        v[x0:x0 + max(2, nx // 4), gr.y1:gr.y1 + max(2, ny // 3), gr.z1:gr.z2] = True
        wedge, kw = sculpt(T.box_masks(gr), gr, v), dict(σvac=0.01, pcg_tol=1e-10, qp_exchange=1.0)
    else:
        raise KeyError(kind)
    st = T.Stepper.make(md, gr, wedge, **kw)
    return st, T.initial_state(md, gr, wedge, H), H


def _args(case):
    return case["kind"], case["nx"], case["ny"], case["nz"], case["buf"]


def _start(s, rng):
    """The seed state with smooth random dips of |Ψ| (up to 10 %) and phases, as a run some time on has them: waves of
    eight nodes and longer, so that neighbouring nodes stay as near as the dynamics keep them."""
    s = s.copy()

    def waves(shape):
        out = 0.0
        for _ in range(3):
            w = 1.0
            for ax, n in enumerate(shape):
                k = 2 * math.pi / float(rng.uniform(8, 32))
                c = np.cos(k * np.arange(n) + float(rng.uniform(0, 2 * math.pi)))
                w = w * c.reshape([-1 if x == ax else 1 for x in range(3)])
            out = out + w / 3
        return out

    for µ in range(s.N):
        shape = s.G[µ].shape
        a, p = waves(shape), waves(shape)
        s.G[µ][...] *= (0.95 + 0.05 * a) * np.exp(0.1j * p)
        s.F[µ][...] = s.G[µ]
    return s


def _current(rng):
    return float(rng.uniform(0.01, 0.05)) * (1 if rng.random() < 0.5 else -1)


def _ramp(st, q, n, polarity):
    """HJ of steps q .. q + n − 1 of the current ramp, up and down."""
    hj = workloads.ramp_hj(st, polarity)
    return [hj(RAMP_TURN - abs(p % (2 * RAMP_TURN) - RAMP_TURN)) for p in range(q, q + n)]


# ------------------------------------------------------------------------------------------------ device state
class _Buffer:
    """A field of a context's resident state as torch reads it; holds the context as long as the view lives."""

    def __init__(self, gs, ptr, shape, node, cplx):
        self.gs = gs
        e = 16 if cplx else 8
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<c16" if cplx else "<f8", "version": 3,
                                         "strides": (e, e * node[0], e * node[0] * node[1]), "data": (ptr, False)}


def _resident(gs):
    """Ψ, θ, V, J and h of the resident state: views of the library's device arrays (all stored with the node shape)."""
    gr, v = gs.st.grid, abi.StateView_t()
    rc = gpu.lib().tdgl_device_state(gs.h, C.byref(v))
    if rc:
        raise gpu.TDGLError(rc, "device state")
    node = gr.node
    link, face = (gr.xlink, gr.ylink, gr.zlink), (gr.hx_shape, gr.hy_shape, gr.hz_shape)
    get = lambda p, shape, cplx=False: torch.as_tensor(
        _Buffer(gs, C.cast(p, C.c_void_p).value, shape, node, cplx), device="cuda")
    return {"psi": [get(v.G[µ], node, True) for µ in range(gs.st.model.N)],
            "theta": [get(v.th[a], link[a]) for a in range(3)], "V": [get(v.V[a], link[a], True) for a in range(3)],
            "J": [get(v.J[a], link[a]) for a in range(3)], "h": [get(v.h[a], face[a]) for a in range(3)]}


def _vector(parts):
    """The three components of a vector field as one array."""
    return torch.cat([p.permute(2, 1, 0).reshape(-1) for p in parts])


# ------------------------------------------------------------------------------------------------ the cases
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "sep":
        gr = T.Grid.make(case["nx"], case["ny"], case["nz"], dx=0.5, buf=case["buf"])
        g = torch.Generator(device=DEV).manual_seed(int(seed))
        shape = (gr.Nx + 1, gr.Nz + 1, gr.Ny + 1)            # plane-major: j fastest, then k, then i
        b = [torch.randn(shape, generator=g, device=DEV, dtype=torch.float64) for _ in range(3)]
        return {"kind": kind, "grid": gr, "b": b, "z": [torch.zeros_like(t) for t in b]}
    if kind == "batch":
        runs = _sweep(case["runs"], case["mix"])
        ctxs = []
        for r in runs:
            gs = gpu.GPUStepper(r.st)
            gs.upload(_start(r.s, rng))
            ctxs.append(gs)
        bt = gpu.Batch(ctxs)
        state = {"kind": kind, "ctxs": ctxs, "batch": bt, "H": [r.H for r in runs], "HJ": [r.HJ for r in runs]}
        bt.steps(LMAX, state["H"], state["HJ"])
        return state
    st, s, H = _plan(*_args(case))
    state = {"kind": kind, "st": st, "H": H}
    s = _start(s, rng)
    gs = state["gs"] = gpu.GPUStepper(st)
    if kind in ("ramp", "hook", "bilayer"):
        state["q"], state["polarity"] = 4000, (1 if rng.random() < 0.5 else -1)
    else:
        state["HJ"] = T.selffield(st, _current(rng))
    if kind == "hook":
        state["s"], state["carry"] = s, abi.Carry(st)
        run(state)
        return state
    gs.upload(s)
    _cycle(state)
    if kind in ("kwt", "plain", "noise", "heat"):
        gs.meter_set(protocol.voltmeter(st.grid, st.masks, max(1, min(8, case["nx"] // 4))))
    return state


@functools.lru_cache(maxsize=2)
def _sweep(n, mix):
    return sweep.sweep_instances(n, seed=mix)


def _steps(kind):
    """Steps of a pass: a cycle of the ladder, and a quarter of one on the large bilayer."""
    return LMAX // 4 if kind == "bilayer" else LMAX


def _cycle(state):
    gs = state["gs"]
    if "q" in state:
        n = _steps(state["kind"])
        rc = gs.steps_ramp(state["H"], _ramp(gs.st, state["q"], n, state["polarity"]))
        state["q"] += n
    else:
        rc = gs.steps(LMAX, state["H"], state["HJ"])
    if rc:
        raise gpu.TDGLError(rc, "the field solve did not converge")


def run(state):
    kind = state["kind"]
    if kind == "sep":
        gr, b, z = state["grid"], state["b"], state["z"]
        g = abi.Grid_t(gr.Nx, gr.Ny, gr.Nz, gr.x1, gr.x2, gr.y1, gr.y2, gr.z1, gr.z2, gr.dx, gr.dy, gr.dz)
        bp, zp = ((C.c_void_p * 3)(*[t.data_ptr() for t in v]) for v in (b, z))
        rc = gpu.lib().tdgl_sep_apply_noalloc(C.byref(g), C.c_double(SEP_A), bp, zp,
                                              C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise gpu.TDGLError(rc, "sep_apply_noalloc")
        return z
    if kind == "batch":
        rc = state["batch"].steps(LMAX, state["H"], state["HJ"])
        if rc:
            raise gpu.TDGLError(rc, "batch")
        return [{"psi": r["psi"][0], "psi2": r["psi"][1]} for r in map(_resident, state["ctxs"])]
    if kind == "hook":                     # one call of the accelerator hook
        gs, s, carry = state["gs"], state["s"], state["carry"]
        gs.upload(s)
        gs.set_carry(carry)
        _cycle(state)
        gs.get_carry(carry)
        gs.download(s)
        vec = lambda c: np.concatenate([getattr(s, c + x).ravel(order="F") for x in "xyz"])
        return {"psi": list(s.G), "V": [s.Vx, s.Vy, s.Vz], "U": [s.Ux, s.Uy, s.Uz], "J": vec("J"), "h": vec("h")}
    _cycle(state)
    gs = state["gs"]
    out = _resident(gs)
    if kind in ("kwt", "plain", "noise", "heat"):
        o = gs.measure()                   # the ladder's voltmeter
        out["obs"] = {k: o[k] for k in ("D", "vsum_in", "vsum_out", "ta_sum", "Itot", "Isam")}
        return out
    # behind an iterative solve a component of J or h is only as good as the field: each as one vector; the link phases
    # as the links V = e^{−iθ} (the longitudinal part of θ in the padding is known to the solve's tolerance only)
    return {"psi": out["psi"], "V": out["V"], "J": _vector(out["J"]), "h": _vector(out["h"])}


SEP_A = 49.5               # (dt/σn) κ²/dx² of the sweep's and the ramp's model


def work(case):
    """Per step: every field the step reads in and every field it makes out, once (Ψ, θ, V, h and the masks in; Ψ, θ,
    V, J and h out), and the arithmetic of one stage per band, the currents, the links and one field solve."""
    if case["kind"] == "batch":
        each = [(np.prod([float(x) for x in r.st.grid.node]), 2, r.st.grid, False) for r in _sweep(case["runs"], case["mix"])]
    else:
        gr = T.Grid.make(case["nx"], case["ny"], case["nz"], dx=0.5, buf=case["buf"])
        bands = 3 if case["kind"] in ("ramp", "hook", "bilayer") else 2
        each = [(np.prod([float(x) for x in gr.node]), bands, gr, case["kind"] in ("ramp", "hook", "bilayer", "fluids"))]
    by = fl = 0.0
    for n, nb, gr, pcg in each:
        solve = 3 * n * (2 * 2 * (gr.Ny + gr.Nz) + 40)     # both directions of the y and z products, the x lines
        if case["kind"] == "sep":
            by, fl = by + 48 * n, fl + solve
            continue
        k = _steps(case["kind"])
        by += k * n * (32 * nb + 3 * (16 + 32 + 8 + 16) + 32 + (24 if pcg else 0))
        fl += k * (n * (nb * 150 + 250) + solve)
        if case["kind"] == "hook":
            by += 2 * n * (32 * nb + 3 * 64)               # the state up and down
    return {"bytes": float(by), "flops": float(fl)}


# ------------------------------------------------------------------------------------------------ in 64 bits
def exact(case, seed):
    """The separable inverse by its three dense transforms, and the cycles of one material with the direct field
    solve as the scheme's formulas give them; None for noise, heat and the iterative solves."""
    if case["kind"] == "sep":
        return _exact_sep(case, seed)
    if case["kind"] in ("kwt", "plain") and case["nx"] * case["ny"] * case["nz"] <= 300_000:
        rng = np.random.default_rng(seed)
        st, s, H = _plan(*_args(case))
        s = _start(s, rng)
        p = _Plain(st, s)
        HJ = T.selffield(st, _current(rng))
        for _ in range(2 * LMAX):
            p.step(H, HJ)
        return {"psi": p.G, "theta": p.th, "V": p.V, "J": p.J, "h": p.h, "obs": None}
    return None


def _bases(n):
    """The eigenbases of the second difference of n points (rows: modes) on points and on edges, and |k|."""
    k = torch.arange(n, device=DEV, dtype=torch.float64)
    i = torch.arange(n, device=DEV, dtype=torch.float64)
    V = torch.cos(math.pi * k[:, None] * (i[None, :] + 0.5) / n) * math.sqrt(2.0 / n)
    V[0] = math.sqrt(1.0 / n)
    U = torch.zeros(n, n - 1, device=DEV, dtype=torch.float64)
    U[1:] = -math.sqrt(2.0 / n) * torch.sin(math.pi * k[1:, None] * (i[None, :-1] + 1.0) / n)
    return V, U, 2 * torch.sin(math.pi * k / (2.0 * n))


def _along(M, X):
    """X with the matrices M applied along its three axes."""
    X = torch.tensordot(M[0], X, dims=([1], [0]))
    X = torch.tensordot(M[1], X, dims=([1], [1])).permute(1, 0, 2)
    return torch.tensordot(X, M[2], dims=([2], [1]))


def _sep_solve(b, n, a):
    """(I + aK)⁻¹ on the three link components b (x, y, z order) over n points an axis."""
    V, U, s = zip(*(_bases(m) for m in n))
    M = [[U[x] if x == c else V[x] for x in range(3)] for c in range(3)]
    hat = [_along(M[c], b[c]) for c in range(3)]
    s = [s[0][:, None, None], s[1][None, :, None], s[2][None, None, :]]
    c0 = 1 + a * (s[0] ** 2 + s[1] ** 2 + s[2] ** 2)
    dot = a * sum(s[c] * hat[c] for c in range(3))
    return [_along([m.T for m in M[c]], (hat[c] + s[c] * dot) / c0) for c in range(3)]


def _exact_sep(case, seed):
    state = prepare(case, seed)
    gr, out = state["grid"], [t.clone() for t in state["z"]]
    n = (gr.Nx - 1, gr.Ny - 1, gr.Nz - 1)
    sl = [tuple(slice(1, 1 + n[x] - (x == c)) for x in (0, 2, 1)) for c in range(3)]
    z = _sep_solve([state["b"][c][sl[c]].permute(0, 2, 1) for c in range(3)], n, SEP_A)
    for c in range(3):
        out[c][sl[c]] = z[c].permute(0, 2, 1)
    return out


def _cis(a, short):
    """e^{ia}, by the scheme's short series where `short`."""
    s = torch.complex(1 - a * a / 2, a * (1 - a * a / 6))
    return torch.where(short, s, torch.polar(torch.ones_like(a), a))


def _turned(V, U):
    """The angle of V U*, and where the scheme takes it by its short series."""
    q = V * U.conj()
    short = (q.real > 0) & (q.imag.abs() <= 0.05)
    return torch.where(short, q.imag + q.imag ** 3 / 6, torch.angle(q)), short


class _Plain:
    """The step of one material with RKL or damped RKC stages (or one Euler pass), the bar field and the separable
    solve, in plain torch."""

    def __init__(self, st, s):
        gr = st.grid
        if st.rkl is None or st.solver != 2 or st.selffield_bc != 1 or any(st.rkl[µ] == 0 and st.nsub[µ] > 1
                                                                          for µ in range(st.N)):
            raise ValueError("not a scheme of this form")
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
        self.st, self.gr = st, gr
        self.G = [up(g) for g in s.G]
        for k in "θφVUJh":
            setattr(self, {"θ": "th", "φ": "ph"}.get(k, k), [up(getattr(s, k + x)) for x in "xyz"])
        self.f, self.tau = up(st.masks.f), [up(getattr(st.masks, "τ" + x)) for x in "xyz"]
        self.bar = {k: up(getattr(st.bar, k)) for k in ("hy_z", "hy_y", "hz_z", "hz_y", "hz_x", "hy_x")}
        self.lo, self.hi = (gr.x1, gr.y1, gr.z1), (gr.x2, gr.y2, gr.z2)

    def _in(self, X, ax=None, d=0):
        """X on the block's inner nodes, moved by d along ax."""
        return X[tuple(slice(self.lo[x] + d * (x == ax), self.hi[x] + d * (x == ax)) for x in range(3))]

    def _face(self, ax, at):
        """The block's node range with index `at` (1-based) along ax."""
        return tuple(at - 1 if x == ax else slice(self.lo[x] - 1, self.hi[x] + 1) for x in range(3))

    def _ghosts(self, X, L):
        for ax in range(3):
            lo, hi = self.lo[ax], self.hi[ax]
            X[self._face(ax, lo)] = L[ax][self._face(ax, lo)] * X[self._face(ax, lo + 1)]
            X[self._face(ax, hi + 1)] = L[ax][self._face(ax, hi)].conj() * X[self._face(ax, hi)]

    def _euler(self, S, L, µ, cf):
        g = self._in(S)
        acc = g + cf.c * g * (self._in(self.f) * cf.ε - cf.β * g.abs() ** 2)
        for ax, k in enumerate((cf.kx, cf.ky, cf.kz)):
            acc = acc + k * (self._in(L[ax]) * self._in(S, ax, 1) - 2 * g + self._in(L[ax], ax, -1).conj() * self._in(S, ax, -1))
        for ν in range(self.st.N):
            if ν != µ:
                acc = acc + cf.cpl[ν] * self._in(self.G[ν])
        if cf.γ2 > 0:
            q = 1 + cf.γ2 * g.abs() ** 2
            d = torch.sqrt(q) * (acc - g)
            acc = g + d - cf.γ2 * g * (g.conj() * d).real / q
        return acc

    def _band(self, µ):
        st, dt = self.st, self.st.dt
        ns, rc = st.rkl[µ], st.rkc[µ] if st.rkc is not None else None
        rot = st.rotframe
        q = 1.0 if ns == 0 else rc.q if rc is not None else ns * (ns + 1) / 2
        cf = st.bcs[µ] if ns else st.bc[µ]
        L, A, B, Om, rate = self.V, self.G[µ], self.G[µ], None, None
        for j in range(1, max(ns, 1) + 1):
            g = self._in(B)
            v = self._euler(B, L, µ, cf)
            if rot and j == 1:
                a2 = g.abs() ** 2
                w = ((g.conj() * (v - g)).imag / (a2 * dt / q)).clamp(-0.5 / dt, 0.5 / dt)
                w = torch.where(a2 > 1e-3, w, torch.zeros_like(w))
                Om = torch.zeros_like(self.f)
                self._in(Om)[...] = w
                for ax in range(3):
                    Om[self._face(ax, self.lo[ax])] = Om[self._face(ax, self.lo[ax] + 1)]
                    Om[self._face(ax, self.hi[ax] + 1)] = Om[self._face(ax, self.hi[ax])]
            if rot:
                v = v - 1j * (w * dt / q) * g
            if j > 1:
                mu, nu = (rc.μ[j - 1], rc.ν[j - 1]) if rc is not None else ((2 * j - 1) / j, (1 - j) / j)
                v = mu * v + nu * self._in(A)
            if rot and j == max(ns, 1):
                v = v * torch.polar(torch.ones_like(w), w * dt)
            C_ = self.G[µ].clone()
            self._in(C_)[...] = v
            if j < ns:
                c = rc.c[j - 1] if rc is not None else j * (j + 1) / (ns * (ns + 1))
                if st.extrap:
                    if rate is None:   # (angle over the step, short) of each link; the frame adds its own turn
                        rate = [_turned(self.V[ax], self.U[ax]) for ax in range(3)]
                        if rot:
                            rate = [(r + torch.diff(Om, dim=ax) * dt, None) for ax, (r, _) in enumerate(rate)]
                    L = [self.V[ax] * _cis(r * c, (r * c).abs() <= 0.05 if rot else short)
                         for ax, (r, short) in enumerate(rate)]
                self._ghosts(C_, L)
            A, B = B, C_
        return B

    def step(self, H, HJ):
        st, gr, fc = self.st, self.gr, self.st.fc
        Nx, Ny, Nz = gr.Nx, gr.Ny, gr.Nz
        F = [self._band(µ) for µ in range(st.N)]
        cut = lambda X, ax, d=0, r=None: X[tuple(slice((0 if x == r else 1) + d * (x == ax), (Nx, Ny, Nz)[x] + d * (x == ax))
                                                 for x in range(3))]
        inc = ((1, 2, fc.sxy, fc.sxz), (2, 0, fc.syz, fc.syx), (0, 1, fc.szx, fc.szy))
        for ax in range(3):
            V = cut(self.V[ax], ax, 0, ax)
            cur = sum(st.wa[ax][µ] * (cut(G, ax, 0, ax).conj() * V * cut(G, ax, 1, ax)).imag for µ, G in enumerate(self.G))
            cut(self.J[ax], ax, 0, ax)[...] = cur
            # φ = θ + d1 τ J minus the curl of h: −s (∂ of the next component) + s (∂ of the one after)
            p, r, s1, s2 = inc[ax]
            d = lambda hc, along: cut(self.h[hc], along, 0, ax) - cut(self.h[hc], along, -1, ax)
            cut(self.ph[ax], ax, 0, ax)[...] = (cut(self.th[ax], ax, 0, ax) + fc.d1 * cut(self.tau[ax], ax, 0, ax) * cur
                                                - s1 * d(r, p) + s2 * d(p, r))
        n = (Nx - 1, Ny - 1, Nz - 1)
        sl = [tuple(slice(1, 1 + n[x] - (x == c)) for x in range(3)) for c in range(3)]
        z = _sep_solve([self.ph[c][sl[c]] - self.th[c][sl[c]] for c in range(3)], n, fc.a)
        for c in range(3):
            self.ph[c][sl[c]] = self.th[c][sl[c]] + z[c]
        for ax in range(3):
            p = cut(self.ph[ax], ax, 0, ax)
            cut(self.U[ax], ax, 0, ax)[...] = torch.polar(torch.ones_like(p), -p)
        px, py, pz = self.ph
        one, hs = (1, 1, 1), (gr.dx, gr.dy, gr.dz)
        for c, (a, b) in enumerate(((1, 2), (2, 0), (0, 1))):   # h_c = ∂_a φ_b − ∂_b φ_a on the inner plaquettes
            r = tuple(slice(one[x], (Nx, Ny, Nz)[x] - (x != c)) for x in range(3))
            mv = lambda X, ax: X[tuple(slice(r[x].start + (x == ax), r[x].stop + (x == ax)) for x in range(3))]
            pa, pb = self.ph[a], self.ph[b]
            self.h[c][r] = (mv(pb, a) - pb[r] - mv(pa, b) + pa[r]) / (hs[a] * hs[b])
        hx, hy, hz = self.h
        B = self.bar
        hx[0] = hx[-1] = 0.0
        hx[:, 0] = hx[:, -1] = 0.0
        for e, at in ((0, 0), (1, -1)):
            hy[:, :, at] = HJ * B["hy_z"][:, e]
            hz[:, :, at] = H + HJ * B["hz_z"][:, e]
        for e, at in ((0, 0), (1, -1)):
            hy[:, at, :] = HJ * B["hy_y"][e]
            hz[:, at, :] = H + HJ * B["hz_y"][e]
        for at in (0, -1):
            hy[at] = HJ * B["hy_x"]
            hz[at] = H + HJ * B["hz_x"]
        blk = tuple(slice(self.lo[x] - 1, self.hi[x] + 1) for x in range(3))
        for µ in range(st.N):
            self._ghosts(F[µ], self.U)
            self.G[µ] = self.G[µ].clone()
            self.G[µ][blk] = F[µ][blk]
        self.th, self.ph = self.ph, self.th
        self.V, self.U = self.U, self.V
