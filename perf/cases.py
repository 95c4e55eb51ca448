"""The calls this framework is used for, as timed cases.

A case is one pass of a program over the public entry points: a field goes
into a resident context, the time stepper (or the network, or the
diagnostics) works on it, and the result comes back.  Sizes follow the
repository's own configurations: the 512^3 run of bench.py and its rkf45,
ensemble, learned and spectrum workloads, the 64^3 double precision run of the
parity tests, the trapped imaginary-time run directory of the tests, and
ragged grids like those of the parity tests.

Fields are smooth random ones (Fourier modes up to a cut-off with random
amplitudes and phases, mean density 1), which carry a tangle of vortices as
the runs' states do; in a trap they are cut by the Thomas-Fermi profile.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

import gpe_b200
from gpe_b200 import GpeBatch, GpeParams, GpeSolver, run_loop
from gpe_b200._lib import pinned_empty
from gpe_b200.cnn import CoarseCorrector

H = 0.5      # grid spacing of every run but the C2-like ones
NLAYERS = 4  # of the network

DEV = "cuda"


# ------------------------------------------------------------------------------
# cases

def _steps(name, nx, ny, nz, steps, **kw):
    """A run of `steps` steps: set_state, advance, get_state_device."""
    c = dict(kind="steps", nx=nx, ny=ny, nz=nz, steps=steps, h=H, dt=0.005, scheme="rk4", eqn=4,
             bcs=1, order=4, precision=16, kahan=False, omega=0.0, urhs=0.0, diss=0.0, real=True)
    c.update(kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the headline run of the benchmark: one large periodic grid in
        # complex64 with compensated accumulation
        _steps("grid_512_f32", 512, 512, 512, 4, precision=8, kahan=True),
        # the plain fine path of the learned workload (order 2, its largest dt)
        _steps("fine_256_f32", 256, 256, 256, 16, precision=8, kahan=True, order=2, dt=0.02, h=0.25),
        # the reference's own precision on an ordinary grid
        _steps("grid_256_f64", 256, 256, 256, 6),
        # a small double precision run: launches and latency
        _steps("line_64_f64", 64, 64, 64, 50, order=2, dt=0.01),
        # adaptive Cash-Karp steps on the reflective ring-and-pulse grid
        _steps("ring_128_rk45", 128, 128, 128, 8, scheme="rk45", bcs=2, h=0.4),
        # a moving frame with a sponge at the walls (equation 1) on a ragged grid
        _steps("sponge_ragged_f64", 150, 93, 71, 10, eqn=1, bcs=2, dt=0.01, urhs=0.3, diss=0.5),
        # the reference's loop in imaginary time: one solver(), get_norm() and
        # renormalise() per step on a small trapped grid, host arrays in and out
        _steps("trap_imag_loop", 40, 40, 40, 20, kind="loop", scheme="rk2", bcs=2, order=2,
               dt=0.002, omega=0.3, real=False),
        # a parameter scan: uneven trapped grids stepped together
        dict(name="ensemble_f32", kind="ensemble", members=24, largest=128, steps=10, precision=8,
             kahan=False, order=2, pick=0),
        # the learned coarse path: a coarse step and the network's correction
        dict(name="learned_128", kind="learned", nx=128, ny=128, nz=128, steps=8),
        # its training: loss and gradients of one pair
        dict(name="train_128", kind="train", nx=128, ny=128, nz=128),
        # the diagnostics of an output time: energy, mass, momentum, spectrum,
        # condensate and vortex line length
        dict(name="observe_256_f64", kind="observe", nx=256, ny=256, nz=256, precision=16, order=4),
        # vortex points of a ragged grid for the output files
        dict(name="zeros_ragged_f32", kind="zeros", nx=120, ny=97, nz=83, precision=8, order=2),
    ]


def _size(rng, lo, hi):
    """A grid size spread over its logarithm; every other one odd or unround."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n if rng.random() < 0.5 else max(lo, min(hi, 16 * ((n + 8) // 16)))


def draw(rng):
    kind = rng.choice(["steps"] * 6 + ["loop", "ensemble", "learned", "train", "observe", "zeros"])
    precision = rng.choice([8, 16])
    kahan = precision == 8 and rng.random() < 0.6
    order = rng.choice([2, 4])
    n = [_size(rng, 16, 320) for _ in range(3)]
    if kind == "steps":
        scheme = rng.choice(["rk4", "rk4", "rk4", "rk45", "rk2", "euler"])
        # an adaptive step in complex64 depends on the last digits of its error
        # estimate, so adaptive runs are drawn in double precision
        if scheme == "rk45":
            precision, kahan, n = 16, False, [min(v, 144) for v in n]
        eqn = rng.choice([4, 4, 4, 2, 1])
        return _steps(None, *n, rng.randint(3, 8), scheme=scheme, precision=precision, kahan=kahan,
                      order=order, bcs=rng.choice([1, 2]), eqn=eqn,
                      dt=0.001 if scheme == "euler" else 0.005,
                      omega=rng.choice([0.0, 0.05]) if eqn == 4 and scheme != "rk45" else 0.0,
                      urhs=round(rng.uniform(0.1, 0.6), 3) if eqn < 3 and rng.random() < 0.5 else 0.0,
                      diss=round(rng.uniform(0.1, 1.0), 3) if eqn == 1 and rng.random() < 0.5 else 0.0)
    if kind == "loop":
        m = [_size(rng, 16, 96) for _ in range(3)]
        return _steps(None, *m, rng.randint(5, 20), kind="loop", scheme=rng.choice(["rk2", "rk4"]),
                      bcs=2, order=order, dt=0.002, omega=0.3, real=False)
    if kind == "ensemble":
        return dict(kind="ensemble", members=rng.randint(3, 24), largest=rng.choice([48, 64, 96, 128]),
                    steps=rng.randint(4, 10), precision=precision, kahan=kahan, order=order,
                    pick=rng.randint(1, 10000))
    if kind in ("learned", "train"):
        m = dict(kind=kind, nx=16 * rng.randint(2, 8), ny=_size(rng, 24, 128), nz=_size(rng, 24, 128))
        return dict(m, steps=rng.randint(3, 8)) if kind == "learned" else m
    if kind == "observe":
        return dict(kind="observe", nx=n[0], ny=n[1], nz=n[2], precision=precision, order=order)
    z = [_size(rng, 16, 128) for _ in range(3)]
    return dict(kind="zeros", nx=z[0], ny=z[1], nz=z[2], precision=precision, order=order)


# ------------------------------------------------------------------------------
# inputs

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _field(nx, ny, nz, h, kmax, seed):
    """(nz, ny, nx) complex128: random modes of |k| <= kmax, mean density 1."""
    g = _generator(seed)
    k = [2 * math.pi * torch.fft.fftfreq(n, d=h, device=DEV, dtype=torch.float64) for n in (nz, ny, nx)]
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    # at least the lowest modes of the largest box side are in
    cut = max(kmax, 2.1 * math.pi / (h * max(nx, ny, nz))) ** 2
    a = torch.randn((nz, ny, nx), generator=g, device=DEV, dtype=torch.complex128)
    a = torch.fft.ifftn(torch.where(k2 <= cut, a, torch.zeros((), device=DEV, dtype=a.dtype)))
    return a / torch.sqrt(torch.mean(a.real ** 2 + a.imag ** 2))


def _axis(n, h):
    return -(n - 1) * h / 2 + h * torch.arange(n, device=DEV, dtype=torch.float64)


def _trap(shape, h, omega):
    nz, ny, nx = shape
    x, y, z = _axis(nx, h), _axis(ny, h), _axis(nz, h)
    return 0.5 * omega ** 2 * (x[None, None, :] ** 2 + y[None, :, None] ** 2 + z[:, None, None] ** 2)


def _trapped(psi, h, omega):
    if not omega:
        return psi
    return psi * torch.sqrt(torch.clamp(1.0 - _trap(psi.shape, h, omega), min=0.0))


def _dtype(precision):
    return torch.complex128 if precision == 16 else torch.complex64


def _params(nx, ny, nz, h, **kw):
    return GpeParams(nx=nx, ny=ny, nz=nz, xr=(nx - 1) * h / 2, yr=(ny - 1) * h / 2,
                     zr=(nz - 1) * h / 2, g=1.0, mu=1.0, **kw)


def _members(case):
    """(n, omega) of every ensemble member: the sizes and traps of the scan."""
    r = np.random.default_rng(case["pick"])
    sizes = [n for n in (32, 48, 64, 96, 128) if n <= case["largest"]]
    return [(int(r.choice(sizes)), float(r.uniform(0.05, 0.15))) for _ in range(case["members"])]


def _psi(case, seed):
    """The case's input field(s), complex128 rounded to the run's precision."""
    kind = case["kind"]
    if kind == "ensemble":
        return [_trapped(_field(n, n, n, H, 0.8, seed * 1000 + r), H, om).to(_dtype(case["precision"]))
                for r, (n, om) in enumerate(_members(case))]
    n = case["nx"], case["ny"], case["nz"]
    if kind in ("learned", "train"):
        return _field(*n, H, 1.0, seed).to(torch.complex64)
    psi = _trapped(_field(*n, case.get("h", H), 1.0, seed), case.get("h", H), case.get("omega", 0.0))
    return psi.to(_dtype(case["precision"])).contiguous()


def _weights():
    z = np.load(os.path.join(os.path.dirname(gpe_b200.__file__), "data", "cnn_weights.npz"))
    return z["w"], z["b"], float(z["out_scale"])


LEARNED = dict(scheme="rk4", eqn_to_solve=4, bcs=1, order=4, precision=8, kahan=True, fd_match=0.5)
LEARNED_DT = 0.04


def _target(psi, seed):
    """A training target: the input with a small smooth change."""
    nz, ny, nx = psi.shape
    return (psi + 0.02 * _field(nx, ny, nz, H, 1.0, seed + 7919)).to(torch.complex64)


def prepare(case, seed):
    kind = case["kind"]
    psi = _psi(case, seed)
    s = {"case": case, "psi": psi}
    if kind == "ensemble":
        prms = [_params(n, n, n, H, scheme="rk4", eqn_to_solve=4, bcs=2, order=case["order"],
                        precision=case["precision"], kahan=case["kahan"], omx=om, omy=om, omz=om)
                for n, om in _members(case)]
        s["batch"] = GpeBatch(prms, 0.01)
        s["out"] = [torch.empty_like(p) for p in psi]
        return s
    if kind in ("learned", "train"):
        w, b, scale = _weights()
        prm = _params(case["nx"], case["ny"], case["nz"], H, **LEARNED)
        s["solver"] = GpeSolver(prm, dt=LEARNED_DT)
        s["net"] = CoarseCorrector(case["nx"], case["ny"], case["nz"], train=kind == "train",
                                   out_scale=scale, preserve_norm=kind == "learned")
        s["net"].set_weights(w, b)
        if kind == "learned":
            s["net"].attach(s["solver"])
            s["out"] = torch.empty_like(psi)
        else:
            s["solver"].set_state(psi)
            s["target"] = _target(psi, seed)
        return s
    if kind in ("observe", "zeros"):
        prm = _params(case["nx"], case["ny"], case["nz"], H, scheme="euler", eqn_to_solve=4, bcs=1,
                      order=case["order"], precision=case["precision"])
        s["solver"] = GpeSolver(prm, dt=0.005)
        s["solver"].set_state(psi)
        if kind == "zeros":
            # a page-locked buffer for the point list, kept from call to call
            s["points"] = pinned_empty((2 * psi.numel(), 3), np.float64)
            s["points"][:] = 0.0
        return s
    om = case["omega"]
    prm = _params(case["nx"], case["ny"], case["nz"], case["h"], scheme=case["scheme"],
                  eqn_to_solve=case["eqn"], bcs=case["bcs"], order=case["order"],
                  real_time=case["real"], precision=case["precision"], kahan=case["kahan"],
                  Urhs=case["urhs"], diss_amp=case["diss"], omx=om, omy=om, omz=om)
    s["solver"] = GpeSolver(prm, tau=case["dt"])
    s["dt"] = s["solver"].dt
    if kind == "loop":
        s["psi"] = psi.cpu().numpy()
    else:
        s["out"] = torch.empty_like(psi)
    return s


# ------------------------------------------------------------------------------
# one pass

def _real(norms, precision):
    # the norms of a complex64 state are as exact as that state: 32 bits
    return norms if precision == 16 else norms.astype(np.float32)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        b = state["batch"]
        b.set_states(state["psi"])
        norms = b.advance(case["steps"])
        for m, out in zip(b.members, state["out"]):
            m.get_state_device(out)
        return {"psi": state["out"], "norms": _real(norms, case["precision"])}
    s = state["solver"]
    if kind == "train":
        loss, dw, db = state["net"].grad(s, state["target"])
        # the network works in bfloat16 with 32-bit sums, and so is its loss
        return {"loss": np.float32(loss), "dw": dw, "db": db}
    if kind == "observe":
        e, h4 = s.energy()
        mass, mom = s.diagnostics()
        c = s.condensed_particles()
        return {"energy": e, "h4": h4, "mass": mass, "momentum": mom, "row": c.row, "eta": c.eta,
                "nharm": c.nharm, "F": c.F, "length": s.linelength()}
    if kind == "zeros":
        counts, _ = s.zeros(out=state["points"])
        # the buffer whole (zero past the points, whose number differs from field to field)
        return {"counts": counts, "points": state["points"]}
    if kind == "loop":
        s.t, s.im_t, s.p, s.dt = 0.0, 0.0, 0, state["dt"]
        s.set_state(state["psi"])
        rec = run_loop(s, case["steps"], renorm=True)
        return {"psi": s.get_state(np.complex128 if case["precision"] == 16 else np.complex64),
                "norms": np.array([r[2] for r in rec])}
    if kind == "learned":
        s.set_state(state["psi"])
        norms = s.advance(case["steps"])
        s.get_state_device(state["out"])
        return {"psi": state["out"], "norms": _real(norms, 8)}
    s.t, s.im_t, s.p, s.dt = 0.0, 0.0, 0, state["dt"]
    s.set_state(state["psi"])
    norms = s.advance(case["steps"])
    s.get_state_device(state["out"])
    return {"psi": state["out"], "norms": _real(norms, case["precision"])}


# ------------------------------------------------------------------------------
# work: what a pass cannot do without

def _sites(case):
    return case["nx"] * case["ny"] * case["nz"]


def _rhs_flops(order):
    """Real operations of one right-hand side at one site: the Laplacian's 3
    axes (2 or 4 neighbours each) and the nonlinear term, on both parts."""
    return 2 * (3 * (3 if order == 2 else 6) + 2) + 12


STAGES = {"euler": 1, "rk2": 2, "rk4": 4, "rk45": 6}


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        n = sum(m ** 3 for m, _ in _members(case))
        per = 4 * (_rhs_flops(case["order"]) + 4)
        # in, every step reads and writes psi (and its compensation), out
        b = case["precision"] * n * (2 + case["steps"] * (4 if case["kahan"] else 2) + 2)
        return {"bytes": b, "flops": n * case["steps"] * per}
    n = _sites(case)
    if kind in ("steps", "loop"):
        st = STAGES[case["scheme"]]
        b = case["precision"] * n * (2 + case["steps"] * (4 if case["kahan"] else 2) + 2)
        return {"bytes": b, "flops": n * case["steps"] * st * (_rhs_flops(case["order"]) + 8)}
    net = 2 * 27 * (2 * 16 + 16 * 16 + 16 * 16 + 16 * 2)
    if kind == "learned":
        return {"bytes": 8 * n * (4 + case["steps"] * 6),
                "flops": n * case["steps"] * (net + 4 * (_rhs_flops(4) + 8))}
    if kind == "train":
        # forward, weight gradients, and input gradients of layers 1..3
        back = 2 * 27 * (16 * 16 + 16 * 16 + 16 * 2)
        return {"bytes": 8 * n * 2, "flops": n * (2 * net + back)}
    es = case["precision"]
    if kind == "observe":
        # each of the four diagnostics reads the field, the transform writes it
        return {"bytes": es * n * 6, "flops": n * (5 * math.log2(n) + _rhs_flops(case["order"]) + 80)}
    return {"bytes": es * n + 24 * n // 2, "flops": n * 60}


# ------------------------------------------------------------------------------
# 64-bit values in plain torch

def _gather(n, bcs, s):
    i = torch.arange(n, device=DEV) + s
    if bcs == 1:
        return i % n
    i = i.abs()
    return torch.where(i > n - 1, 2 * (n - 1) - i, i)


def _shift(u, axis, s, bcs):
    return u.index_select(axis, _gather(u.shape[axis], bcs, s))


def _laplacian(u, h, order, bcs, match=0.0):
    if order == 2:
        c1, c2 = 1.0 / h ** 2, 0.0
    elif match:
        c1, c2 = (4.0 - match ** 2) / (3.0 * h ** 2), (match ** 2 - 1.0) / (12.0 * h ** 2)
    else:
        c1, c2 = 16.0 / (12.0 * h ** 2), -1.0 / (12.0 * h ** 2)
    lap = -6.0 * (c1 + c2) * u
    for axis in range(3):
        lap += c1 * (_shift(u, axis, 1, bcs) + _shift(u, axis, -1, bcs))
        if c2:
            lap += c2 * (_shift(u, axis, 2, bcs) + _shift(u, axis, -2, bcs))
    return lap


def _rhs(case, h, match=0.0):
    """f(u) of the case's equation with g = mu = 1."""
    eqn, bcs, order = case.get("eqn", 4), case["bcs"], case["order"]
    shape = case["nz"], case["ny"], case["nx"]
    om, U, amp = case.get("omega", 0.0), case.get("urhs", 0.0), case.get("diss", 0.0)
    V = _trap(shape, h, om) if om else 0.0
    sponge = 0.0
    if eqn == 1 and amp:
        for axis, n in ((2, shape[2]), (1, shape[1]), (0, shape[0])):
            x = _axis(n, h)
            edge = float(x[0]) + (n - 3) * h
            view = [1, 1, 1]
            view[axis] = n
            sponge = sponge + (amp * (1.0 + torch.tanh(x - edge) * torch.tanh(x + edge))).view(view)

    def f(u):
        lap = _laplacian(u, h, order, bcs, match)
        d2 = u.real ** 2 + u.imag ** 2
        if eqn == 4:
            return 1j * (0.5 * lap + (1.0 - V - d2) * u)
        if eqn == 2:
            r = 1j * (lap - d2 * u)
        else:
            r = (0.5j + 0.5 * sponge) * (lap + (1.0 - d2) * u)
        if U:
            gx = _shift(u, 2, 1, bcs) - _shift(u, 2, -1, bcs)
            if order == 2:
                gx = gx / (2.0 * h)
            else:
                gx = (8.0 * gx - (_shift(u, 2, 2, bcs) - _shift(u, 2, -2, bcs))) / (12.0 * h)
            r = r + U * gx
        return r

    return f


def _weights_1d(n):
    w = torch.ones(n, device=DEV, dtype=torch.float64)
    ends = (3.0 / 8.0, 7.0 / 6.0, 23.0 / 24.0)
    for q in range(3):
        w[q] = ends[q]
        w[n - 1 - q] = ends[q]
    return w


def _norm(u, h):
    nz, ny, nx = u.shape
    d2 = u.real ** 2 + u.imag ** 2
    d2 = torch.tensordot(d2, _weights_1d(nx), dims=([2], [0]))
    d2 = torch.tensordot(d2, _weights_1d(ny), dims=([1], [0]))
    return float(torch.dot(d2, _weights_1d(nz))) * h ** 3


def _step(scheme, f, u, dt):
    if scheme == "euler":
        return u + dt * f(u)
    if scheme == "rk2":
        return u + dt * f(u + 0.5 * dt * f(u))
    k1 = f(u)
    k2 = f(u + 0.5 * dt * k1)
    k3 = f(u + 0.5 * dt * k2)
    k4 = f(u + dt * k3)
    return u + (dt / 6.0) * (k1 + 2.0 * k2 + 2.0 * k3 + k4)


CK = ((0.2,), (0.075, 0.225), (0.3, -0.9, 1.2), (-11 / 54, 2.5, -70 / 27, 35 / 27),
      (1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096))
CK_C = (37 / 378, 0.0, 250 / 621, 125 / 594, 0.0, 512 / 1771)
CK_D = (2825 / 27648, 0.0, 18575 / 48384, 13525 / 55296, 277 / 14336, 0.25)


def _adaptive_step(f, u, dt):
    """One accepted Cash-Karp step in real time; (new u, next dt)."""
    k1 = f(u)
    dt0 = dt
    while True:
        k = [dt * k1]
        for row in CK:
            k.append(dt * f(u + sum(b * kk for b, kk in zip(row, k))))
        err = sum((c - d) * kk for c, d, kk in zip(CK_C, CK_D, k) if c != d)
        scal = u.abs() + dt0 * k1.abs() + 1e-30
        errmax = float((err.abs() / scal).max()) / 1e-6
        if errmax <= 1.0:
            grow = 0.9 * errmax ** -0.2 if errmax > (5.0 / 0.9) ** -5.0 else 5.0
            return u + sum(c * kk for c, kk in zip(CK_C, k) if c), dt * grow
        dt = max(0.9 * dt * errmax ** -0.25, 0.1 * dt)


def _exact_steps(case, psi):
    u = psi.to(torch.complex128)
    h = case["h"]
    f = _rhs(case, h)
    norms = []
    dt = case["dt"]
    if case["kind"] == "loop":
        # imaginary time: dt = -i tau, psi renormalised to one after every step
        u = u / math.sqrt(_norm(u, h))
        for _ in range(case["steps"]):
            u = _step(case["scheme"], f, u, -1j * dt)
            norms.append(_norm(u, h))
            u = u / math.sqrt(norms[-1])
        return {"psi": u, "norms": np.array(norms)}
    for _ in range(case["steps"]):
        if case["scheme"] == "rk45":
            u, dt = _adaptive_step(f, u, dt)
        else:
            u = _step(case["scheme"], f, u, dt)
        norms.append(_norm(u, h))
    return {"psi": u, "norms": np.array(norms)}


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _net(u, w, b):
    """The network's 2-channel output: 27 shifted products per layer."""
    a = torch.stack([u.real, u.imag])
    for layer in range(NLAYERS):
        n_in, n_out = (2 if layer == 0 else 16), (2 if layer == NLAYERS - 1 else 16)
        out = b[layer][:n_out].view(n_out, 1, 1, 1)
        for t in range(27):
            d = 1 - t // 9, 1 - (t // 3) % 3, 1 - t % 3
            s = torch.roll(a, shifts=d, dims=(1, 2, 3))
            out = out + (w[layer, t, :n_out, :n_in] @ s.reshape(n_in, -1)).view(n_out, *u.shape)
        a = _gelu(out) if layer < NLAYERS - 1 else out
    return a


def _exact_learned(case, psi):
    w, b, scale = _weights()
    w = torch.from_numpy(w).to(DEV, torch.float64)
    b = torch.from_numpy(b).to(DEV, torch.float64)
    u = psi.to(torch.complex128)
    f = _rhs(dict(case, bcs=1, order=4), H, match=LEARNED["fd_match"])
    norms = []
    for _ in range(case["steps"]):
        u = _step("rk4", f, u, LEARNED_DT)
        norms.append(_norm(u, H))
        d = scale * _net(u, w, b)
        u = u + torch.complex(d[0], d[1])
        u = u * math.sqrt(norms[-1] / _norm(u, H))
    return {"psi": u, "norms": np.array(norms)}


def _exact_train(case, psi, target):
    w, b, scale = _weights()
    w = torch.from_numpy(w).to(DEV, torch.float64).requires_grad_()
    b = torch.from_numpy(b).to(DEV, torch.float64).requires_grad_()
    u, t = psi.to(torch.complex128), target.to(torch.complex128)
    d = scale * _net(u, w, b)
    e = torch.complex(d[0], d[1]) + u - t
    loss = torch.mean(e.real ** 2 + e.imag ** 2)
    loss.backward()
    return {"loss": float(loss.detach()), "dw": w.grad, "db": b.grad}


def _k2(n):
    i = torch.arange(n, device=DEV)
    return torch.where(i <= (n - 1) // 2 + 1, i, n - i) ** 2


def _exact_observe(case, psi):
    u = psi.to(torch.complex128)
    nz, ny, nx = u.shape
    V = float(u.numel())
    d2 = u.real ** 2 + u.imag ** 2
    lap = _laplacian(u, H, case["order"], 1)
    kin = -(lap.real * u.real + lap.imag * u.imag)
    cell = H ** 3
    out = {"energy": float((kin + 0.5 * d2 ** 2).sum()) * cell,
           "h4": float((0.5 * kin + 0.5 * d2 ** 2 - d2).sum()) * cell,
           "mass": float(d2.sum()) * cell}
    mom = []
    for axis in (2, 1, 0):
        d = _shift(u, axis, 1, 1) - _shift(u, axis, -1, 1)
        if case["order"] == 2:
            d = d / (2.0 * H)
        else:
            d = (8.0 * d - (_shift(u, axis, 2, 1) - _shift(u, axis, -2, 1))) / (12.0 * H)
        p = -(u.real - 1.0) * d.imag - u.imag * d.real
        p = torch.tensordot(p, _weights_1d(nx), dims=([2], [0]))
        p = torch.tensordot(p, _weights_1d(ny), dims=([1], [0]))
        mom.append(float(torch.dot(p, _weights_1d(nz))) * cell)
    out["momentum"] = np.array(mom)
    a = torch.fft.ifftn(u) * math.sqrt(V)
    p = a.real ** 2 + a.imag ** 2
    n0, M = float(p[0, 0, 0]), out["mass"]
    rho0 = n0 / V
    dk = 2.0 * math.pi / (nx - 1)

    def term(n):
        k = -math.pi + dk * torch.arange(n, device=DEV, dtype=torch.float64)
        return (-2.0 * torch.cos(2.0 * k * H) + 32.0 * torch.cos(k * H) - 30.0) / H ** 2

    q = -((term(nx)[None, None, :] + term(ny)[None, :, None]) + term(nz)[:, None, None]) / 12.0
    q = q[q != 0.0]
    tot = float(((q + rho0) / (q * q + 2.0 * rho0 * q)).sum())
    temp = (M - n0) / tot
    energy0 = (M ** 2 + (M - n0) ** 2) / (2.0 * V)
    box = float((nx - 1) * (ny - 1) * (nz - 1)) * cell
    out["row"] = {"M_density": M / box, "n0_over_V": n0 / V, "M": M, "n0": n0, "temp": temp,
                  "temp2": (M / box - n0 / V) / tot, "H_over_V": (energy0 + temp * (V - 1.0)) / V}
    k2 = (_k2(nz)[:, None, None] + _k2(ny)[None, :, None] + _k2(nx)[None, None, :]).reshape(-1)
    p = p.reshape(-1)
    p, k2 = p[k2 > 0], k2[k2 > 0]
    kmag = torch.sqrt(k2.to(torch.float64))
    nf = nx // 2
    F = torch.zeros(int(kmag.max()) + 2 + nf, device=DEV, dtype=torch.float64)
    F.index_add_(0, torch.ceil(kmag).to(torch.int64), p)
    out["F"] = torch.cumsum(F, 0)[1:nf + 1]
    shell = torch.floor(torch.abs(torch.log(0.5 * kmag / math.pi) / math.log(2.0))).to(torch.int64)
    eta = []
    for m in range(7):
        of = p[shell == m]
        eta.append(float(of.mean()) if of.numel() else 0.0)
    out["eta"] = np.array(eta)
    out["nharm"] = None
    # the length is a walk over cells in order with a carried point, not a formula
    out["length"] = None
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "zeros":
        # a list of points found cell by cell: the lists are compared entry by entry
        return None
    psi = _psi(case, seed)
    if kind == "ensemble":
        got = []
        for p, (n, om) in zip(psi, _members(case)):
            c = dict(kind="steps", nx=n, ny=n, nz=n, h=H, dt=0.01, steps=case["steps"], scheme="rk4",
                     bcs=2, order=case["order"], omega=om)
            got.append(_exact_steps(c, p))
        return {"psi": [g["psi"] for g in got], "norms": np.array([g["norms"] for g in got])}
    if kind == "learned":
        return _exact_learned(case, psi)
    if kind == "train":
        return _exact_train(case, psi, _target(psi, seed))
    if kind == "observe":
        return _exact_observe(case, psi)
    return _exact_steps(case, psi)
