"""The work a user of this package has it do, as cases of one pass each: operator
calls, time steps of the solver's configurations, and training of the learned
closure, from the smallest calls (where launches count) to the largest blocks
one step of which takes tens of milliseconds.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs on the GPU, operators / solver / closure
    run(state)           one pass through the public entry points
    exact(case, seed)    what run returns on a fresh state, in 64 bits, by plain torch
    work(case)           bytes and operations one pass cannot do without
    tolerance(case)      how far two correct implementations may differ

Families (case["family"]):
  deriv    a compact first derivative of `fields` fields along `dirs`
  filter   a compact filter of `fields` fields along `dirs`, one after the other
  box      one time step of a periodic box (decaying isotropic turbulence)
  channel  one time step between two isothermal walls, stretched mesh
  ogrid    one time step around a cylinder (O-grid, wall, sponge, DSM)
  mlp      the learned closure alone: an Adam step, or inference in BF16
"""
from __future__ import annotations

import math

import numpy as np
import torch

import mpi_3dcompact_b200 as m

GAMMA, PR = 1.4, 0.7
R_GAS = 1.0 / GAMMA
CP = R_GAS * GAMMA / (GAMMA - 1.0)
LIBRARY = {"FP64": m.FP64, "FP32": m.FP32BULK}
DTYPE = {"FP64": torch.float64, "FP32": torch.float32}
WALL = "CONST_T_WALL"
WEIGHTS = "mpi_3dcompact_b200/data/mlp_sgs_hit128.bin"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one field of a 64^3 block, one direction, as a program
        # that replaces one calc1stDerivField call does it
        {"name": "pade6_64_fp64", "family": "deriv", "op": "PADE6", "nx": 64, "ny": 64, "nz": 64, "walls": False,
         "precision": "FP64", "fields": 1, "dirs": "y"},
        # the velocity and temperature gradients of the headline block
        {"name": "penta10_256_fp32", "family": "deriv", "op": "PENTA10", "nx": 256, "ny": 256, "nz": 256,
         "walls": False, "precision": "FP32", "fields": 4, "dirs": "xyz"},
        # ragged lines, one of them between walls (Dirichlet closures), in FP64
        {"name": "pade6_ragged_fp64", "family": "deriv", "op": "PADE6", "nx": 150, "ny": 97, "nz": 75, "walls": True,
         "precision": "FP64", "fields": 4, "dirs": "xyz"},
        # the conserved-state filter of the O-grid (512-point theta lines, wall to far field, 64-point span)
        {"name": "compact10_ogrid_fp32", "family": "filter", "op": "COMPACT10", "alphaF": 0.49, "nx": 512, "ny": 256,
         "nz": 64, "walls": True, "precision": "FP32", "fields": 5, "dirs": "yzx"},
        # small DNS box, FP64 throughout: latency and launches
        {"name": "hit64_fp64", "family": "box", "nx": 64, "ny": 64, "nz": 64, "fd": "PADE6", "filter": "COMPACT10",
         "alphaF": 0.49, "rk": "RK4", "les": "NOMODEL", "precision": "FP64", "storage": "FULL"},
        # the headline configuration: 256^3, FP32 work fields over an FP64 state
        {"name": "hit256_fp32", "family": "box", "nx": 256, "ny": 256, "nz": 256, "fd": "PENTA10",
         "filter": "COMPACT8", "alphaF": 0.45, "rk": "LSLDDRK4", "les": "VREMAN", "precision": "FP32",
         "storage": "FULL"},
        # the same block in FP64, which the headline number is compared with
        {"name": "hit256_fp64", "family": "box", "nx": 256, "ny": 256, "nz": 256, "fd": "PENTA10",
         "filter": "COMPACT8", "alphaF": 0.45, "rk": "LSLDDRK4", "les": "VREMAN", "precision": "FP64",
         "storage": "FULL"},
        # LES with the learned closure (tensor-core inference in every stage)
        {"name": "les128_mlp_fp32", "family": "box", "nx": 128, "ny": 128, "nz": 128, "fd": "PADE6",
         "filter": "COMPACT10", "alphaF": 0.49, "rk": "RK4", "les": "MLP", "precision": "FP32", "storage": "FULL"},
        # the lean dataflow of blocks that fill the HBM, with their 1024-point lines on fewer planes
        {"name": "lean1024_mlp_fp32", "family": "box", "nx": 1024, "ny": 512, "nz": 32, "fd": "PENTA10",
         "filter": "COMPACT8", "alphaF": 0.45, "rk": "LSLDDRK4", "les": "MLP", "precision": "FP32",
         "storage": "LEAN"},
        # wall-bounded flow on a stretched mesh (per-point metrics), no line a multiple of 32
        {"name": "channel_ragged_fp64", "family": "channel", "nx": 100, "ny": 97, "nz": 60, "rk": "TVDRK3",
         "les": "NOMODEL", "precision": "FP64"},
        # the O-grid cylinder with the dynamic Smagorinsky model
        {"name": "ogrid_dsm_fp32", "family": "ogrid", "nx": 512, "ny": 256, "nz": 64, "precision": "FP32"},
        # one optimiser step of the closure's training, at the batch its training script uses
        {"name": "mlp_train_64k", "family": "mlp", "op": "train", "batch": 65536},
    ]


def _log(rng, lo, hi):
    """A size between lo and hi, even over its logarithm; two in three as they fall, the rest multiples of 16."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n if rng.random() < 2 / 3 else max(lo, n // 16 * 16)


def draw(rng):
    family = rng.choice(("deriv", "deriv", "filter", "box", "box", "box", "channel", "ogrid", "mlp"))
    precision = rng.choice(("FP64", "FP32"))
    if family in ("deriv", "filter"):
        case = {"family": family, "nx": _log(rng, 24, 512), "ny": _log(rng, 24, 256), "nz": _log(rng, 24, 256),
                "walls": rng.random() < 0.5, "precision": precision, "fields": rng.randint(1, 5),
                "dirs": rng.choice(("x", "y", "z", "xyz", "yzx"))}
        if family == "deriv":
            case["op"] = rng.choice(("PADE6", "PENTA10"))
        else:
            case["op"] = rng.choice(("COMPACT8", "COMPACT10"))
            case["alphaF"] = rng.choice((0.45, 0.49))
        return case
    if family == "box":
        lean = rng.random() < 0.2
        les = rng.choice(("NOMODEL", "VREMAN", "MLP") if lean else ("NOMODEL", "VREMAN", "MLP", "DSM"))
        top = 128 if les == "DSM" else 200
        return {"family": "box", "nx": _log(rng, 400, 1024) if lean else _log(rng, 32, top), "ny": _log(rng, 32, top),
                "nz": _log(rng, 32, 96 if lean else top), "fd": rng.choice(("PADE6", "PENTA10")),
                "filter": rng.choice(("COMPACT8", "COMPACT10")), "alphaF": rng.choice((0.45, 0.49)),
                "rk": rng.choice(("RK4", "TVDRK3", "KENRK4", "LSLDDRK4")), "les": les, "precision": precision,
                "storage": "LEAN" if lean else "FULL"}
    if family == "channel":
        return {"family": "channel", "nx": _log(rng, 32, 160), "ny": _log(rng, 48, 160), "nz": _log(rng, 32, 128),
                "rk": rng.choice(("TVDRK3", "RK4")), "les": rng.choice(("NOMODEL", "VREMAN")),
                "precision": precision}
    if family == "ogrid":
        return {"family": "ogrid", "nx": _log(rng, 128, 512), "ny": _log(rng, 96, 256), "nz": _log(rng, 24, 64),
                "precision": precision}
    return {"family": "mlp", "op": rng.choice(("train", "infer")), "batch": _log(rng, 1000, 400000)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _noise(shape, g):
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)


def _turbulence(shape, g, k0=4.0, mt=0.3):
    """A solenoidal random velocity with the energy spectrum k^4 exp(-2 (k/k0)^2) on a 2 pi box, rms |u| = mt."""
    k = [torch.fft.fftfreq(n, d=1.0 / n, dtype=torch.float64, device="cuda") for n in shape]
    kz, ky, kx = torch.meshgrid(*k, indexing="ij")
    k2 = kx * kx + ky * ky + kz * kz
    amp = torch.sqrt(k2) * torch.exp(-k2 / k0 ** 2)
    uh = [torch.fft.fftn(_noise(shape, g)) * amp for _ in range(3)]
    div = (kx * uh[0] + ky * uh[1] + kz * uh[2]) / torch.where(k2 > 0, k2, 1.0)
    u = [torch.fft.ifftn(c - kk * div).real.contiguous() for c, kk in zip(uh, (kx, ky, kz))]
    rms = torch.sqrt(sum((c * c).mean() for c in u))
    return [c * (mt / rms) for c in u]


def _fields(case, seed):
    """Input fields of an operator: a smooth random field plus a little noise, in the operator's precision."""
    g = _gen(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    ax = [2 * math.pi * torch.arange(n, dtype=torch.float64, device="cuda") / n for n in shape]
    out = []
    for _ in range(case["fields"]):
        k = torch.randint(1, 5, (3,), device="cuda", generator=g)
        p = 6.0 * torch.rand(4, dtype=torch.float64, device="cuda", generator=g)
        f = (torch.sin(k[0] * ax[0] + p[0])[:, None, None] * torch.sin(k[1] * ax[1] + p[1])[None, :, None]
             * torch.sin(k[2] * ax[2] + p[2])[None, None, :] + 1.0 + 0.1 * p[3])
        out.append((f + 0.01 * _noise(shape, g)).to(DTYPE[case["precision"]]))
    return out


def _bcs(case):
    """1 where the direction ends at walls (Dirichlet closures): y, with "walls"."""
    return (0, 1 if case.get("walls") or case["family"] in ("channel", "ogrid") else 0, 0)


def _channel_metrics(case):
    """J, J11 .. J33 of a 4 x 2 x 2 channel clustered toward the walls by a hyperbolic tangent."""
    shape = (case["nz"], case["ny"], case["nx"])
    eta = np.arange(case["ny"]) / (case["ny"] - 1.0)
    dy = 3.2 / np.cosh(1.6 * (2 * eta - 1)) ** 2 / math.tanh(1.6)
    inv = [np.full(shape, 0.25), np.broadcast_to((1.0 / dy)[:, None], shape), np.full(shape, 0.5)]
    zero = np.zeros(shape)
    return [inv[0] * inv[1] * inv[2]] + [inv[i] if i == j else zero for i in range(3) for j in range(3)]


def _ogrid_mesh(case):
    """theta (clockwise, so that J > 0), r from 0.5 to 30 in geometric steps, a span of 2."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    th = 2 * math.pi * np.arange(nx) / nx
    r = 0.5 * 60.0 ** (np.arange(ny) / (ny - 1.0))
    shape = (nz, ny, nx)
    x = np.ascontiguousarray(np.broadcast_to(r[:, None] * np.cos(th), shape))
    y = np.ascontiguousarray(np.broadcast_to(-r[:, None] * np.sin(th), shape))
    z = np.ascontiguousarray(np.broadcast_to((2.0 * np.arange(nz) / nz)[:, None, None], shape))
    return x, y, z


def _initial(case, seed):
    """(rho, U, V, W, p) of the flow's initial state, FP64 on the GPU."""
    g = _gen(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    one = torch.ones(shape, dtype=torch.float64, device="cuda")
    if case["family"] == "ogrid":   # uniform flow at Mach 0.2, 1 % perturbed
        return [one, 0.2 * (1 + 0.01 * _noise(shape, g)), 0.002 * _noise(shape, g), 0.002 * _noise(shape, g),
                one / GAMMA]
    u = _turbulence(shape, g, mt=0.3 if case["family"] == "box" else 0.05)
    if case["family"] == "channel":   # a parabolic profile with disturbances that vanish at the walls
        eta = torch.arange(case["ny"], dtype=torch.float64, device="cuda") / (case["ny"] - 1.0)
        y = torch.tanh(1.6 * (2 * eta - 1)) / math.tanh(1.6)
        w = (1 - y * y)[None, :, None]
        u = [w * c for c in u]
        u[0] = u[0] + 0.3 * w
    return [one, *u, one / GAMMA]


def _mu(case):
    return {"box": 2.5e-4 if case.get("les") in ("MLP", "DSM") else 1e-3, "channel": 1e-3, "ogrid": 0.2 / 3900.0}[
        case["family"]]


SPONGE = {"kind": "CYLINDRICAL", "strength": 1.0, "orient": 2, "cyl_axis": [0.0, 0.0, 0.0], "rmin": 24.0}


def _options(case):
    grid, precision = (case["nx"], case["ny"], case["nz"]), LIBRARY[case["precision"]]
    if case["family"] == "box":
        return m.Options(grid=grid, fd=case["fd"], filter=case["filter"], alphaF=case["alphaF"], mu_ref=_mu(case),
                         rk=case["rk"], cfl=0.5, les=case["les"], les_avg="GLOBAL" if case["les"] in ("DSM", "MLP")
                         and case["storage"] == "FULL" else "NONE", precision=precision, storage=case["storage"],
                         mlp_fallback_frac=1.0)
    bc = (m.PERIODIC_SOLVE, m.DIRICHLET_SOLVE, m.PERIODIC_SOLVE)
    if case["family"] == "channel":
        return m.Options(grid=grid, fd="PADE6", filter="COMPACT10", alphaF=0.49, mu_ref=_mu(case), rk=case["rk"],
                         cfl=0.5, les=case["les"], precision=precision, bc=bc,
                         bc_kind=("PERIODIC", "PERIODIC", WALL, WALL, "PERIODIC", "PERIODIC"))
    return m.Options(grid=grid, fd="PADE6", filter="COMPACT10", alphaF=0.49, mu_ref=_mu(case), rk="KENRK4", cfl=0.5,
                     les="DSM", les_avg="GLOBAL", dsm_test_filter=1, precision=precision, bc=bc,
                     bc_kind=("INTERNALLY_PERIODIC", "INTERNALLY_PERIODIC", "ADIABATIC_WALL", "SPONGE", "PERIODIC",
                              "PERIODIC"), sponge=SPONGE, periodic_disp=((0, 0, 0), (0, 0, 0), (0, 0, 2.0)))


def _mlp_inputs(case, seed):
    """Parameters (Xavier-uniform), normalisation, a batch of raw features and of normalised targets."""
    r = np.random.default_rng(1000 + int(seed))
    p = np.zeros(9090, dtype=np.float32)
    at = 0
    for nin, nout in ((9, 64), (64, 64), (64, 64), (64, 2)):
        a = math.sqrt(6.0 / (nin + nout))
        p[at:at + nin * nout] = r.uniform(-a, a, nin * nout)
        p[at + nin * nout:at + nin * nout + nout] = r.uniform(-0.1, 0.1, nout)
        at += nin * nout + nout
    mean, std = r.uniform(-1, 1, 9).astype(np.float32), r.uniform(0.5, 2, 9).astype(np.float32)
    g = _gen(seed)
    n = case["batch"]
    z = torch.randn((n, 9), device="cuda", generator=g)
    x = z * torch.tensor(std, device="cuda") + torch.tensor(mean, device="cuda")
    y = torch.stack((torch.tanh(z[:, 0] * z[:, 1]), z[:, 2]), dim=1) + 0.1 * torch.randn((n, 2), device="cuda",
                                                                                          generator=g)
    return p, mean, std, x.contiguous(), y.contiguous()


class _View:
    """A device array of the solver's as torch takes it; keeps the solver, whose memory it is."""

    def __init__(self, solver, ptr, shape):
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "data": (int(ptr), False),
                                         "version": 2}


def prepare(case, seed):
    if case["family"] in ("deriv", "filter"):
        f = _fields(case, seed)
        shape, bcs, ops = tuple(f[0].shape), _bcs(case), []
        for d in case["dirs"]:
            d = "xyz".index(d)
            if case["family"] == "deriv":
                cls = {"PADE6": m.Pade6, "PENTA10": m.Penta10}[case["op"]]
                ops.append(cls(shape, bcs[d], d, precision=LIBRARY[case["precision"]]))
            else:
                cls = {"COMPACT8": m.Compact8Filter, "COMPACT10": m.Compact10Filter}[case["op"]]
                ops.append(cls(case["alphaF"], shape, bcs, d, precision=LIBRARY[case["precision"]]))
        outs = [[torch.empty_like(a) for a in f] for _ in ops]
        return {"family": case["family"], "f": f, "ops": ops, "outs": outs}
    if case["family"] == "mlp":
        p, mean, std, x, y = _mlp_inputs(case, seed)
        net = m.MLPClosure(seed=0)
        inf = np.full(9, np.inf, dtype=np.float32)
        net.set_normalization(mean, std, -inf, inf, np.zeros(2, np.float32), np.ones(2, np.float32))
        net.set_params(p)
        return {"family": "mlp", "op": case["op"], "net": net, "x": x, "y": y, "out": torch.empty_like(y)}
    s = m.CurvilinearCSolver(_options(case))
    if case["family"] == "box":
        s.set_box_metrics(2 * math.pi)
    elif case["family"] == "channel":
        s.set_metrics(_channel_metrics(case))
    else:
        x, y, z = _ogrid_mesh(case)
        s.set_mesh(x, y, z)
        s.set_sponge(m.sponge_sigma(s.opt, x, y, z))
    s.set_initial_conditions(*[a.cpu().numpy() for a in _initial(case, seed)])
    if case.get("les") == "MLP":
        net = m.MLPClosure(seed=0)
        net.load(WEIGHTS)
        s.set_mlp(net)
    return {"family": "step", "solver": s}


def run(state):
    family = state["family"]
    if family == "deriv":
        for op, out in zip(state["ops"], state["outs"]):
            if len(out) == 1:
                op.calc1stDerivField(state["f"][0], out[0])
            else:
                op.calc1stDerivFields(state["f"], out)
        return state["outs"]
    if family == "filter":
        src = state["f"]
        for op, out in zip(state["ops"], state["outs"]):
            op.filterFields(src, out)
            src = out
        return src
    if family == "mlp":
        net = state["net"]
        if state["op"] == "train":
            loss = net.train_step(state["x"], state["y"], 1e-3)
            return {"loss": loss, "params": net.params()}
        net.infer_bf16(state["x"], state["out"])
        return state["out"]
    s = state["solver"]
    s.step(1)
    return [torch.as_tensor(_View(s, p, s.shape), device="cuda") for p in s.conserved_device_ptrs()]


# ---------------------------------------------------------------------------
# the same in 64 bits by plain torch: every line operator as a dense matrix
# A^-1 B of its left- and right-hand sides
# ---------------------------------------------------------------------------
def _banded(n, lhs, rhs, periodic, wrap_only=0):
    """Dense A (lhs) and B (rhs) of interior stencils {offset: value}; wrap_only = +1 / -1 keeps the entries of B
    that wrap past the end / the start only."""
    a, b = np.zeros((n, n)), np.zeros((n, n))
    for mat, st, only in ((a, lhs, 0), (b, rhs, wrap_only)):
        for i in range(n):
            for k, v in st.items():
                j = i + k
                side = 1 if j >= n else -1 if j < 0 else 0
                if side != 0 and not periodic or only and side != only:
                    continue
                mat[i, j % n] += v
    return a, b


def _rows(a, b, rows):
    """Boundary rows {i: (lhs {offset: value}, rhs list from node 0)} and their mirror images (`sign` for derivatives)."""
    n = a.shape[0]
    for i, (lhs, rhs, sign) in rows.items():
        for r, flip in ((i, False), (n - 1 - i, True)):
            a[r], b[r] = 0.0, 0.0
            for k, v in lhs.items():
                a[r, r - k if flip else r + k] += v
            for j, v in enumerate(rhs):
                b[r, n - 1 - j if flip else j] += sign * v if flip else v


def _deriv_parts(op, n, wall):
    if op == "PADE6":
        lhs, c = {-1: 1 / 3, 0: 1.0, 1: 1 / 3}, {1: 14 / 18, 2: 1 / 36}
        rows = {0: ({0: 1.0, 1: 2.0}, [-5 / 2, 2.0, 1 / 2], -1),
                1: ({-1: 1 / 6, 0: 1.0, 1: 1 / 2}, [-5 / 9, -1 / 2, 1.0, 1 / 18], -1)}
    else:
        lhs = {-2: 1 / 20, -1: 1 / 2, 0: 1.0, 1: 1 / 2, 2: 1 / 20}
        c = {1: 17 / 24, 2: 101 / 600, 3: 1 / 600}
        rows = {0: ({0: 1.0, 1: 5.0}, [-197 / 60, -5 / 12, 5.0, -5 / 3, 5 / 12, -1 / 20], -1),
                1: ({-1: 1 / 12, 0: 1.0, 1: 5 / 4}, [-79 / 240, -77 / 60, 55 / 48, 5 / 9, -5 / 48, 1 / 60, -1 / 720], -1),
                2: ({-2: 1 / 36, -1: 4 / 9, 0: 1.0, 1: 4 / 9, 2: 1 / 36},
                    [-25 / 216, -20 / 27, 0.0, 20 / 27, 25 / 216], -1)}
    rhs = {s * k: s * v for k, v in c.items() for s in (1, -1)}
    return lhs, rhs, rows if wall else {}


def _deriv_matrix(op, n, wall):
    lhs, rhs, rows = _deriv_parts(op, n, wall)
    a, b = _banded(n, lhs, rhs, not wall)
    _rows(a, b, rows)
    return np.linalg.solve(a, b) * ((n - 1.0) if wall else n)


def _filter_matrix(op, af, n, wall):
    if op == "COMPACT10":
        c = [(193 + 126 * af) / 256, (105 + 302 * af) / 256, (-15 + 30 * af) / 64, (45 - 90 * af) / 512,
             (-5 + 10 * af) / 256, (1 - 2 * af) / 512]
        t = [[1 + 1022 * af, 1014 + 20 * af, 45 + 934 * af, -120 + 240 * af, 210 - 420 * af, -252 + 504 * af,
              210 - 420 * af, -120 + 240 * af, 45 - 90 * af, -10 + 20 * af, 1 - 2 * af],
             [-1 + 2 * af, 10 + 1004 * af, 979 + 90 * af, 120 + 784 * af, -210 + 420 * af, 252 - 504 * af,
              -210 + 420 * af, 120 - 240 * af, -45 + 90 * af, 10 - 20 * af, -1 + 2 * af],
             [1 - 2 * af, -10 + 20 * af, 45 + 934 * af, 904 + 240 * af, 210 + 604 * af, -252 + 504 * af,
              210 - 420 * af, -120 + 240 * af, 45 - 90 * af, -10 + 20 * af, 1 - 2 * af],
             [-1 + 2 * af, 10 - 20 * af, -45 + 90 * af, 120 + 784 * af, 814 + 420 * af, 252 + 520 * af,
              -210 + 420 * af, 120 - 240 * af, -45 + 90 * af, 10 - 20 * af, -1 + 2 * af]]
        t = [[v / 1024 for v in r] for r in t]
    else:
        c = [(93 + 70 * af) / 128, (7 + 18 * af) / 16, (-7 + 14 * af) / 32, (1 - 2 * af) / 16, (-1 + 2 * af) / 128]
        t = [[1 + 254 * af, 248 + 16 * af, 28 + 200 * af, -56 + 112 * af, 70 - 140 * af, -56 + 112 * af, 28 - 56 * af,
              -8 + 16 * af, 1 - 2 * af],
             [-1 + 2 * af, 8 + 240 * af, 228 + 56 * af, 56 + 144 * af, -70 + 140 * af, 56 - 112 * af, -28 + 56 * af,
              8 - 16 * af, -1 + 2 * af],
             [1 - 2 * af, -8 + 16 * af, 28 + 200 * af, 200 + 112 * af, 70 + 116 * af, -56 + 112 * af, 28 - 56 * af,
              -8 + 16 * af, 1 - 2 * af]]
        t = [[v / 256 for v in r] for r in t]
    a, b = _banded(n, {-1: af, 0: 1.0, 1: af}, {s * k: v / 2 for k, v in enumerate(c) for s in (1, -1)} | {0: c[0]},
                   not wall)
    if wall:
        _rows(a, b, {0: ({0: 1.0}, [1.0], 1), **{r: ({-1: af, 0: 1.0, 1: af}, row, 1) for r, row in enumerate(t, 1)}})
    return np.linalg.solve(a, b)


def _testfilter_matrix(n, wall):
    """The test filter of the dynamic model: 11-point right-hand side, pentadiagonal left-hand side."""
    w = [7 / 24, 175 / 768, 5 / 48, 35 / 1536, 0.0, -1 / 1536]
    a, b = _banded(n, {-2: 5 / 24, 0: 7 / 12, 2: 5 / 24}, {s * k: v for k, v in enumerate(w) for s in (1, -1)},
                   not wall)
    if wall:
        e = [11 / 16, 15 / 64, -3 / 32, 1 / 64]
        t = [[31 / 32, 5 / 32, -5 / 16, 5 / 16, -5 / 32, 1 / 32], [1 / 32, 27 / 32, 5 / 16, -5 / 16, 5 / 32, -1 / 32],
             [-1 / 32, 5 / 32, 11 / 16, 5 / 16, -5 / 32, 1 / 32]]
        t += [[0.0] * (r - 3) + e[:0:-1] + e for r in (3, 4)]
        _rows(a, b, {r: ({0: 1.0}, row, 1) for r, row in enumerate(t)})
    return np.linalg.solve(a, b)


def _cuda(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _along(mat, f, d):
    if d == 0:
        return torch.matmul(f, mat.T)
    if d == 1:
        return torch.matmul(mat, f)
    return torch.matmul(mat, f.reshape(f.shape[0], -1)).reshape(f.shape)


def _filtered(mat, f, d, bcs):
    """One direction of a filter: lines on a wall of another direction pass through."""
    out = _along(mat, f, d)
    for o in range(3):
        if o != d and bcs[o]:
            for at in (0, -1):
                out.select(2 - o, at).copy_(f.select(2 - o, at))
    return out


class _Exact:
    """One time step of a case's flow, FP64."""

    def __init__(self, case):
        self.case, self.bcs = case, _bcs(case)
        self.n = (case["nx"], case["ny"], case["nz"])
        self.fd = case.get("fd", "PADE6")
        self.dxi = [1.0 / (n - 1.0) if w else 1.0 / n for n, w in zip(self.n, self.bcs)]
        self.D = [_cuda(_deriv_matrix(self.fd, n, w)) for n, w in zip(self.n, self.bcs)]
        ft, af = case.get("filter", "COMPACT10"), case.get("alphaF", 0.49)
        self.F = [_cuda(_filter_matrix(ft, af, n, w)) for n, w in zip(self.n, self.bcs)]
        self.les = case.get("les", "DSM")
        if self.les == "DSM":
            self.T = [_cuda(_testfilter_matrix(n, w)) for n, w in zip(self.n, self.bcs)]
        self.mu_ref = _mu(case)
        self.sigma = None
        if case["family"] == "box":
            one = torch.ones((1, 1, 1), dtype=torch.float64, device="cuda")
            L, zero = 2 * math.pi, 0.0 * one
            self.J, self.Jm = one / L ** 3, [[one / L if i == j else zero for j in range(3)] for i in range(3)]
        elif case["family"] == "channel":
            met = [_cuda(a) for a in _channel_metrics(case)]
            self.J, self.Jm = met[0], [met[1:4], met[4:7], met[7:10]]
        else:
            self.mesh(*_ogrid_mesh(case))

    def d(self, f, k):
        return _along(self.D[k], f, k)

    def mesh(self, x, y, z):
        """Metrics of the O-grid from its coordinates: cofactors of the products of their derivatives; z, the one
        translated direction, has its values shifted by the span beyond its ends."""
        X = [_cuda(a) for a in (x, y, z)]
        n = self.n[2]
        lhs, rhs, _ = _deriv_parts(self.fd, n, False)
        up, down = (_banded(n, {0: 1.0}, rhs, True, side)[1] for side in (1, -1))
        wrap = _cuda(np.linalg.solve(_banded(n, lhs, {}, True)[0], up - down) * n)

        def dt(w, c, k):   # d(w X_c)/dxi_k
            f = self.d(w * X[c], k)
            return f + 2.0 * _along(wrap, w, 2) if k == 2 and c == 2 else f
        one = torch.ones_like(X[0])
        e1, e2 = [dt(one, 0, j) for j in range(3)], [dt(one, 1, j) for j in range(3)]
        va, vb, vc = (lambda j, k: dt(e1[j], 1, k)), (lambda j, k: dt(e1[j], 2, k)), (lambda j, k: dt(e2[j], 2, k))
        rows = []
        for i, j in ((1, 2), (2, 0), (0, 1)):
            rows.append([vc(i, j) - vc(j, i), vb(j, i) - vb(i, j), va(i, j) - va(j, i)])
        det = 0.0
        for i in range(3):
            for c in range(3):
                det = det + dt(rows[i][c], c, i) / 3.0
        self.J = 1.0 / det
        self.Jm = [[self.J * c for c in r] for r in rows]
        rad = torch.sqrt(X[0] ** 2 + X[1] ** 2)
        rmax = max(float(X[0].abs().max()), float(X[1].abs().max()))
        s = (rad - SPONGE["rmin"]) / (rmax - SPONGE["rmin"])
        self.sigma = torch.where(rad > SPONGE["rmin"], 0.068 * s ** 2 + 0.845 * s ** 8, 0.0 * s)

    # -- thermodynamics, walls --------------------------------------------
    def prims(self, q):
        rho = q[0]
        u = [c / rho for c in q[1:4]]
        p = (GAMMA - 1) * (q[4] - 0.5 * rho * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2))
        t = p / (rho * R_GAS)
        return [*u, p, t, self.mu_ref * t ** 0.76]

    def wall_faces(self):
        return {"box": (), "channel": ((0, False), (-1, False)), "ogrid": ((0, True),)}[self.case["family"]]

    @staticmethod
    def neumann(t, at):
        c = (360, -450, 400, -225, 72, -10)
        return sum(v * t[:, (k if at == 0 else -1 - k), :] for k, v in enumerate(c, 1)) / 147.0

    def start(self, rho, u, v, w, p):
        u = [u.clone(), v.clone(), w.clone()]
        t = p / (rho * R_GAS)
        mu = self.mu_ref * t ** 0.76
        for at, adiabatic in self.wall_faces():
            for c in u:
                c[:, at, :] = 0.0
            if adiabatic:
                t[:, at, :] = self.neumann(t, at)
        p = rho * R_GAS * t
        self.q1 = [rho, rho * u[0], rho * u[1], rho * u[2],
                   p / (GAMMA - 1) + 0.5 * rho * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)]
        self.target = [a.clone() for a in self.q1]
        self.pr = [*u, p, t, mu]
        self.k2 = [torch.zeros_like(rho) for _ in range(5)]

    def wall_prestep(self, q, pr):
        if not self.wall_faces():
            return pr
        pr = [a.clone() for a in pr]
        for at, adiabatic in self.wall_faces():
            f = (slice(None), at)
            if adiabatic:
                pr[4][f] = self.neumann(pr[4], at)
            for k in range(3):
                pr[k][f] = 0.0
                q[1 + k][f] = 0.0
            pr[3][f] = q[0][f] * R_GAS * pr[4][f]
            q[4][f] = pr[3][f] / (GAMMA - 1)
        return pr

    # -- closures ------------------------------------------------------------
    def hat(self, f):
        for d in (1, 2, 0):
            f = _filtered(self.T[d], f, d, self.bcs)
        return f

    def vreman(self, gu, rho):
        d1 = (self.dxi[0] * self.dxi[1] * self.dxi[2] / self.J) ** (2.0 / 3.0)
        b = {(i, j): d1 * (gu[i][0] * gu[j][0] + gu[i][1] * gu[j][1] + gu[i][2] * gu[j][2])
             for i, j in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))}
        # the sum of squares takes dw/dy twice and leaves dv/dz out, as the model is defined here
        a = sum(g * g for r in gu for g in r) - gu[1][2] ** 2 + gu[2][1] ** 2
        bb = (b[0, 0] * b[1, 1] - b[0, 1] ** 2 + b[0, 0] * b[2, 2] - b[0, 2] ** 2 + b[1, 1] * b[2, 2] - b[1, 2] ** 2)
        mu = 2.5 * 0.17 ** 2 * rho * torch.sqrt(bb.clamp(min=1e-12) / (a + 1e-12))
        return torch.minimum(mu, 0.05 * d1 * torch.sqrt(2.0 * a))

    def dsm_mu(self, gu, q):
        rho = q[0]
        S = {(i, j): 0.5 * (gu[i][j] + gu[j][i]) for i in range(3) for j in range(i, 3)}
        mag = torch.sqrt(sum((2.0 if i == j else 4.0) * s * s for (i, j), s in S.items()))
        tr = (S[0, 0] + S[1, 1] + S[2, 2]) / 3
        Sh = {k: self.hat(s) for k, s in S.items()}
        trh = (Sh[0, 0] + Sh[1, 1] + Sh[2, 2]) / 3
        rh, mh = self.hat(rho), self.hat(mag)
        uh = [self.hat(c) for c in q[1:4]]
        M, L = {}, {}
        for (i, j), s in S.items():
            same = 1.0 if i == j else 0.0
            M[i, j] = self.hat(2 * rho * mag * (s - same * tr)) - 8 * rh * mh * (Sh[i, j] - same * trh)
            L[i, j] = self.hat(q[1 + i] * q[1 + j] / rho) - uh[i] * uh[j] / rh
        ci = 8 * rh * mh * mh - self.hat(2 * rho * mag * mag)
        lkk = L[0, 0] + L[1, 1] + L[2, 2]
        lm = sum((1.0 if i == j else 2.0) * (L[i, j] - (lkk / 3 if i == j else 0.0)) * M[i, j] for i, j in M)
        mm = sum((1.0 if i == j else 2.0) * M[i, j] ** 2 for i, j in M)
        mu = rho * mag * (lm.mean() / mm.mean())
        return mu, 2 * rho * mag * mag * (lkk.mean() / ci.mean()), (mag, rh, mh, uh)

    def dsm_k(self, gt, q, t, ctx):
        mag, rh, mh, uh = ctx
        rho, rth = q[0], self.hat(q[0] * t)
        nn = nk = 0.0
        for i in range(3):
            ni = 4 * rh * mh * self.hat(gt[i]) - self.hat(rho * mag * gt[i])
            ki = self.hat(q[1 + i] * t) - uh[i] * rth / rho
            nn, nk = nn + ni * ni, nk + ki * ni
        return -CP * (nk.mean() / nn.mean()) * rho * mag

    def learned(self, gu, gt, rho, t):
        with open(WEIGHTS, "rb") as f:
            w = np.frombuffer(f.read()[8:], dtype=np.float32)
        mean, std, lo, hi, ym, ys, p = np.split(w, [9, 18, 27, 36, 38, 40])
        delta = (self.dxi[0] * self.dxi[1] * self.dxi[2] / self.J) ** (1.0 / 3.0)
        G = torch.stack([torch.stack(r, -1) for r in gu], -2)
        S, W = 0.5 * (G + G.transpose(-1, -2)), 0.5 * (G - G.transpose(-1, -2))
        s2, w2 = (S * S).sum((-1, -2)), (W * W).sum((-1, -2))
        SS, WW = S @ S, W @ W
        e, sw = 1e-30, s2 + w2
        mag = torch.sqrt(2 * s2)
        x = [torch.log1p(rho * delta ** 2 * mag / (self.mu_ref * t ** 0.76)), w2 / (sw + e),
             (SS * S).sum((-1, -2)) / (s2 ** 1.5 + e), (S * WW).sum((-1, -2)) / (sw ** 1.5 + e),
             (SS * WW).sum((-1, -2)) / (sw * sw + e), (gu[0][0] + gu[1][1] + gu[2][2]) / (torch.sqrt(sw) + e),
             delta * torch.sqrt(gt[0] ** 2 + gt[1] ** 2 + gt[2] ** 2) / t, delta * mag / torch.sqrt(t), torch.log(rho)]
        del G, S, W, SS, WW
        x = torch.stack([a.reshape(-1) for a in x], 1)
        x = (torch.clamp(x, _cuda(lo), _cuda(hi)) - _cuda(mean)) / _cuda(std)
        o = torch.cat([_network(_cuda(p), c)[0] for c in x.split(1 << 20)]) * _cuda(ys) + _cuda(ym)
        mu = o[:, 0].reshape(rho.shape).clamp(min=0.0) * rho * delta ** 2 * mag
        return mu, CP * mu / o[:, 1].reshape(rho.shape).clamp(0.1, 10.0)

    # -- one stage -------------------------------------------------------------
    def rhs(self, q, pr, dt):
        J, Jm, les = self.J, self.Jm, self.les
        u, (p, t, mu) = pr[:3], pr[3:]
        uc = [sum(Jm[i][c] * u[c] for c in range(3)) for i in range(3)]

        def grad(f):
            g = [self.d(f, k) for k in range(3)]
            return [sum(Jm[k][c] * g[k] for k in range(3)) for c in range(3)]
        gu = [grad(c) for c in u]
        ms = ks = None
        if les == "VREMAN":
            ms = self.vreman(gu, q[0])
            ks = CP * ms / 0.9
        elif les == "DSM":
            ms, tkk, ctx = self.dsm_mu(gu, q)
            p = p - 0.5 * tkk
            t = p / (q[0] * R_GAS)
            mu = self.mu_ref * t ** 0.76
        gt = grad(t)
        if les == "DSM":
            ks = self.dsm_k(gt, q, t, ctx)
        elif les == "MLP":
            ms, ks = self.learned(gu, gt, q[0], t)
        me, ke = mu, CP / PR * mu
        if ms is not None:
            me, ke = (mu + ms).clamp(min=0.0), (ke + ks).clamp(min=0.0)
        div = gu[0][0] + gu[1][1] + gu[2][2]
        tau = [[me * (gu[i][j] + gu[j][i] - (2 / 3 * div if i == j else 0.0)) for j in range(3)] for i in range(3)]
        vis = [sum(u[c] * tau[c][j] for c in range(3)) + ke * gt[j] for j in range(3)]
        k2, mass = [], None
        for e in range(5):
            r = 0.0
            for i in range(3):
                if e == 0:
                    f = q[0] * uc[i]
                elif e < 4:
                    f = q[e] * uc[i] + Jm[i][e - 1] * p - sum(Jm[i][c] * tau[e - 1][c] for c in range(3))
                else:
                    f = (q[4] + p) * uc[i] - sum(Jm[i][c] * vis[c] for c in range(3))
                df = self.d(f / J, i)
                if e == 0 and i == 1:
                    mass = df
                r = r - df
            if self.sigma is not None:
                r = r + self.sigma * (self.target[e] - q[e]) / J
            if 0 < e < 4:   # the momentum right-hand sides add to the last stage's, as the scheme is defined here
                r = r + self.k2[e]
            k2.append(r * (dt * J))
        for at, _ in self.wall_faces():
            f = (slice(None), at)
            k2[0][f] = -dt * J[f] * mass[f]
            for e in range(1, 5):
                k2[e][f] = 0.0
        if self.sigma is not None:
            for e in range(5):
                k2[e][:, -1] = 0.0
        self.k2 = k2

    def step(self):
        u, sos = self.pr[:3], torch.sqrt(GAMMA * self.pr[3] / self.q1[0])
        dt = 0.5 / float(sum(self.Jm[k][k] * (u[k].abs() + sos) / self.dxi[k] for k in range(3)).max())
        rk = self.case.get("rk", "KENRK4")
        A, B = {"RK4": ((1 / 6, 1 / 3, 1 / 3, 1 / 6), (0.5, 0.5, 1.0)), "TVDRK3": ((1, 2, 3), ()),
                "KENRK4": ((0.0, -6234157559845 / 12983515589748, -6194124222391 / 4410992767914,
                            -31623096876824 / 15682348800105, -12251185447671 / 11596622555746),
                           (494393426753 / 4806282396855, 4047970641027 / 5463924506627,
                            9795748752853 / 13190207949281, 4009051133189 / 8539092990294,
                            1348533437543 / 7166442652324)),
                "LSLDDRK4": ((0.0, -0.60512264332862261228, -2.04375640234761394333, -0.74069990637544192841,
                              -4.42317651302968168941),
                             (0.26874543888713438496, 0.8014706973220802933, 0.50515704269422722538,
                              0.56235680379000296407, 0.05900655127758823335))}[rk]
        q1, qk = self.q1, self.q1
        acc, reg = q1, None
        for s in range(len(A)):
            self.rhs(qk, self.wall_prestep(qk, self.pr), dt)
            k2 = self.k2
            if rk == "RK4":
                acc = [a + A[s] * k for a, k in zip(acc, k2)]
                qk = [a + B[s] * k for a, k in zip(q1, k2)] if s < 3 else acc
            elif rk == "TVDRK3":
                c = ((0, 1, 1), (3 / 4, 1 / 4, 1 / 4), (1 / 3, 2 / 3, 2 / 3))[s]
                qk = [c[0] * a + c[1] * b + c[2] * k for a, b, k in zip(q1, qk, k2)]
            else:
                reg = k2 if s == 0 else [k + A[s] * r for k, r in zip(k2, reg)]
                qk = [b + B[s] * r for b, r in zip(qk, reg)]
            self.pr = self.prims(qk)
        out = []
        for f in qk:   # the first step's filter runs along y, z, x
            for d in (1, 2, 0):
                f = _filtered(self.F[d], f, d, self.bcs)
            out.append(f)
        return out


def _network(p, x):
    """(outputs, pre- and post-activations) of the 9-64-64-64-2 GELU network, x normalised."""
    at, h, kept = 0, x, []
    for nin, nout in ((9, 64), (64, 64), (64, 64), (64, 2)):
        w, b = p[at:at + nin * nout].reshape(nout, nin), p[at + nin * nout:at + nin * nout + nout]
        at += nin * nout + nout
        z = h @ w.T + b
        kept.append((h, z, w))
        h = torch.nn.functional.gelu(z, approximate="tanh") if nout == 64 else z
    return h, kept


def exact(case, seed):
    if case["family"] in ("deriv", "filter"):
        f, bcs, outs = [a.double() for a in _fields(case, seed)], _bcs(case), []
        for d in case["dirs"]:
            d = "xyz".index(d)
            n = (case["nx"], case["ny"], case["nz"])[d]
            if case["family"] == "deriv":
                mat = _cuda(_deriv_matrix(case["op"], n, bcs[d]))
                outs.append([_along(mat, a, d) for a in f])
            else:
                mat = _cuda(_filter_matrix(case["op"], case["alphaF"], n, bcs[d]))
                f = [_filtered(mat, a, d, bcs) for a in f]
        return outs if case["family"] == "deriv" else f
    if case["family"] == "mlp":
        p, mean, std, x, y = _mlp_inputs(case, seed)
        x = (x.double() - _cuda(mean)) / _cuda(std)
        p = _cuda(p).requires_grad_(case["op"] == "train")
        o = _network(p, x)[0]
        if case["op"] == "infer":
            return o
        loss = ((o - y.double()) ** 2).sum() / case["batch"]
        g, = torch.autograd.grad(loss, p)
        return {"loss": float(loss.detach()), "params": (p - 1e-3 * g / (g.abs() + 1e-8)).detach()}
    s = _Exact(case)
    s.start(*_initial(case, seed))
    return s.step()


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how far results may differ
# ---------------------------------------------------------------------------
def work(case):
    if case["family"] == "mlp":
        # 8832 weights: two operations each forward, four more backward
        b, train = case["batch"], case["op"] == "train"
        return {"bytes": b * 44.0 + (9090 * 4 * 7 if train else 0), "flops": b * 8832 * (6.0 if train else 2.0)}
    n = float(case["nx"] * case["ny"] * case["nz"])
    if case["family"] in ("deriv", "filter"):
        size = 8 if case["precision"] == "FP64" else 4
        k, dirs = case["fields"], len(case["dirs"])
        # every input once; each direction's derivative, or the last filtered fields, once
        return {"bytes": n * size * k * (1.0 + (dirs if case["family"] == "deriv" else 1)),
                "flops": n * k * dirs * {"PADE6": 12.0, "PENTA10": 19.0, "COMPACT8": 17.0, "COMPACT10": 20.0}[case["op"]]}
    # per stage: the state and the scheme's second register read and written (FP64), and the filter of the step;
    # 27 line derivatives and about 250 operations of fluxes and update per point and stage
    rk = case.get("rk", "KENRK4")
    stages = {"RK4": 4, "TVDRK3": 3, "KENRK4": 5, "LSLDDRK4": 5.5}[rk]
    flops = 27 * (19.0 if case.get("fd") == "PENTA10" else 12.0) + 250
    les = case.get("les", "DSM")
    if les == "MLP":
        flops += 2 * 8832 + 150
    elif les == "DSM":   # 34 test filters of three directions
        flops += 34 * 3 * 27 + 200
    elif les == "VREMAN":
        flops += 60
    return {"bytes": n * (stages * 160.0 + 80.0), "flops": n * (stages * flops + 5 * 3 * 18)}


def tolerance(case):
    # about four times the distance of one pass from its 64-bit counterpart
    if case["family"] == "mlp":
        return {"rel": 1e-6, "max": 5e-3} if case["op"] == "train" else {"rel": 2e-2, "max": 2e-1}
    fp64 = case["precision"] == "FP64"
    if case["family"] == "deriv":   # differences of neighbours: relative to a derivative of a field with small scales
        return {"rel": 6e-14, "max": 6e-13} if fp64 else {"rel": 3e-5, "max": 3e-4}
    if case["family"] == "filter":
        return {"rel": 1e-14, "max": 1e-13} if fp64 else {"rel": 1e-5, "max": 6e-5}
    if case.get("les") == "MLP" and fp64:   # BF16 inside the closure
        return {"rel": 3e-7, "max": 6e-6}
    if case["family"] == "ogrid" and fp64:   # metrics by cancelling products; the span momentum is small
        return {"rel": 3e-12, "max": 3e-10}
    return {"rel": 1e-13, "max": 1e-12} if fp64 else {"rel": 1e-5, "max": 2e-4}
