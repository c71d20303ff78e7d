"""What a user of this library has it do, as cases that can be timed: the fermion-matrix operators, CG solves, point-source
propagators, log det M, the force and leapfrog trajectories, through the package's public entry points.

Sizes are those of the repository's own workloads: honeycomb 3x3 with Nt=16 (the CPU-runnable HMC configuration),
5x5 and 6x6 with Nt=32 (chain batches, correlators), 12x12 with Nt=64, beta=8, U=3 and 64 right-hand sides (the headline
workload), 24x24 with Nt=128, beta=12 (the precision configuration). Fields are phi ~ N(0, delta U), right-hand sides
complex Gaussians or point sources. Solves use tolerances tight enough that the solution
itself is determined, and trajectories a coupling at which they do not amplify rounding.

`exact` evaluates the same quantities with torch in complex128: operators as einsums, solves and the equal-time Green
functions through the block-cyclic matrix M reduced to chunk boundaries (its blocks stay well conditioned at any beta).
"""
import functools
import math

import numpy as np
import torch

import nsl_gb300 as N
from nsl_gb300.action import HubbardFermionAction, HubbardGaugeAction
from nsl_gb300.configuration import Configuration
from nsl_gb300.integrator import Leapfrog, LeapfrogRealForce
from nsl_gb300.measurement import TwoPointCorrelator

DEV = "cuda"
OPS = ("M", "Mdagger", "MMdagger", "MdaggerM")


def listed():
    return [
        # one vector on the smallest lattice of the repository: what a call costs when the work is nothing
        _apply("apply_m_3x3", "honeycomb:3x3", 16, 4.0, 2.0, 1, "M", "fp64"),
        # the plain FP64 operator, the drop-in of the reference's, on the headline workload
        _apply("apply_mmdag_12x12_fp64", "honeycomb:12x12", 64, 8.0, 3.0, 64, "MMdagger", "fp64"),
        # the inner operator of the mixed-precision solver on the headline workload
        _apply("apply_m_12x12_split", "honeycomb:12x12", 64, 8.0, 3.0, 64, "M", "bf16split"),
        # and on the largest lattice of the repository
        _apply("apply_mdag_24x24_split", "honeycomb:24x24", 128, 12.0, 3.0, 8, "Mdagger", "bf16split"),
        # CG as the reference's constructor gives it (FP64, one system, recurrence rule)
        {"name": "cg_reference_3x3", "kind": "cg", "lattice": "honeycomb:3x3", "Nt": 16, "beta": 4.0, "U": 2.0, "rhs": 1,
         "mode": "shared", "precision": "fp64", "stop": "recurrence", "eps": 1e-12},
        # the batched mixed-precision solve, certified in double-double: every right-hand side its own system
        {"name": "cg_mixed_12x12", "kind": "cg", "lattice": "honeycomb:12x12", "Nt": 64, "beta": 4.0, "U": 1.0, "rhs": 64,
         "mode": "per_rhs", "precision": "bf16split", "stop": "true_residual_dd", "eps": 1e-12},
        # what the correlator service does with a batch of requests of different shapes: one grouped solve
        {"name": "cg_group_mix", "kind": "group", "shapes": "honeycomb:3x3:16,ring:18:64,honeycomb:5x5:32,honeycomb:6x6:64",
         "beta": 4.0, "U": 1.0, "precision": "bf16split", "stop": "true_residual_dd", "eps": 1e-12},
        # a two-point correlator with the class's default arithmetic
        {"name": "correlator_6x6", "kind": "correlator", "lattice": "honeycomb:6x6", "Nt": 32, "beta": 4.0, "U": 1.0,
         "sources": 2, "precision": "tf32x3", "eps": 1e-11},
        # one HMC trajectory of the CPU-runnable configuration
        {"name": "leapfrog_3x3", "kind": "leapfrog", "lattice": "honeycomb:3x3", "Nt": 16, "beta": 4.0, "U": 1.0, "nconf": 1,
         "nmd": 10, "real": True, "precision": "fp64"},
        # a batch of chains on a lattice whose size divides no tile
        {"name": "chains_5x5", "kind": "leapfrog", "lattice": "honeycomb:5x5", "Nt": 32, "beta": 4.0, "U": 1.0, "nconf": 16,
         "nmd": 10, "real": True, "precision": "fp64"},
        # one force of the headline HMC: the stratified FP64 gradient of both species
        {"name": "force_12x12", "kind": "force", "lattice": "honeycomb:12x12", "Nt": 64, "beta": 8.0, "U": 3.0,
         "precision": "fp64"},
        # the action of the accept step there: two stratified log dets
        {"name": "action_12x12", "kind": "action", "lattice": "honeycomb:12x12", "Nt": 64, "beta": 8.0, "U": 3.0, "nconf": 1},
    ]


def _apply(name, lattice, Nt, beta, U, rhs, op, precision, disc="exp"):
    return {"name": name, "kind": "apply", "lattice": lattice, "Nt": Nt, "beta": beta, "U": U, "rhs": rhs, "op": op,
            "precision": precision, "disc": disc}


def _pure(case):
    return {k: v for k, v in case.items() if k != "name"}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_lattice(rng, max_sites):
    """A honeycomb of L1 x L2 unit cells or a ring, 4 sites up, sizes spread over their logarithm."""
    n = _log_int(rng, 8, max_sites)
    if rng.random() < 0.25:
        return "ring:%d" % n
    L1 = max(2, int(round(math.sqrt(n / 2))) + rng.choice((-1, 0, 0, 1)))
    L2 = max(2, int(n / 2 / L1))
    return "honeycomb:%dx%d" % (L1, L2)


def draw(rng):
    kind = rng.choice(("apply", "apply", "apply", "cg", "cg", "group", "correlator", "leapfrog", "leapfrog", "force", "action"))
    U = round(rng.uniform(1.0, 3.0), 2)
    if kind == "apply":
        lat = _draw_lattice(rng, 1152)
        Nx = _sites(lat)
        Nt = _log_int(rng, 8, 128)
        rhs = max(1, min(_log_int(rng, 1, 128), 2_000_000 // (Nx * Nt)))
        precision = rng.choice(("fp64", "fp64", "bf16split", "bf16split", "tf32x3", "fp32"))
        disc = "diag" if precision == "fp64" and rng.random() < 0.25 else "exp"
        if precision == "fp64":  # the FP64 operator is the slow one
            rhs = max(1, min(rhs, 400_000_000 // (Nx * Nx * Nt)))
        return _pure(_apply("", lat, Nt, round(Nt * rng.uniform(0.06, 0.25), 3), U, rhs, rng.choice(OPS), precision, disc))
    if kind == "cg":
        if rng.random() < 0.5:  # the reference's rule, one system
            lat, Nt = _draw_lattice(rng, 72), _log_int(rng, 8, 32)
            return {"kind": "cg", "lattice": lat, "Nt": Nt, "beta": round(Nt * rng.uniform(0.06, 0.15), 3), "U": 1.0,
                    "rhs": rng.choice((1, 2, 5)), "mode": "shared", "precision": "fp64", "stop": "recurrence", "eps": 1e-12}
        lat, Nt = _draw_lattice(rng, 400), _log_int(rng, 16, 64)
        rhs = max(1, min(_log_int(rng, 1, 64), 1_000_000 // (_sites(lat) * Nt)))
        return {"kind": "cg", "lattice": lat, "Nt": Nt, "beta": round(Nt * 0.0625, 3), "U": 1.0, "rhs": rhs,
                "mode": "per_rhs", "precision": "bf16split", "stop": "true_residual_dd", "eps": 1e-12}
    if kind == "group":
        shapes = ",".join("%s:%d" % (_draw_lattice(rng, 80), _log_int(rng, 12, 48)) for _ in range(rng.choice((2, 3, 4))))
        return {"kind": "group", "shapes": shapes, "beta": 2.0, "U": 1.0, "precision": "bf16split", "stop": "true_residual_dd",
                "eps": 1e-12}
    if kind == "correlator":
        lat, Nt = _draw_lattice(rng, 72), _log_int(rng, 12, 40)
        return {"kind": "correlator", "lattice": lat, "Nt": Nt, "beta": round(Nt * 0.1, 3), "U": 1.0,
                "sources": rng.choice((1, 2)), "precision": rng.choice(("tf32x3", "bf16split")), "eps": 1e-11}
    if kind == "leapfrog":
        lat, Nt = _draw_lattice(rng, 128), _log_int(rng, 8, 48)
        nconf = max(1, min(_log_int(rng, 1, 32), 20_000_000 // (_sites(lat) ** 2 * Nt)))
        return {"kind": "leapfrog", "lattice": lat, "Nt": Nt, "beta": round(min(4.0, Nt * 0.125), 3), "U": 1.0, "nconf": nconf,
                "nmd": rng.choice((3, 5, 10)), "real": rng.random() < 0.7, "precision": "fp64"}
    lat, Nt = _draw_lattice(rng, 288), _log_int(rng, 12, 64)
    if kind == "force":
        fast = rng.random() < 0.3  # the tensor-core force, at the temperatures where it keeps its digits
        beta = min(1.5, Nt * 0.0625) if fast else min(8.0, Nt * rng.uniform(0.06, 0.15))
        return {"kind": "force", "lattice": lat, "Nt": Nt, "beta": round(beta, 3), "U": U, "precision": "bf16split" if fast else "fp64"}
    beta = min(8.0, Nt * rng.uniform(0.06, 0.15))
    nconf = max(1, min(_log_int(rng, 1, 16), 16_000_000 // (_sites(lat) ** 2 * Nt)))
    return {"kind": "action", "lattice": lat, "Nt": Nt, "beta": round(beta, 3), "U": U, "nconf": nconf}


# ---- inputs ------------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _lattice(spec):
    kind, size = spec.split(":")
    if kind == "ring":
        return N.Ring(int(size))
    return N.Honeycomb(tuple(int(v) for v in size.split("x")))


def _sites(spec):
    kind, size = spec.split(":")
    return int(size) if kind == "ring" else 2 * math.prod(int(v) for v in size.split("x"))


def _shapes(case):
    """(lattice, Nt) of every instance of a case."""
    if case["kind"] == "group":
        out = []
        for s in case["shapes"].split(","):
            kind, size, Nt = s.split(":")
            out.append((kind + ":" + size, int(Nt)))
        return out
    return [(case["lattice"], case["Nt"])]


def _fields(case, seed):
    """phi ~ N(0, delta U) per instance and configuration, and the Gaussian vectors of the case."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    out = []
    for lat, Nt in _shapes(case):
        n = _sites(lat)
        lead = (case["nconf"],) if case.get("nconf", 1) > 1 else ()
        phi = torch.randn(lead + (Nt, n), generator=g, device=DEV, dtype=torch.float64) * math.sqrt(case["beta"] / Nt * case["U"])
        v = None
        if case["kind"] in ("apply", "cg"):
            v = torch.randn((case["rhs"], Nt, n, 2), generator=g, device=DEV, dtype=torch.float64)
            v = torch.view_as_complex(v)
        elif case["kind"] == "leapfrog":  # momenta are real
            v = torch.randn(lead + (Nt, n), generator=g, device=DEV, dtype=torch.float64).to(torch.complex128)
        elif case["kind"] == "group":  # a point source on every site of slice 0
            v = torch.zeros((n, Nt, n), device=DEV, dtype=torch.complex128)
            v[torch.arange(n), 0, torch.arange(n)] = 1.0
        out.append((phi.to(torch.complex128), v))
    return out


def _params(case):
    return {"Nt": case["Nt"], "beta": case["beta"], "U": case["U"]}


def prepare(case, seed):
    kind, fields = case["kind"], _fields(case, seed)
    phi, v = fields[0]
    state = {"case": case, "phi": phi, "v": v}
    if kind in ("apply", "cg", "correlator"):
        cls = N.HubbardDiag if case.get("disc") == "diag" else N.HubbardExp
        fm = cls(_lattice(case["lattice"]), case["Nt"], case["beta"])
        fm.populate(phi)
        state["fm"] = fm
        if kind == "cg":
            eps = case["eps"] * float(torch.linalg.vector_norm(v if case["mode"] == "shared" else v[0]))
            state["cg"] = N.CG(fm, N.MatrixCombination.MMdagger, eps, 200_000, mode=case["mode"], precision=case["precision"],
                               stop=case["stop"])
        elif kind == "correlator":
            state["correlator"] = TwoPointCorrelator(fm, eps=case["eps"], precision=case["precision"])
    elif kind == "group":
        items = []
        for (lat, Nt), (phi, v) in zip(_shapes(case), fields):
            fm = N.HubbardExp(_lattice(lat), Nt, case["beta"])
            fm.populate(phi)
            items.append((fm, v))
        state["items"] = items
    else:
        fermion = HubbardFermionAction(_lattice(case["lattice"]), _params(case), force_precision=case.get("precision", "fp64"))
        state["action"] = HubbardGaugeAction(_params(case)) + fermion
        if kind == "leapfrog":
            state["integrator"] = (LeapfrogRealForce if case["real"] else Leapfrog)(state["action"], 1.0, case["nmd"])
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "apply":
        return getattr(state["fm"], case["op"])(state["v"], precision=case["precision"])
    if kind == "cg":
        return state["cg"](state["v"])
    if kind == "group":
        xs, _, _ = N.cg_group(state["items"], eps=case["eps"], maxIter=200_000, precision=case["precision"], stop=case["stop"])
        return xs
    if kind == "correlator":
        return state["correlator"].measure(state["phi"], case["sources"])
    if kind == "leapfrog":
        q, p = state["integrator"](Configuration({"phi": state["phi"]}), Configuration({"phi": state["v"]}))
        return {"q": q["phi"], "p": p["phi"]}
    if kind == "force":
        return state["action"].force(state["phi"])["phi"]
    if case["nconf"] == 1:
        return np.array([state["action"].eval(state["phi"])])
    return state["action"].eval_batch(state["phi"])


def work(case):
    """Each input read once, each output written once, and the arithmetic of the reference's formulas: 4 real flops per
    element of the real Nx x Nx products of an operator application (two in MM^dagger); a CG solve at least Nt / 2
    iterations (a source's influence travels one slice per application); log det the Nt products and one LU per species;
    the gradient two such chains and one inverse, each complex product 8 Nx^3."""
    flops = data = 0.0
    for lat, Nt in _shapes(case):
        n, kind = _sites(lat), case["kind"]
        rhs = {"apply": case.get("rhs"), "cg": case.get("rhs"), "group": n, "correlator": n * case.get("sources", 1)}.get(kind, 1)
        one = 4.0 * Nt * n * n * rhs
        base = 8.0 * n * n + 16.0 * Nt * n
        nconf = case.get("nconf", 1)
        if kind == "apply":
            flops += one * (2 if case["op"] in ("MMdagger", "MdaggerM") else 1)
            data += base + 32.0 * Nt * n * rhs
        elif kind in ("cg", "group", "correlator"):
            flops += 2 * one * (Nt // 2)
            data += base + (32.0 * Nt * n * rhs if kind != "correlator" else 16.0 * Nt * n * n)
        elif kind == "action":
            flops += nconf * 2 * (8.0 * n ** 3 * Nt + 8.0 / 3 * n ** 3)
            data += 8.0 * n * n + nconf * 16.0 * Nt * n
        else:
            forces = case["nmd"] + 1 if kind == "leapfrog" else 1
            flops += nconf * forces * 2 * (2 * 8.0 * n ** 3 * Nt + 8.0 * n ** 3)
            data += 8.0 * n * n + nconf * (64.0 if kind == "leapfrog" else 32.0) * Nt * n
    return {"bytes": data, "flops": flops}


# ---- the same quantities in complex128, without this library ---------------------------------------------------------
def _hops(spec):
    """Nearest-neighbour hopping of the ring or the periodic honeycomb (sites in the order A, B per unit cell; a pair of sites is
    linked once however many of its images touch)."""
    kind, size = spec.split(":")
    n = _sites(spec)
    K = np.zeros((n, n))
    if kind == "ring":
        for i in range(n):
            K[i, (i + 1) % n] = K[(i + 1) % n, i] = 1.0
        return torch.from_numpy(K).to(DEV)
    L1, L2 = (int(v) for v in size.split("x"))
    for l2 in range(L2):
        for l1 in range(L1):
            # the A site of a cell at (1/2, 0) touches the B site (-1/2, 0) of its own cell and of the cells one lattice vector on
            a = 2 * (l1 + L1 * l2)
            for d1, d2 in ((0, 0), (1, 0), (0, 1)):
                b = 2 * ((l1 + d1) % L1 + L1 * ((l2 + d2) % L2)) + 1
                K[a, b] = K[b, a] = 1.0
    return torch.from_numpy(K).to(DEV)


def _expm(K, d):
    w, V = torch.linalg.eigh(K)
    return ((V * torch.exp(d * w)) @ V.T).to(torch.complex128)


class _Exact:
    """M of one species for fields phi (..., Nt, Nx): (M psi)_t = psi_t - B_t A_{t-1} psi_{t-1}, A_t = E diag(ph_t), B_0 = -1."""

    def __init__(self, spec, Nt, beta, phi, sgn=1):
        K = _hops(spec)
        self.Nt, self.n, self.d = Nt, K.shape[0], beta / Nt
        self.E, self.Ei = _expm(K, sgn * self.d), _expm(K, -sgn * self.d)
        self.ph, self.phi_inv = torch.exp(1j * sgn * phi), torch.exp(-1j * sgn * phi)
        rho = float(K.sum(0).max())
        self.k = max(1, min(Nt, int(2.0 / (self.d * rho))))
        self.starts = list(range(0, Nt, self.k))

    def M(self, v):
        z = torch.roll((self.ph * v) @ self.E.T, 1, -2)
        z[..., 0, :] *= -1
        return v - z

    def Mdagger(self, v):
        z = torch.roll(v @ self.E.conj(), -1, -2)
        z[..., -1, :] *= -1
        return v - self.ph.conj() * z

    def A(self, t):
        return self.E * self.ph[..., t, None, :]

    def reduced(self):
        """M with every slice between chunk starts eliminated, (..., J Nx, J Nx)."""
        J, n = len(self.starts), self.n
        lead = self.ph.shape[:-2]
        R = torch.zeros(lead + (J, n, J, n), dtype=torch.complex128, device=DEV)
        eye = torch.eye(n, dtype=torch.complex128, device=DEV)
        for j, s in enumerate(self.starts):
            R[..., j, :, j, :] += eye
            C = eye
            for t in range(s, self.starts[j + 1] if j + 1 < J else self.Nt):
                C = self.A(t) @ C
            R[..., (j + 1) % J, :, j, :] += C if j + 1 == J else -C
        return R.reshape(lead + (J * n, J * n))

    def solve(self, b):
        """M^{-1} b for b (rhs, Nt, Nx), one configuration."""
        J, n, rhs = len(self.starts), self.n, b.shape[0]
        ends = self.starts[1:] + [self.Nt]
        c = torch.zeros((J, rhs, n), dtype=torch.complex128, device=DEV)
        for j, s in enumerate(self.starts):
            w = torch.zeros((rhs, n), dtype=torch.complex128, device=DEV)
            for t in range(s, ends[j]):  # what the sources inside the chunk send to the next start
                if t > s:
                    w = w + b[:, t]
                w = (w * self.ph[t]) @ self.E.T
            c[(j + 1) % J] += -w if j + 1 == J else w
            c[j] += b[:, s]
        y = torch.linalg.solve(self.reduced(), c.permute(0, 2, 1).reshape(J * n, rhs)).reshape(J, n, rhs)
        x = torch.empty_like(b)
        for j, s in enumerate(self.starts):
            w = y[j].T
            x[:, s] = w
            for t in range(s + 1, ends[j]):
                w = b[:, t] + (w * self.ph[t - 1]) @ self.E.T
                x[:, t] = w
        return x

    def solve_dagger(self, b):
        """M^{-dagger} b, as solve() with the chunks closed at their last slices."""
        J, n, rhs, Nt = len(self.starts), self.n, b.shape[0], self.Nt
        # (M^dagger x)_t = x_t - s_t conj(ph_t) o (E^T x_{t+1}), s_{Nt-1} = -1: eliminate towards the chunk ends
        Ec, phc = self.E.conj(), self.ph.conj()
        stops = [s - 1 for s in self.starts[1:]] + [Nt - 1]  # last slice of each chunk
        c = torch.zeros((J, rhs, n), dtype=torch.complex128, device=DEV)
        for j, s in enumerate(self.starts):  # x at stop of chunk j - 1 from chunk j
            w = torch.zeros((rhs, n), dtype=torch.complex128, device=DEV)
            for t in range(stops[j], s - 1, -1):
                if t < stops[j]:
                    w = w + b[:, t]
                w = (w @ Ec) * phc[t - 1]
            c[(j - 1) % J] += -w if j == 0 else w
            c[j] += b[:, stops[j]]
        R = torch.zeros((J, n, J, n), dtype=torch.complex128, device=DEV)
        eye = torch.eye(n, dtype=torch.complex128, device=DEV)
        for j, s in enumerate(self.starts):
            R[j, :, j, :] += eye
            C = eye
            for t in range(stops[j], s - 1, -1):
                C = phc[t - 1][:, None] * (Ec.T @ C)
            R[(j - 1) % J, :, j, :] += C if j == 0 else -C
        y = torch.linalg.solve(R.reshape(J * n, J * n), c.permute(0, 2, 1).reshape(J * n, rhs)).reshape(J, n, rhs)
        x = torch.empty_like(b)
        for j, s in enumerate(self.starts):
            w = y[j].T
            x[:, stops[j]] = w
            for t in range(stops[j] - 1, s - 1, -1):
                w = b[:, t] + (w @ Ec) * phc[t]
                x[:, t] = w
        return x

    def logdet(self):
        sign, la = torch.linalg.slogdet(self.reduced())
        return torch.complex(la, torch.angle(sign))

    def grad(self):
        """i diag of the equal-time blocks of M^{-1}: inverted at the chunk starts, carried by W(t+1) = A_t W(t) A_t^{-1}."""
        J, n = len(self.starts), self.n
        lead = self.ph.shape[:-2]
        inv = torch.linalg.inv(self.reduced()).reshape(lead + (J, n, J, n))
        out = torch.empty(lead + (self.Nt, n), dtype=torch.complex128, device=DEV)
        ends = self.starts[1:] + [self.Nt]
        for j, s in enumerate(self.starts):
            W = inv[..., j, :, j, :]
            for t in range(s, ends[j]):
                out[..., t, :] = 1j * torch.diagonal(W, dim1=-2, dim2=-1)
                if t + 1 < ends[j]:
                    W = (self.A(t) @ W) @ (self.phi_inv[..., t, :, None] * self.Ei)
        return out


def _force(case, phi):
    gp = _Exact(case["lattice"], case["Nt"], case["beta"], phi, 1).grad()
    gh = _Exact(case["lattice"], case["Nt"], case["beta"], phi, -1).grad()
    return -phi / (case["beta"] / case["Nt"] * case["U"]) - (gp - gh)


def _too_long(case):
    """Whether the dense boundary systems would take longer than some seconds."""
    cost = 0.0
    for lat, Nt in _shapes(case):
        rho = 2.0 if lat.startswith("ring") else 3.0
        J = -(-Nt // max(1, min(Nt, int(2 * Nt / (case["beta"] * rho)))))
        m = J * _sites(lat)
        times = 2 * case.get("nconf", 1) * (case["nmd"] + 1 if case["kind"] == "leapfrog" else 1)
        cost += 8.0 * m ** 3 * times
        if m > 20_000 or 64.0 * m * m * case.get("nconf", 1) > 60e9:
            return True
    return cost > 6e12


def exact(case, seed):
    kind, fields = case["kind"], _fields(case, seed)
    phi, v = fields[0]
    if kind == "apply":
        if case["disc"] == "diag":
            K = (case["beta"] / case["Nt"] * _hops(case["lattice"])).to(torch.complex128)
            ph = torch.exp(1j * phi)

            def M(x):
                z = torch.roll(ph * x, 1, -2)
                z[..., 0, :] *= -1
                return x - x @ K.T - z

            def Mdagger(x):
                z = torch.roll(x, -1, -2)
                z[..., -1, :] *= -1
                return x - x @ K.conj() - ph.conj() * z
        else:
            e = _Exact(case["lattice"], case["Nt"], case["beta"], phi)
            M, Mdagger = e.M, e.Mdagger
        return {"M": M, "Mdagger": Mdagger, "MMdagger": lambda x: M(Mdagger(x)), "MdaggerM": lambda x: Mdagger(M(x))}[case["op"]](v)
    if _too_long(case):
        return None
    if kind in ("cg", "group"):
        xs = []
        for (lat, Nt), (phi, b) in zip(_shapes(case), fields):
            e = _Exact(lat, Nt, case["beta"], phi)
            xs.append(e.solve_dagger(e.solve(b)))
        return xs[0] if kind == "cg" else xs
    if kind == "correlator":
        Nt, n, e = case["Nt"], _sites(case["lattice"]), _Exact(case["lattice"], case["Nt"], case["beta"], phi)
        corr = torch.zeros((Nt, n, n), dtype=torch.complex128, device=DEV)
        for t0 in range(0, Nt, max(1, Nt // case["sources"])):
            b = torch.zeros((n, Nt, n), dtype=torch.complex128, device=DEV)
            b[torch.arange(n), t0, torch.arange(n)] = 1.0
            x = torch.roll(e.solve(b), -t0, 1)
            if t0:
                x[:, Nt - t0:] *= -1
            corr += x.permute(1, 2, 0)
        return (corr / case["sources"]).cpu().numpy()
    if kind == "force":
        return _force(case, phi)
    if kind == "action":
        S = (phi ** 2).sum((-2, -1)) / (2 * case["beta"] / case["Nt"] * case["U"])
        for sgn in (1, -1):
            S = S - _Exact(case["lattice"], case["Nt"], case["beta"], phi, sgn).logdet()
        return S.reshape(-1).cpu().numpy()
    eps = 1.0 / case["nmd"]
    q, p = phi.clone(), v.clone()

    def F(q):
        f = _force(case, q)
        return f.real.to(torch.complex128) if case["real"] else f

    p = p + eps / 2 * F(q)
    for step in range(case["nmd"]):
        q = q + eps * p
        p = p + (eps / 2 if step + 1 == case["nmd"] else eps) * F(q)
    return {"q": q, "p": p}
