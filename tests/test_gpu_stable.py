"""The stratified log det M and gradient on the GPU (nsl_gb300/csrc/stable.cu) against the oracle.

Small lattices: against i diag(M^{-1}) and the dense log-determinant of M (M is well conditioned, so a dense inverse
is exact to ~1e-14 where the time-slice product is not). Honeycomb 12x12, Nt = 64, beta = 8 and 24x24, Nt = 128,
beta = 12: against the oracle's stratified forms on selected slices (tests/golden/stable_cfg*.npz, made by
tests/golden/make_stable_golden.py), and, on every slice, the similarity invariant tr G(s) (the sum over sites of a
gradient row is the same for every time slice). Bars: 1e-12 relative (max-norm over the compared rows) for the
gradient and the force (5e-12 at beta = 12 on 24x24, where two stratified evaluations with different chunkings, QR
methods and wraps agree to 2e-12..4e-12, measured: the conditioning of G itself), 1e-12 relative (modulo 2 pi i) for
log det.
"""
import os

import numpy as np
import pytest

from conftest import GOLDEN_CASES, ROOT, load_golden, rel_err
from oracle import nsl_oracle as O

pytestmark = pytest.mark.gpu


def mod2pi(z):
    return complex(z.real, (z.imag + np.pi) % (2 * np.pi) - np.pi)


def _field(Nx, Nt, beta, seed, U=3.0, mu=0.0, complex_phi=False):
    rng = np.random.default_rng(seed)
    phi = rng.standard_normal((Nt, Nx)) * np.sqrt(beta / Nt * U) + 0j
    if complex_phi:
        phi = phi + 0.2j * rng.standard_normal(phi.shape)
    return phi


def _lat(L):
    import nsl_gb300 as N

    return N.Honeycomb(L) if isinstance(L, tuple) else N.Ring(L)


SMALL = [((2, 2), 32, 12.0, 0, 0.0, False), ((3, 3), 32, 12.0, 1, 0.0, False), ((2, 2), 16, 8.0, 0, 0.3, True),
         (6, 24, 10.0, 1, 0.0, False), ((3, 3), 16, 4.0, 0, 0.0, False), ((4, 4), 13, 9.0, 1, 0.0, False)]


@pytest.mark.parametrize("L,Nt,beta,species,mu,cphi", SMALL)
def test_stratified_vs_dense_inverse(L, Nt, beta, species, mu, cphi):
    import nsl_gb300 as N

    lat = _lat(L)
    phi = _field(lat.sites(), Nt, beta, 7, mu=mu, complex_phi=cphi)
    h = N.HubbardExp(lat, Nt, beta, mu, N.Species(species))
    h.set_stabilisation("stratified")
    h.populate(phi)
    ho = O.HubbardExp(lat.hopping_matrix(), Nt, beta, mu, species)
    ho.populate(phi)
    n = Nt * lat.sites()
    Md = ho.M_dense().reshape(n, n)
    want = 1j * np.diag(np.linalg.inv(Md)).reshape(Nt, lat.sites())
    assert rel_err(np.asarray(h.gradLogDetM()), want) < 1e-12
    s, l = np.linalg.slogdet(Md)
    ld = h.logDetM()
    ref = complex(l, np.angle(s))
    assert abs(mod2pi(ld - ref)) <= 1e-12 * max(1.0, abs(ref)), (ld, ref)
    assert -np.pi < ld.imag <= np.pi


def test_auto_selects_the_form_by_temperature():
    """AUTO takes the direct product where it is accurate (beta rho <= 14) and the stratified form beyond."""
    import nsl_gb300 as N

    for L, Nt, beta, stratified in (((3, 3), 16, 2.0, False), ((3, 3), 32, 12.0, True)):
        lat = _lat(L)
        phi = _field(lat.sites(), Nt, beta, 3)
        g = {}
        for mode in ("auto", "plain", "stratified"):
            h = N.HubbardExp(lat, Nt, beta)
            h.set_stabilisation(mode)
            h.populate(phi)
            g[mode] = np.asarray(h.gradLogDetM())
        assert np.array_equal(g["auto"], g["stratified" if stratified else "plain"])


@pytest.mark.parametrize("name", GOLDEN_CASES)
@pytest.mark.parametrize("species,tag", [(0, "P"), (1, "H")])
def test_stratified_vs_reference_fixtures(name, species, tag):
    """Within the reference's own rounding (~1e-15 at beta <= 2, 2e-12 at beta = 4, 3e-10 at beta = 8)."""
    from test_gpu_action import make

    g = load_golden(name)
    N, lat = make(g)
    h = N.HubbardExp(lat, g["Nt"], g["beta"], g["mu"])
    h.set_stabilisation("stratified")
    h.populate(g["phi"], N.Species(species))
    bar = 1e-13 if g["beta"] <= 2 else (5e-12 if g["beta"] <= 4 else 1e-9)
    assert rel_err(np.asarray(h.gradLogDetM()), g[f"grad_{tag}"]) < bar
    ref = complex(g[f"logdet_{tag}"])
    assert abs(mod2pi(h.logDetM() - ref)) <= max(bar, 1e-12) * max(1.0, abs(ref))


def _big(name):
    z = np.load(os.path.join(ROOT, "tests", "golden", f"stable_{name}.npz"))
    d = {k: z[k] for k in z.files}
    L1, L2, Nt, beta, U, seed = d["params"]
    d.update(L=(int(L1), int(L2)), Nt=int(Nt), beta=float(beta), U=float(U))
    return d


@pytest.mark.parametrize("name", ["cfg2", "cfg3"])
def test_stratified_low_temperature_configurations(name):
    """Honeycomb 12x12, Nt = 64, beta = 8 and 24x24, Nt = 128, beta = 12 (AUTO selects the stratified form): log det
    and the gradient of both species against the oracle's stratified forms; tr G(s) the same on every slice; the
    fermion force -(grad_P - grad_H) on the compared slices."""
    import nsl_gb300 as N
    from nsl_gb300.action import HubbardFermionAction

    d = _big(name)
    lat = N.Honeycomb(d["L"])
    h = N.HubbardExp(lat, d["Nt"], d["beta"])
    sl = d["slices"]
    grads = {}
    for sp, tag in ((N.Species.Particle, "P"), (N.Species.Hole, "H")):
        h.populate(d["phi"], sp)
        ref = complex(d[f"logdet_{tag}"])
        ld = h.logDetM()
        assert abs(mod2pi(ld - ref)) <= 1e-12 * abs(ref), (ld, ref)
        gr = np.asarray(h.gradLogDetM())
        assert rel_err(gr[sl], d[f"grad_{tag}"]) < (5e-12 if d["beta"] > 8 else 1e-12)
        rows = gr.sum(axis=1)  # i (Nx - tr G(t+1)): a similarity invariant
        assert np.abs(rows - rows[0]).max() <= 1e-11 * np.abs(rows[0])
        grads[tag] = gr
    F = np.asarray(HubbardFermionAction(lat, {"Nt": d["Nt"], "beta": d["beta"], "mu": 0.0}).force(
        {"phi": d["phi"]})["phi"])
    assert rel_err(F, -(grads["P"] - grads["H"])) < 1e-13
    assert rel_err(F[sl], -(d["grad_P"] - d["grad_H"])) < (5e-12 if d["beta"] > 8 else 1e-12)


def test_stratified_leapfrog_and_delta_h():
    """A LeapfrogRealForce trajectory at beta = 12 (honeycomb 3x3, Nt = 32, Nmd = 6) with the stratified force and
    action against the oracle's trajectory on its stratified forms: fields and momenta to 1e-10, Delta H to 1e-9."""
    import nsl_gb300 as N
    from nsl_gb300.action import HubbardFermionAction, HubbardGaugeAction
    from nsl_gb300.integrator import LeapfrogRealForce

    lat = N.Honeycomb((3, 3))
    Nt, beta, U, nmd = 32, 12.0, 3.0, 6
    phi = _field(lat.sites(), Nt, beta, 21, U=U)
    p0 = np.random.default_rng(22).standard_normal(phi.shape) + 0j
    params = {"Nt": Nt, "beta": beta, "mu": 0.0, "U": U}
    S = HubbardGaugeAction(params) + HubbardFermionAction(lat, params)
    SO = O.HubbardAction(lat.hopping_matrix(), Nt, beta, U, stable=True)
    for _ in range(3):  # eager, captured, replayed
        q1, p1 = LeapfrogRealForce(S, 1.0, nmd)({"phi": phi}, {"phi": p0})
    qo, po = O.leapfrog(SO, phi, p0, 1.0, nmd, real_force=True)
    assert rel_err(np.asarray(q1["phi"]), qo) < 1e-10
    assert rel_err(np.asarray(p1["phi"]), po) < 1e-10
    dH = (S(q1) + 0.5 * np.sum(np.asarray(p1["phi"]) ** 2)) - (S({"phi": phi}) + 0.5 * np.sum(p0 ** 2))
    dHo = O.hamiltonian(SO.eval(qo), po) - O.hamiltonian(SO.eval(phi), p0)
    assert abs(dH - dHo) < 1e-9 * max(1.0, abs(dHo)), (dH, dHo)


def test_split_force_keeps_direct_product_to_beta_rho_28():
    """Under AUTO the split-BF16 force setting keeps the direct product while beta rho <= 28 (honeycomb 6x6, Nt = 32,
    beta = 8: beta rho = 24), within 1e-7 of the stratified FP64 gradient the FP64 setting takes there; at
    beta rho = 36 it takes the stratified form like the FP64 setting."""
    from test_gpu_action import make

    g = load_golden("honey6x6_nt32_beta8")
    N, lat = make(g)
    grads = {}
    for fp, stab in (("bf16split", "auto"), ("bf16split", "plain"), ("fp64", "auto")):
        h = N.HubbardExp(lat, g["Nt"], g["beta"], g["mu"])
        h.set_force_precision(fp)
        h.set_stabilisation(stab)
        h.populate(g["phi"])
        grads[(fp, stab)] = np.asarray(h.gradLogDetM())
    assert np.array_equal(grads[("bf16split", "auto")], grads[("bf16split", "plain")])
    assert rel_err(grads[("bf16split", "auto")], grads[("fp64", "auto")]) < 1e-7
    lat3 = N.Honeycomb((3, 3))
    phi = _field(18, 32, 12.0, 5)
    out = {}
    for fp in ("bf16split", "fp64"):
        h = N.HubbardExp(lat3, 32, 12.0)
        h.set_force_precision(fp)
        h.populate(phi)
        out[fp] = np.asarray(h.gradLogDetM())
    assert np.array_equal(out["bf16split"], out["fp64"])


@pytest.mark.parametrize("Nx", [1, 2, 15, 16, 17, 31, 32, 33, 48, 65])
@pytest.mark.parametrize("Nt,beta", [(12, 9.0), (7, 8.0), (5, 8.25)])
def test_stratified_panel_edges(Nx, Nt, beta):
    """The Cholesky-QR sweep at the edges of its 16-column panels, with several slices per chunk, one slice per chunk within
    the first-order second pass, and one slice per chunk of a condition beyond it (exp(2 delta rho) = e^6.6): gradient and
    log det of both species against the dense inverse of M. Bar: relative perturbations of 256 eps of the slices (the
    rounding of a few hundred operations each) move M^-1 by 256 eps |M^-1|^2 |M| and log det M by n 256 eps |M^-1| |M|;
    1e-13 where that is smaller."""
    import nsl_gb300 as N

    eps = 256 * 2.0 ** -53
    lat = N.Ring(Nx)
    phi = _field(Nx, Nt, beta, 100 + Nx)
    for species in (0, 1):
        h = N.HubbardExp(lat, Nt, beta, 0.0, N.Species(species))
        h.set_stabilisation("stratified")
        h.populate(phi)
        ho = O.HubbardExp(lat.hopping_matrix(), Nt, beta, 0.0, species)
        ho.populate(phi)
        n = Nt * Nx
        Md = ho.M_dense().reshape(n, n)
        inv = np.linalg.inv(Md)
        nM, nI = np.linalg.norm(Md, 2), np.linalg.norm(inv, 2)
        want = 1j * np.diag(inv).reshape(Nt, Nx)
        err = np.abs(np.asarray(h.gradLogDetM()) - want).max()
        assert err <= max(1e-13 * np.abs(want).max(), eps * nI ** 2 * nM), (species, err)
        s, l = np.linalg.slogdet(Md)
        ref = complex(l, np.angle(s))
        assert abs(mod2pi(h.logDetM() - ref)) <= max(1e-13 * abs(ref), n * eps * nI * nM)


@pytest.mark.parametrize("mode", ["plain", "stratified"])
@pytest.mark.parametrize("Nx", [5, 32, 33, 72, 130])
def test_nan_field_stays_inside_the_matrices(Nx, mode):
    """A field with a NaN turns every matrix into NaN, and no pivot search finds a largest entry: log det and gradient are NaN
    too (or a reported error), and the handle's next evaluation is what a new handle gives."""
    import nsl_gb300 as N

    Nt, beta = 6, 3.0
    phi = _field(Nx, Nt, beta, Nx)
    bad = phi.copy()
    bad[2, Nx // 2] = np.nan

    def evaluate(h, f):
        h.populate(f)
        return h.logDetM(), np.asarray(h.gradLogDetM())

    h, fresh = N.HubbardExp(N.Ring(Nx), Nt, beta), N.HubbardExp(N.Ring(Nx), Nt, beta)
    for x in (h, fresh):
        x.set_stabilisation(mode)
    try:
        ld, g = evaluate(h, bad)
        assert not np.isfinite(ld) and not np.isfinite(g).any()
    except RuntimeError:
        pass
    (ld, g), (ld0, g0) = evaluate(h, phi), evaluate(fresh, phi)
    assert ld == ld0 and np.array_equal(g, g0)


@pytest.mark.parametrize("kind,a", [("im", 0.5), ("im", 2.0), ("im", 4.0), ("scale", 45.0), ("scale", -45.0),
                                    ("installed", 2.0), ("installed", 8.0), ("installed", 16.0)])
def test_stratified_beyond_the_first_order_second_pass(monkeypatch, kind, a):
    """Chunk products whose condition the lattice does not bound, one slice each (so that no wrap inside a chunk amplifies
    anything): Im phi of +-a per site (a condition of exp(2 a) and more), a common Im phi of a (entries of exp(+-a), out of
    FP32's range after the correction), and an installed exp(delta K) of a times the hopping (a condition of exp(a)). Gradient and
    log det of both species against the dense inverse of M, within the bar of test_stratified_panel_edges."""
    import nsl_gb300 as N

    monkeypatch.setenv("NSLG_STRAT_CHUNK", "1")
    eps = 256 * 2.0 ** -53
    Nx, Nt, beta = 24, 12, 3.0
    lat = N.Ring(Nx)
    rng = np.random.default_rng(31)
    phi = rng.standard_normal((Nt, Nx)) * np.sqrt(beta / Nt) + 0j
    if kind == "im":
        phi = phi + 1j * a * rng.choice((-1.0, 1.0), (Nt, Nx))
    elif kind == "scale":
        phi = phi + 1j * a * np.where(np.arange(Nt) % 2 == 0, 1.0, -1.0)[:, None]
    else:
        w, V = np.linalg.eigh(np.array(lat.hopping_matrix()).real)
        for s in (1, -1):
            lat.set_exp_hopping_matrix(s * beta / Nt, (V * np.exp(a * s * beta / Nt * w)) @ V.T + 0j)
    for species in (0, 1):
        h = N.HubbardExp(lat, Nt, beta, 0.0, N.Species(species))
        h.set_stabilisation("stratified")
        h.populate(phi)
        ho = O.HubbardExp(lat.hopping_matrix(), Nt, beta, 0.0, species)
        for s in (1, -1):
            ho.set_expK(s * beta / Nt, h.exp_hopping_matrix(s * beta / Nt))
        ho.populate(phi)
        n = Nt * Nx
        Md = ho.M_dense().reshape(n, n)
        inv = np.linalg.inv(Md)
        nM, nI = np.linalg.norm(Md, 2), np.linalg.norm(inv, 2)
        want = 1j * np.diag(inv).reshape(Nt, Nx)
        err = np.abs(np.asarray(h.gradLogDetM()) - want).max()
        assert err <= max(1e-13 * np.abs(want).max(), eps * nI ** 2 * nM), (species, err)
        s, l = np.linalg.slogdet(Md)  # (tr K = 0: an installed exp(delta K) has determinant 1 too)
        ref = complex(l, np.angle(s))
        assert abs(mod2pi(h.logDetM() - ref)) <= max(1e-13 * abs(ref), n * eps * nI * nM)


@pytest.mark.parametrize("chunk,a", [("1", 30.0), ("2", 20.0)])
def test_stratified_breakdown_is_an_error(monkeypatch, chunk, a):
    """Chunk products of condition exp(a k) > 1e8 leave their Gram matrix without a Cholesky factor: log det, gradient and a
    trajectory (eager and captured) report that instead of returning NaN, and the handle goes on with another matrix."""
    import nsl_gb300 as N
    from nsl_gb300.action import HubbardFermionAction, HubbardGaugeAction
    from nsl_gb300.integrator import Leapfrog

    monkeypatch.setenv("NSLG_STRAT_CHUNK", chunk)
    Nx, Nt, beta = 24, 12, 3.0
    lat = N.Ring(Nx)
    w, V = np.linalg.eigh(np.array(lat.hopping_matrix()).real)
    good = {s * beta / Nt: (V * np.exp(s * beta / Nt * w)) @ V.T + 0j for s in (1, -1)}
    bad = {s * beta / Nt: (V * np.exp(a * s * beta / Nt * w)) @ V.T + 0j for s in (1, -1)}
    phi = _field(Nx, Nt, beta, 4)
    params = {"Nt": Nt, "beta": beta, "U": 1.0}
    S = HubbardGaugeAction(params) + HubbardFermionAction(lat, params, stabilisation="stratified")
    h = S._mask_and_fm()[1]
    lf = Leapfrog(S, 0.2, 2)
    run = lambda: lf({"phi": phi}, {"phi": 0.1 * phi})
    for d, E in good.items():
        h.set_exp_hopping_matrix(d, E)
    h.populate(phi, N.Species.Particle)
    ld, g = h.logDetM(), np.asarray(h.gradLogDetM())
    q = [np.asarray(run()[0]["phi"]) for _ in range(3)]
    for d, E in bad.items():
        h.set_exp_hopping_matrix(d, E)
    h.populate(phi, N.Species.Particle)
    for f in (h.logDetM, h.gradLogDetM, lambda: S.eval(phi), lambda: S.force(phi), run, run, run):
        with pytest.raises(RuntimeError, match="ill-conditioned"):
            f()
    for d, E in good.items():
        h.set_exp_hopping_matrix(d, E)
    h.populate(phi, N.Species.Particle)
    assert h.logDetM() == ld and np.array_equal(np.asarray(h.gradLogDetM()), g)
    assert all(np.array_equal(np.asarray(run()[0]["phi"]), v) for v in q)
