"""GPU parity of the fermion-matrix applications against the reference (golden fixtures) and the oracle.

FP64 bar: 1e-12 max-norm relative error (the reference's own M tests use digits10, test_fermionMatrixHubbardExp.cpp).
FP32 inner operator bar: 1e-5 relative (single-precision products over Nx terms).
"""
import numpy as np
import pytest

from conftest import GOLDEN_CASES, load_golden, rel_err

pytestmark = pytest.mark.gpu

OPS = (("M", "M"), ("Mdagger", "Mdag"), ("MMdagger", "MMdag"), ("MdaggerM", "MdagM"))


def make_lattice(g):
    from nsl_gb300.lattice import Honeycomb, Ring

    spec = g["lattice_spec"]
    return Ring(int(spec[1])) if spec[0] == "ring" else Honeycomb((int(spec[1]), int(spec[2])))


@pytest.mark.parametrize("name", GOLDEN_CASES)
@pytest.mark.parametrize("species,tag", [(0, "P"), (1, "H")])
def test_operators_vs_reference(name, species, tag):
    import nsl_gb300 as N

    g = load_golden(name)
    hfm = N.HubbardExp(make_lattice(g), g["Nt"], g["beta"], g["mu"])
    hfm.populate(g["phi"], N.Species(species))
    for fn, key in OPS:
        out = getattr(hfm, fn)(g["psi"])
        assert rel_err(out, g[f"{key}_{tag}"]) < 1e-12, fn


@pytest.mark.parametrize("name", GOLDEN_CASES)
def test_exp_hopping_matrix_vs_reference(name):
    import nsl_gb300 as N

    g = load_golden(name)
    hfm = N.HubbardExp(make_lattice(g), g["Nt"], g["beta"], g["mu"])
    d = g["beta"] / g["Nt"]
    assert rel_err(hfm.exp_hopping_matrix(d), g["expK_pos"]) < 1e-13
    assert rel_err(hfm.exp_hopping_matrix(-d), g["expK_neg"]) < 1e-13


def test_installed_reference_exp_matches():
    """With the reference's own exp(delta K) installed (its memo entry), results agree to rounding."""
    import nsl_gb300 as N

    g = load_golden("honey3x3_nt16")
    lat = make_lattice(g)
    d = g["beta"] / g["Nt"]
    lat.set_exp_hopping_matrix(d, g["expK_pos"])
    hfm = N.HubbardExp(lat, g["Nt"], g["beta"], g["mu"])
    hfm.populate(g["phi"])
    assert rel_err(hfm.M(g["psi"]), g["M_P"]) < 1e-14


def test_torch_cuda_tensors_and_batch_dims():
    import torch

    import nsl_gb300 as N
    from oracle import nsl_oracle as O

    g = load_golden("honey6x6_nt32_beta8")
    hfm = N.HubbardExp(make_lattice(g), g["Nt"], g["beta"])
    phi = torch.from_numpy(g["phi"]).cuda()
    hfm.populate(phi)
    rng = np.random.default_rng(3)
    psi = rng.standard_normal((2, 3, g["Nt"], g["Nx"])) + 1j * rng.standard_normal((2, 3, g["Nt"], g["Nx"]))
    out = hfm.MMdagger(torch.from_numpy(psi).cuda())
    assert out.is_cuda and tuple(out.shape) == psi.shape
    h = O.HubbardExp(g["hops"], g["Nt"], g["beta"])
    h.populate(g["phi"])
    assert rel_err(out.cpu().numpy(), h.MMdagger(psi)) < 1e-12


@pytest.mark.parametrize("L,Nt,beta,R", [((12, 12), 64, 8.0, 4), ((8, 8), 16, 2.0, 7), ((5, 5), 33, 3.0, 3),
                                         ((24, 24), 128, 12.0, 1)])
def test_operators_vs_oracle_larger(L, Nt, beta, R):
    """Larger and ragged shapes (Nx, Nt*R not multiples of the tile) against the oracle, up to the honeycomb 24x24,
    Nt = 128, beta = 12 configuration (Nx = 1152)."""
    import nsl_gb300 as N
    from oracle import nsl_oracle as O

    lat = N.Honeycomb(L)
    rng = np.random.default_rng(7)
    Nx = lat.sites()
    phi = rng.standard_normal((Nt, Nx)) * np.sqrt(beta / Nt * 3.0) + 0j
    psi = rng.standard_normal((R, Nt, Nx)) + 1j * rng.standard_normal((R, Nt, Nx))
    hfm = N.HubbardExp(lat, Nt, beta)
    hfm.populate(phi)
    h = O.HubbardExp(lat.hopping_matrix(), Nt, beta)
    h.populate(phi)
    for fn, _ in OPS:
        assert rel_err(getattr(hfm, fn)(psi), getattr(h, fn)(psi)) < 1e-12, fn
        assert rel_err(getattr(hfm, fn)(psi, precision="fp32"), getattr(h, fn)(psi)) < 2e-5, fn


def test_complex_hopping_matrix():
    """Complex kappa (ring with a twist) -> complex exp(delta K): the complex-by-complex product path."""
    import nsl_gb300 as N
    from oracle import nsl_oracle as O

    lat = N.Ring(10, kappa=np.exp(0.3j))
    rng = np.random.default_rng(9)
    phi = rng.random((12, 10)) + 1j * rng.random((12, 10))
    psi = rng.standard_normal((2, 12, 10)) + 1j * rng.standard_normal((2, 12, 10))
    hfm = N.HubbardExp(lat, 12, 1.5, 0.1)
    hfm.populate(phi)
    h = O.HubbardExp(lat.hopping_matrix(), 12, 1.5, 0.1)
    h.populate(phi)
    for fn, _ in OPS:
        assert rel_err(getattr(hfm, fn)(psi), getattr(h, fn)(psi)) < 1e-12, fn


def test_batched_equals_single():
    """test_fermionMatrixHubbardExp.cpp:362-468: a batch equals its slices applied one by one."""
    import nsl_gb300 as N

    lat = N.Ring(8)
    rng = np.random.default_rng(11)
    phi = rng.random((10, 8)) + 0j
    psi = rng.random((10, 10, 8)) + 1j * rng.random((10, 10, 8))
    hfm = N.HubbardExp(lat, 10, 2.0)
    hfm.populate(phi)
    for fn, _ in OPS:
        full = getattr(hfm, fn)(psi)
        for n in range(10):
            assert np.array_equal(full[n], getattr(hfm, fn)(psi[n])), fn


def test_errors_are_reported():
    import nsl_gb300 as N
    from nsl_gb300._lib import NslgError

    lat = N.Ring(4)
    hfm = N.HubbardExp(lat, 4, 1.0)
    with pytest.raises(NslgError):
        hfm.M(np.zeros((4, 4), dtype=np.complex128))  # not populated
    hfm.populate(np.zeros((4, 4)))
    with pytest.raises(ValueError):
        hfm.M(np.zeros((3, 4), dtype=np.complex128))
    empty = hfm.M(np.zeros((0, 4, 4), dtype=np.complex128))
    assert empty.shape == (0, 4, 4)


@pytest.mark.parametrize("L,Nt,R", [((12, 12), 64, 4), ((3, 3), 16, 3), ((5, 5), 33, 2), ((2, 2), 8, 5),
                                    ((24, 24), 16, 1), ((8, 8), 12, 3)])
def test_split_bf16_operator(L, Nt, R):
    """Exact-accumulation split-BF16 tensor-core operator: FP64-class. Six balanced 9-bit digits carry 53 bits per
    operand, rounded to nearest, so the product's error is that of an FP64 product (~1e-15 of the output's maximum;
    bar 2e-14 against the oracle and against the device's FP64 operator, vs 2e-5 for the FP32-class operators);
    ragged tiles and K > 1024 (Nx = 1152) included."""
    import nsl_gb300 as N
    from oracle import nsl_oracle as O

    beta = 4.0
    lat = N.Honeycomb(L)
    Nx = lat.sites()
    rng = np.random.default_rng(23)
    phi = rng.standard_normal((Nt, Nx)) * np.sqrt(beta / Nt * 3.0) + 0j
    psi = rng.standard_normal((R, Nt, Nx)) + 1j * rng.standard_normal((R, Nt, Nx))
    hfm = N.HubbardExp(lat, Nt, beta)
    hfm.populate(phi)
    h = O.HubbardExp(lat.hopping_matrix(), Nt, beta)
    h.populate(phi)
    for fn, _ in OPS:
        got = getattr(hfm, fn)(psi, precision="bf16split")
        assert rel_err(got, getattr(h, fn)(psi)) < 2e-14, fn
        assert rel_err(got, getattr(hfm, fn)(psi, precision="fp64")) < 2e-14, fn


def test_split_bf16_digit_bound_refuses_delocalised_exp():
    """exp(delta K) at delta = 4 on honeycomb 12x12 is delocalised: its digit sums can exceed FP32's exact range for
    some operand, so the split-BF16 operator reports an error instead of an inexact result (the FP64 operator still
    runs)."""
    import nsl_gb300 as N

    lat = N.Honeycomb((12, 12))
    Nt, beta = 2, 8.0
    Nx = lat.sites()
    rng = np.random.default_rng(5)
    hfm = N.HubbardExp(lat, Nt, beta)
    hfm.populate(rng.standard_normal((Nt, Nx)) * 0.1 + 0j)
    psi = rng.standard_normal((1, Nt, Nx)) + 0j
    with pytest.raises(RuntimeError, match="delocalised"):
        hfm.M(psi, precision="bf16split")
    hfm.M(psi, precision="fp64")


@pytest.mark.parametrize("Nx", [1, 2, 31, 33, 64, 65, 127, 255, 256, 257, 320])
@pytest.mark.parametrize("Nt,R", [(1, 1), (3, 2), (7, 5), (64, 6)])
def test_cuda_core_operator_splits(Nx, Nt, R):
    """The CUDA-core operators at the edges of their work split (whole rows up to 256 sites, runs of sites beyond; 1 to 8
    rows per thread), with a real and a complex, non-symmetric exp(delta K), against the same formula in numpy. A sum of
    Nx complex products in any order, its factors rounded once, is within 4 (Nx + 8) eps of the sum of their moduli."""
    import nsl_gb300 as N

    rng = np.random.default_rng(100 * Nx + Nt)
    phi = rng.standard_normal((Nt, Nx)) + 0.3j * rng.standard_normal((Nt, Nx))
    psi = rng.standard_normal((R, Nt, Nx)) + 1j * rng.standard_normal((R, Nt, Nx))
    ph = np.exp(1j * phi)
    sign = np.where(np.arange(Nt) == 0, -1.0, 1.0)[:, None]
    for E in (rng.standard_normal((Nx, Nx)) + 0j, rng.standard_normal((Nx, Nx)) + 1j * rng.standard_normal((Nx, Nx))):
        lat = N.Ring(Nx)
        lat.set_exp_hopping_matrix(0.125, E)
        fm = N.HubbardExp(lat, Nt, 0.125 * Nt)
        fm.populate(phi)
        wantM = psi - sign * np.roll((ph * psi) @ E.T, 1, 1)
        sizeM = np.abs(psi) + np.roll(np.abs(ph * psi) @ np.abs(E).T, 1, 1)
        wantD = psi - np.conj(ph) * np.roll(sign * (psi @ E.T), -1, 1)
        sizeD = np.abs(psi) + np.abs(ph) * np.roll(np.abs(psi) @ np.abs(E).T, -1, 1)
        for prec, eps in (("fp64", 2.0 ** -53), ("fp32", 2.0 ** -24)):
            for op, want, size in (("M", wantM, sizeM), ("Mdagger", wantD, sizeD)):
                err = np.abs(getattr(fm, op)(psi, precision=prec) - want)
                assert np.all(err <= 4 * (Nx + 8) * eps * size), (prec, op, (err / size).max())


@pytest.mark.parametrize("Nx", [1, 16, 17, 32, 33, 63, 96, 145, 320])
@pytest.mark.parametrize("kind", ["identity", "banded", "far", "zero_row", "dense"])
def test_split_operator_skips_zero_digits(Nx, kind):
    """The split-BF16 operator with exp(delta K) whose digit blocks are mostly empty: the identity, a narrow band, a band
    plus entries in far k-blocks that only low digits represent, a zero row, and a dense one. Bound: operands rounded to
    2^-53 of their row's maximum and the dropped orders, 32 Nx 2^-53 max|E| max|Y| per row. A matrix beyond the
    digit-sum bound (the dense one at 320 sites) is refused."""
    import nsl_gb300 as N
    from test_split_digits import bounds_ok, digit_sum_bounds

    Nt, R = 5, 3
    rng = np.random.default_rng(Nx)
    i, j = np.arange(Nx)[:, None], np.arange(Nx)[None, :]
    E = np.eye(Nx)
    if kind == "banded":
        E = np.exp(-3.0 * np.abs(i - j)) * (np.abs(i - j) < 6)
    elif kind == "far":
        E = E + 2.0 ** -40 * (np.abs(i - j) > Nx // 2) + 2.0 ** -20 * (np.abs(i - j) == 3)
    elif kind == "zero_row":
        E[Nx // 2] = 0.0
    elif kind == "dense":
        E = rng.uniform(-1, 1, (Nx, Nx)) / Nx + E
    lat = N.Ring(Nx)
    lat.set_exp_hopping_matrix(0.125, E)
    fm = N.HubbardExp(lat, Nt, 0.125 * Nt)
    phi = rng.standard_normal((Nt, Nx)) + 0j
    psi = (rng.standard_normal((R, Nt, Nx)) + 1j * rng.standard_normal((R, Nt, Nx))) * np.exp(rng.uniform(-9, 9, (R, Nt, 1)))
    fm.populate(phi)
    ph = np.exp(1j * phi)
    sign = np.where(np.arange(Nt) == 0, -1.0, 1.0)[:, None]
    if not bounds_ok(digit_sum_bounds(E)):
        with pytest.raises(RuntimeError, match="delocalised"):
            fm.M(psi, precision="bf16split")
            fm.ctx.synchronize()
        return
    eps = 32 * Nx * 2.0 ** -53 * np.abs(E).max()
    for op, want, row in (("M", psi - sign * np.roll((ph * psi) @ E.T, 1, 1), np.roll(np.abs(psi).max(2), 1, 1)),
                          ("Mdagger", psi - np.conj(ph) * np.roll(sign * (psi @ E.T), -1, 1),
                           np.roll(np.abs(psi).max(2), -1, 1))):
        err = np.abs(getattr(fm, op)(psi, precision="bf16split") - want).max(2)
        assert np.all(err <= eps * row + 2.0 ** -51 * np.abs(want).max(2)), (op, (err / row).max())


def test_replacing_exp_hopping_replaces_what_was_derived_from_it():
    """set_exp_hopping_matrix on a handle that has used the old exp(+-delta K) in every form (planes, 3xTF32 and digit planes,
    captured solves and trajectories): afterwards every call gives what a handle that never saw the old matrix gives, and a
    certified solve solves the new system."""
    import nsl_gb300 as N
    from nsl_gb300.action import HubbardFermionAction, HubbardGaugeAction
    from nsl_gb300.configuration import Configuration
    from nsl_gb300.integrator import Leapfrog
    from oracle import nsl_oracle as O
    from test_gpu_cg_dd import _same_operator

    Nt, beta, R = 32, 2.0, 4  # 2304 elements per right-hand side: past the resident kernel, 9216 in all for double-double
    rng = np.random.default_rng(8)
    w, V = np.linalg.eigh(np.array(N.Honeycomb((6, 6)).hopping_matrix()).real)
    new = {s * beta / Nt: (V * np.exp(0.9 * s * beta / Nt * w)) @ V.T + 0j for s in (1, -1)}

    def build(installed):
        lat = N.Honeycomb((6, 6))
        if installed:
            for d, E in new.items():
                lat.set_exp_hopping_matrix(d, E)
        params = {"Nt": Nt, "beta": beta, "U": 1.0}
        action = HubbardGaugeAction(params) + HubbardFermionAction(lat, params, force_precision="bf16split")
        return N.HubbardExp(lat, Nt, beta), Leapfrog(action, 1.0, 2)

    phi = (rng.standard_normal((Nt, 72)) * np.sqrt(beta / Nt)).astype(np.complex128)
    mom = rng.standard_normal((Nt, 72)).astype(np.complex128)
    b = rng.standard_normal((R, Nt, 72)) + 1j * rng.standard_normal((R, Nt, 72))
    eps = 1e-12 * np.linalg.norm(b[0])

    def use(fm, lf):
        fm.populate(phi, N.Species.Particle)
        out = [getattr(fm, op)(b, precision=p) for op in ("M", "MMdagger") for p in ("fp64", "fp32", "tf32x3", "bf16split")]
        out += list(fm.apply_dd(N.MatrixCombination.MMdagger, b))
        for p in ("bf16split", "tf32x3"):
            cg = N.CG(fm, N.MatrixCombination.MMdagger, eps, 20000, mode="per_rhs", precision=p, stop="true_residual_dd")
            out += [cg(b), cg.x_lo_]
            assert cg.stats["converged"] == R, (p, cg.stats)
        for _ in range(2):  # the second trajectory is captured
            q, p = lf(Configuration({"phi": phi}), Configuration({"phi": mom}))
        return out + [q["phi"], p["phi"]]

    fm, lf = build(False)
    old = use(fm, lf)
    for h in (fm, lf.action_._mask_and_fm()[1]):
        for d, E in new.items():
            h.set_exp_hopping_matrix(d, E)
    got, want = use(fm, lf), use(*build(True))
    for k, (g, v, o) in enumerate(zip(got, want, old)):
        assert np.array_equal(g, v), (k, rel_err(g, v), rel_err(g, o))
    x, lo = got[10], got[11]
    ho = _same_operator(fm, phi)
    assert max(np.linalg.norm(O.residual_dd(ho, "MMdagger", b[r], x[r], lo[r])) for r in range(R)) <= 1.01 * eps


def test_operator_calls_from_several_threads_and_streams():
    """One handle, three threads, each with its own stream: an application reads its operand after the work queued on its caller's
    stream (here a copy behind a delay), and that stream's later work reads the result, whichever calls come between."""
    import threading

    import nsl_gb300 as N
    import torch

    fm = N.HubbardExp(N.Honeycomb((3, 3)), 16, 4.0)
    rng = np.random.default_rng(0)
    fm.populate(rng.standard_normal((16, 18)) + 0j)
    src = [torch.from_numpy(rng.standard_normal((40, 2, 16, 18)) + 1j * rng.standard_normal((40, 2, 16, 18))).cuda()
           for _ in range(3)]
    want = [torch.stack([fm.M(v) for v in s]).cpu() for s in src]
    got, errors = [None] * 3, []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                out = torch.zeros_like(src[k])
                psi = torch.zeros_like(src[k][0])
                for i in range(len(src[k])):
                    torch.cuda._sleep(20000)
                    psi.copy_(src[k][i])
                    out[i].copy_(fm.M(psi))
                torch.cuda.current_stream().synchronize()
                got[k] = out.cpu()
        except Exception as e:  # pragma: no cover
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert all(torch.equal(g, w) for g, w in zip(got, want))


@pytest.mark.parametrize("Nx,Nt,R", [(18, 16, 5), (72, 7, 9), (97, 5, 13), (288, 3, 11)])
def test_tf32_operator_row_sizes_and_non_finite_values(Nx, Nt, R):
    """The 3xTF32 operator on rows of sizes 2^-60 to 2^90, rows of zeros, values outside FP32's range, infinities and NaN. Scaling
    a row by a power of two scales its result exactly (the splits work on bit patterns); ordinary rows agree with FP64 to
    8 Nx 2^-21 of the sum of moduli. Where a row holds a value FP32 cannot (or an infinity, or a NaN), what it reaches is not
    finite, and nothing else changes."""
    import nsl_gb300 as N

    rng = np.random.default_rng(Nx)
    fm = N.HubbardExp(N.Ring(Nx), Nt, 0.1 * Nt)
    fm.populate(rng.standard_normal((Nt, Nx)) + 0j)
    E = np.abs(fm.exp_hopping_matrix(0.1))
    base = rng.standard_normal((R, Nt, Nx)) + 1j * rng.standard_normal((R, Nt, Nx))
    base[0] = 0.0
    base[1, Nt // 2] = 0.0
    # (r, t) reaches (r, t +- 1) and itself: one scale per right-hand side
    scale = 2.0 ** rng.integers(-60, 91, (R, 1, 1))
    psi, clean = base * scale, {}
    for op, shift in (("M", 1), ("Mdagger", -1)):
        one = getattr(fm, op)(base, precision="tf32x3")
        terms = np.roll(np.abs(base) @ E.T, shift, 1)
        assert (np.abs(one - getattr(fm, op)(base)) <= 8 * Nx * 2.0 ** -21 * terms).all(), op
        clean[op] = getattr(fm, op)(psi, precision="tf32x3")
        assert np.array_equal(clean[op], one * scale), op
    for bad in (1e40, np.inf, -np.inf, np.nan):
        for part in (1.0, 1j):
            x = psi.copy()
            t, r = Nt - 1, R - 1
            x[r, t, Nx // 2] = bad * part if np.isfinite(bad) or part == 1.0 else complex(0.0, bad)
            for op, to in (("M", (t + 1) % Nt), ("Mdagger", t - 1)):
                got = getattr(fm, op)(x, precision="tf32x3")
                same = np.ones((R, Nt), bool)
                same[r, to] = same[r, t] = False
                assert np.array_equal(got[same], clean[op][same]), (bad, part, op)
                assert not np.isfinite(got[r, to]).any(), (bad, part, op)
                elsewhere = np.arange(Nx) != Nx // 2  # psi itself enters its own slice at that site alone
                assert np.array_equal(got[r, t, elsewhere], clean[op][r, t, elsewhere]), (bad, part, op)
