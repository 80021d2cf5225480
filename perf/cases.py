"""The work that users of this package have it do, for timing and comparing.

A pass takes a state in the reference's host layout onto the device, advances
it and reads the result back, the way a host program does between two of its
diagnostics (or, with one step a pass, the way the drop-in ``step_ch()`` does
at every step).  Every pass starts from the prepared state, so it can be
repeated.  Sizes and options are those of the package's own configurations:
the 64^2 to 1024^2 torus, the 512 x 256 force-free dipole, the ensemble of
uneven tori, the 256^2 adjoint and the con-to-prim entry.
"""
import functools
import math

import numpy as np

import harm_ramt_b200 as hb
from harm_ramt_b200 import ensemble

# What one RK2 step of a zone cannot do without: the state and the geometry
# tables moved once per substep (FP64, and with FP32 faces), and the
# arithmetic of both substeps' faces, sources and inversions.
STEP_BYTES = {"fp64": 2032.0, "mixed": 1696.0}
STEP_FLOPS = 8000.0
ZONE_BYTES = 8 * hb.NPR

LIMITERS = {"mc": hb.LIM_MC, "para": hb.LIM_PARA}
SOLVERS = {"hll": hb.FLUX_HLL, "laxf": hb.FLUX_LAXF}
PRECISIONS = {"fp64": hb.PREC_FP64, "mixed": hb.PREC_MIXED}


def _torus(n1, n2, steps, develop, lim="para", flux="hll", precision="fp64", switch=0, currents=False, tryagain=False):
    return dict(kind="torus", n1=n1, n2=n2, steps=steps, develop=develop, lim=lim, flux=flux, precision=precision,
                switch=switch, currents=currents, tryagain=tryagain)


def listed():
    return [
        # the drop-in step of a small torus: one step per call, bound by launches and copies
        dict(_torus(64, 64, 1, 200, lim="mc"), name="shim_64"),
        # a resolution study's small run between two diagnostics
        dict(_torus(128, 128, 50, 300, lim="mc"), name="torus_128"),
        # the benchmark torus: PPM, HLL with the per-zone switch
        dict(_torus(512, 512, 20, 400, switch=3), name="torus_512"),
        # the same torus behind the drop-in step, its state crossing the link every step
        dict(_torus(512, 512, 1, 400, switch=3), name="shim_512"),
        # the production grid
        dict(_torus(1024, 1024, 10, 200, switch=3), name="torus_1024"),
        # the benchmark torus with FP32 faces
        dict(_torus(512, 512, 20, 400, switch=3, precision="mixed"), name="torus_512_mixed"),
        # an odd grid with the reference's default inversions (retry chain) and its diagnostic currents
        dict(_torus(245, 131, 40, 200, flux="laxf", currents=True, tryagain=True), name="torus_245x131_currents"),
        # the force-free rotator, FP64 and with FP32 faces
        dict(kind="dipole", n1=512, n2=256, steps=20, develop=200, lim="mc", flux="laxf", precision="fp64",
             name="dipole_512x256"),
        dict(kind="dipole", n1=512, n2=256, steps=20, develop=200, lim="mc", flux="laxf", precision="mixed",
             name="dipole_512x256_mixed"),
        # a parameter survey: uneven tori side by side
        dict(kind="ensemble", members=16, grids=7, steps=20, per_launch=10, develop=50, lim="para", flux="hll",
             precision="fp64", name="ensemble_16"),
        # the gradient of a run of the 256^2 torus, two checkpoint segments
        dict(kind="adjoint", n1=256, n2=256, steps=32, checkpoint=16, develop=300, lim="mc", flux="hll",
             name="adjoint_256"),
        # con-to-prim on its own, at the zones of a state of the user's
        dict(kind="invert", n1=256, n2=256, zones=50000, name="invert_50000"),
    ]


def _size(rng, lo, hi):
    """Log-uniform in [lo, hi], odd as often as even."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["torus", "torus", "torus", "dipole", "ensemble", "adjoint", "invert"])
    lim, flux = rng.choice(["mc", "para"]), rng.choice(["hll", "laxf"])
    if kind == "adjoint":
        return dict(kind=kind, n1=_size(rng, 40, 256), n2=_size(rng, 40, 256), steps=rng.randint(6, 32),
                    checkpoint=rng.choice([4, 8, 16]), develop=100, lim=lim, flux=flux)
    if kind == "invert":
        return dict(kind=kind, n1=_size(rng, 40, 256), n2=_size(rng, 40, 256), zones=_size(rng, 100, 50000))
    if kind == "ensemble":
        per_launch = rng.choice([1, 2, 5])
        return dict(kind=kind, members=rng.randint(2, 16), grids=rng.randint(0, 9999),
                    steps=per_launch * rng.randint(1, 4), per_launch=per_launch, develop=50, lim=lim, flux=flux, precision=rng.choice(["fp64", "mixed"]))
    n1, n2 = _size(rng, 48, 1024), _size(rng, 48, 1024)
    steps = max(1, min(50, int(10 * 1024 * 1024 / (n1 * n2)))) if rng.random() < 0.7 else 1
    precision = rng.choice(["fp64", "fp64", "mixed"])
    if kind == "dipole":
        n1, n2 = min(n1, 768), min(n2, 512)
        return dict(kind=kind, n1=n1, n2=n2, steps=steps, develop=100, lim=lim, flux=flux, precision=precision)
    currents = n1 * n2 < 300 * 300 and rng.random() < 0.3
    return _torus(n1, n2, steps, 150, lim, flux, precision, rng.choice([0, 3]), currents, rng.random() < 0.3)


# The metric tables depend on the grid alone; a program that makes many runs
# of one grid keeps them.
@functools.lru_cache(maxsize=4)
def _torus_grid(n1, n2):
    return hb.torus_geometry(hb.torus_params(n1, n2))


def _torus_start(n1, n2, seed):
    """The torus with the seed's own 4% perturbation of the internal energy."""
    par, geom = hb.torus_params(n1, n2, seed=1 + seed % 30000), _torus_grid(n1, n2)
    return par, geom, hb.torus_init(par, geom)


def _context(case, par, geom, precision="fp64", **kw):
    h = hb.HarmGPU(case["n1"], case["n2"], geom["dx1"], geom["dx2"], lim=LIMITERS[case["lim"]],
                   fluxmethod=SOLVERS[case["flux"]], gam=par.gam, gammamax=par.gammamax,
                   precision=PRECISIONS[precision], **kw)
    h.upload_geometry(*(geom[k] for k in ("gcov", "gcon", "gdet", "conn", "floors")))
    return h


def _develop(h, p0, steps):
    """A developed flow from the initial state: prims, pflag, time and dt."""
    h.set_prims(p0)
    h.bound_prims()
    h.set_time(0.0, 1.0e-5, 0)
    h.step_ch(steps)
    st = h.sync()
    return (*h.get_prims(), st["t"], st["dt"])


def _buffers(h):
    """Page-locked host arrays for the state and its flags."""
    return hb.pinned_empty((h.n1m, h.n2m, hb.NPR)), hb.pinned_empty((h.n1m, h.n2m, 5), np.int32)


def _prepare_run(case, seed):
    if case["kind"] == "torus":
        par, geom, p0 = _torus_start(case["n1"], case["n2"], seed)
        opt = dict(fluxadjust=case["switch"], currents=case["currents"], tryagain=case["tryagain"])
    else:
        r = np.random.default_rng(seed)
        par = hb.dipole_params(case["n1"], case["n2"], bpole=float(r.uniform(0.8, 1.2)),
                               omegastar=float(r.uniform(0.15, 0.25)))
        geom = hb.dipole_geometry(par)
        p0 = hb.dipole_init(par, geom)
        opt = dict(eom=hb.EOM_FFDE, bc=hb.BC_STAR, omegastar=par.omegastar)
    first = _context(case, par, geom, **opt)
    p, f, t, dt = _develop(first, p0, case["develop"])
    h = first
    if case["precision"] != "fp64":
        first.close()
        h = _context(case, par, geom, case["precision"], **opt)
    pin, out = _buffers(h), _buffers(h)
    pin[0][...], pin[1][...] = p, f
    return dict(case=case, h=h, pin=pin, out=out, t=t, dt=dt, step=case["develop"])


def _prepare_ensemble(case, seed):
    # the case's grids, each with the seed's own black hole and torus
    specs = [dict(drawn, n1=grid["n1"], n2=grid["n2"]) for grid, drawn in
             zip(ensemble.sample_tori(case["members"], case["grids"]), ensemble.sample_tori(case["members"], seed))]
    made = ensemble.build(hb, specs, lim=LIMITERS[case["lim"]], fluxmethod=SOLVERS[case["flux"]],
                          precision=PRECISIONS[case["precision"]])
    members = [h for h, _ in made]
    e = hb.Ensemble(members, steps_per_launch=case["per_launch"])
    e.step(case["develop"])
    start = [(*h.get_prims(), st["t"], st["dt"]) for h, st in zip(members, e.sync())]
    return dict(case=case, members=members, ensemble=e, start=start, out=[_buffers(h) for h in members])


def _prepare_adjoint(case, seed):
    par, geom, p0 = _torus_start(case["n1"], case["n2"], seed)
    h = _context(case, par, geom)
    p, f, t, dt = _develop(h, p0, case["develop"])
    lam = np.zeros_like(p)
    r = np.random.default_rng(seed)
    lam[hb.NG:-hb.NG, hb.NG:-hb.NG] = r.standard_normal((case["n1"], case["n2"], hb.NPR))
    return dict(case=case, h=h, p=p, f=f, t=t, dt=dt, lam=lam)


def _u_of_p(p, gcov, gcon, g, gam):
    """The evolved conserved vector U(p) at zone centres (momenta with the
    rest-mass flux added to the energy, all times sqrt(-g))."""
    rho, u, util, B = p[:, 0], p[:, 1], p[:, 2:5], p[:, 5:8]
    alpha = 1.0 / np.sqrt(-gcon[:, 0, 0])
    gamma = np.sqrt(1.0 + np.einsum("zi,zij,zj->z", util, gcov[:, 1:, 1:], util))
    ucon = np.empty((len(p), 4))
    ucon[:, 0] = gamma / alpha
    ucon[:, 1:] = util - (gamma * alpha)[:, None] * gcon[:, 0, 1:]
    ucov = np.einsum("zij,zj->zi", gcov, ucon)
    bcon = np.empty_like(ucon)
    bcon[:, 0] = np.einsum("zi,zi->z", B, ucov[:, 1:])
    bcon[:, 1:] = (B + bcon[:, :1] * ucon[:, 1:]) / ucon[:, :1]
    bcov = np.einsum("zij,zj->zi", gcov, bcon)
    bsq = np.einsum("zi,zi->z", bcon, bcov)
    w = rho + gam * u + bsq
    U = np.empty_like(p)
    U[:, 0] = rho * ucon[:, 0]
    U[:, 1:5] = (w * ucon[:, 0])[:, None] * ucov - bcon[:, :1] * bcov
    U[:, 1] += (gam - 1.0) * u + 0.5 * bsq + U[:, 0]
    U[:, 5:8] = B
    return U * g[:, None]


def _states(case, seed):
    """Primitive states at random zones of the torus grid: the range of
    densities, internal energies, Lorentz factors and magnetisations of a
    developed flow, and guesses a step away from them."""
    r = np.random.default_rng(seed)
    par, geom = hb.torus_params(case["n1"], case["n2"]), _torus_grid(case["n1"], case["n2"])
    n = case["zones"]
    zones = np.stack([r.integers(0, case["n1"], n), r.integers(0, case["n2"], n)], axis=1).astype(np.int32)
    at = (zones[:, 0] + hb.NG, zones[:, 1] + hb.NG, 3)
    gcov, gcon, g = geom["gcov"][at], geom["gcon"][at], geom["gdet"][at]
    p = np.empty((n, hb.NPR))
    p[:, 0] = 10.0 ** r.uniform(-4, 0, n)
    p[:, 1] = p[:, 0] * 10.0 ** r.uniform(-2.5, -0.5, n)
    unit = r.standard_normal((n, 3))
    unit /= np.sqrt(np.einsum("zi,zij,zj->z", unit, gcov[:, 1:, 1:], unit))[:, None]
    p[:, 2:5] = unit * r.uniform(0.0, 1.5, n)[:, None]
    unit = r.standard_normal((n, 3))
    unit /= np.sqrt(np.einsum("zi,zij,zj->z", unit, gcov[:, 1:, 1:], unit))[:, None]
    p[:, 5:8] = unit * np.sqrt(2 * (par.gam - 1) * p[:, 1] / 10.0 ** r.uniform(0, 3, n))[:, None]
    guess = p * (1.0 + 0.02 * r.uniform(-1, 1, p.shape))
    return par, geom, zones, _u_of_p(p, gcov, gcon, g, par.gam), guess, p


def _prepare_invert(case, seed):
    par, geom, zones, U, guess, _ = _states(case, seed)
    h = _context(dict(case, lim="mc", flux="hll"), par, geom)
    return dict(case=case, h=h, zones=zones, U=U, guess=guess)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        return _prepare_ensemble(case, seed)
    if kind == "adjoint":
        return _prepare_adjoint(case, seed)
    if kind == "invert":
        return _prepare_invert(case, seed)
    return _prepare_run(case, seed)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "ensemble":
        for h, (p, f, t, dt) in zip(s["members"], s["start"]):
            h.set_prims(p, f)
            h.set_time(t, dt, case["develop"])
        s["ensemble"].step(case["steps"])
        status = s["ensemble"].sync()
        return [(*h.get_prims(out=o), st["t"], st["dt"]) for h, o, st in zip(s["members"], s["out"], status)]
    h = s["h"]
    if kind == "invert":
        return h.invert_zones(hb.INV_2D, s["zones"], s["U"], s["guess"])
    if kind == "adjoint":
        h.set_prims(s["p"], s["f"])
        h.set_time(s["t"], s["dt"], case["develop"])
        J, grad, dts, _ = h.adjoint(case["steps"], case["checkpoint"], w_mass=1.0, w_em=1.0, lam_final=s["lam"])
        return J, grad, dts
    h.set_prims(*s["pin"])
    h.set_time(s["t"], s["dt"], s["step"])
    h.step_ch(case["steps"])
    st = h.sync()
    p, f = h.get_prims(out=s["out"])
    out = dict(prims=p, flags=f, t=st["t"], dt=st["dt"])
    if case.get("currents"):
        out["jcon"], out["fcon"], _ = h.get_currents()
    return out


def work(case):
    kind = case["kind"]
    if kind == "invert":
        # U and the guess in, the primitives and the flag out, the zone's metric; a few Newton iterations
        return dict(bytes=case["zones"] * (3.0 * ZONE_BYTES + 12 + 21 * 8), flops=case["zones"] * 800.0)
    if kind == "ensemble":
        zones = float(sum(t["n1"] * t["n2"] for t in ensemble.sample_tori(case["members"], case["grids"])))
    else:
        zones = float(case["n1"] * case["n2"])
    if kind == "adjoint":
        # the forward run, its values again and their adjoint, each with the geometry; lambda in, the gradient out
        return dict(bytes=zones * (3 * STEP_BYTES["fp64"] * case["steps"] + 3 * ZONE_BYTES),
                    flops=zones * 4 * STEP_FLOPS * case["steps"])
    # the state and the flags cross the link once each way
    return dict(bytes=zones * (STEP_BYTES[case["precision"]] * case["steps"] + 2 * (ZONE_BYTES + 20)),
                flops=zones * STEP_FLOPS * case["steps"])


def exact(case, seed):
    """The inversion's value is the state its U was made from.  A step has no
    short form in plain numpy (it is the whole flow update with its ordered
    repairs, over many steps, and the gradient of that), so the other cases
    give none."""
    if case["kind"] != "invert":
        return None
    return _states(case, seed)[-1], None
