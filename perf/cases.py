"""The work this library is measured on: whole field solves through the public
Python API (the reference's class), batches, the serving loop and the pointwise
map, from toy fields to 20 000 stars.

A case is a dict of plain values; ``kind`` says which entry points it goes
through:

  field    one CCF: run(), then the critical curves, caustics and (on request)
           length scales in host arrays, as a script that plots or bins them
           has them.  ``stars`` = "given" hands the solver the caller's own
           star array with set_stars() before the run, as a simulation
           pipeline does.
  batch    run_batch() over many small fields, then each field's results.
  serving  a Server with four slots: all requests submitted, each waited for,
           read and released.
  map      eval_points() of a field that was solved before: f, f', the lens
           map, the 1/mu bound and the length scale at the caller's points.

The solver's 1/mu error bounds are not among a run's outputs here: they are
bounds on rounding, not results, and no output file of the reference holds
them.  Every run leaves them in the buffers beside the outputs.
"""
import math

import numpy as np

from ccf_gb300 import CCF, Server, derive_params, pinned_empty, run_batch

SALPETER = {"mass_function": "salpeter", "m_lower": 0.08, "m_upper": 1.5, "m_solar": 4.954984}
KROUPA = {"mass_function": "kroupa", "m_lower": 0.08, "m_upper": 1.5, "m_solar": 1.0}
EQUAL = {"mass_function": "equal"}

#: parameters of a case that go to CCF as they are
PARAMS = ("kappa_tot", "kappa_star", "shear", "mass_function", "m_lower", "m_upper", "m_solar", "rectangular", "approx",
          "num_stars", "num_phi", "num_branches", "write_mu_length_scales", "precision", "continuation")


def listed():
    return [
        # a first try at the command line or in a notebook: a dozen stars, the default phi grid; launches and
        # host round trips are all there is
        {"name": "toy_disc_n12", "kind": "field", "kappa_tot": 0.3, "kappa_star": 0.3, "shear": 0.1, **EQUAL,
         "num_stars": 12, "num_phi": 100, "num_branches": 1},
        # the class's own defaults (137 equal stars, a little smooth mass), as the reference's users start from
        {"name": "default_disc_n137", "kind": "field", "kappa_tot": 0.3, "kappa_star": 0.27, "shear": 0.3, **EQUAL,
         "num_stars": 137, "num_phi": 100, "num_branches": 1},
        # a caller's own catalogue with length scales for a caustic-crossing study: odd sizes, a rectangle
        {"name": "given_rect_n419_scales", "kind": "field", "stars": "given", "kappa_tot": 0.55, "kappa_star": 0.4,
         "shear": 0.25, **KROUPA, "rectangular": 1, "num_stars": 419, "num_phi": 420, "num_branches": 7,
         "write_mu_length_scales": 1},
        # the headline field of the benchmark
        {"name": "rect_n2000", "kind": "field", "kappa_tot": 0.45, "kappa_star": 0.35, "shear": 0.35, **SALPETER,
         "rectangular": 1, "num_stars": 2000, "num_phi": 2048, "num_branches": 32},
        # a field of a serving request: many stars, few branches, so that few centres are solved
        {"name": "disc_n7001_nb8", "kind": "field", "kappa_tot": 0.36, "kappa_star": 0.36, "shear": 0.22, **SALPETER,
         "num_stars": 7001, "num_phi": 1008, "num_branches": 8},
        # the large field of the benchmark on a coarser phi grid (its outputs in host arrays are 2 GB)
        {"name": "rect_n20000", "kind": "field", "kappa_tot": 0.7, "kappa_star": 0.6, "shear": 0.2, **KROUPA,
         "rectangular": 1, "num_stars": 20000, "num_phi": 1280, "num_branches": 32},
        # all arithmetic in FP64, for a check of a mixed run
        {"name": "fp64_rect_n600", "kind": "field", "kappa_tot": 0.45, "kappa_star": 0.35, "shear": 0.35, **SALPETER,
         "rectangular": 1, "num_stars": 600, "num_phi": 256, "num_branches": 8, "precision": "fp64"},
        # the reference's own continuation (the full Aberth step for every root)
        {"name": "aberth_disc_n400", "kind": "field", "kappa_tot": 0.3, "kappa_star": 0.3, "shear": 0.1, **EQUAL,
         "num_stars": 400, "num_phi": 128, "num_branches": 4, "continuation": "aberth"},
        # a parameter sweep: many small discs at once, as the benchmark's batch
        {"name": "batch_24_discs", "kind": "batch", "count": 24, "n_min": 50, "n_max": 1000, "num_phi": 512,
         "num_branches": 8},
        # the serving loop: requests of mixed sizes over four slots
        {"name": "serving_6_requests", "kind": "serving", "count": 6, "n_min": 100, "n_max": 4000, "num_phi": 1024,
         "num_branches": 8},
        # the map at many points of a solved field (source-plane grids, checks)
        {"name": "map_n500_20001_points", "kind": "map", "kappa_tot": 0.4, "shear": 0.2, "num_stars": 500,
         "num_points": 20001},
    ]


def _singular(kappa, shear):
    return abs(1 - kappa) < 0.05 or abs(1 - kappa - shear) < 0.05 or abs(1 - kappa + shear) < 0.05


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _convergence(rng, smooth):
    while True:
        ks = rng.uniform(0.1, 0.6)
        kt = ks / (1 - rng.uniform(0.05, 0.3)) if smooth else ks
        g = rng.uniform(0.02, 0.4)
        if not _singular(kt, g):
            return {"kappa_tot": kt, "kappa_star": ks, "shear": g}


def draw(rng):
    """One more case: small, ordinary and large fields, batches, serving and the map."""
    kind = rng.choice(["small", "small", "middle", "middle", "large", "fp64", "aberth", "batch", "serving", "map"])
    if kind == "batch":
        lo = rng.randint(30, 100)
        return {"kind": "batch", "count": rng.randint(6, 24), "n_min": lo, "n_max": rng.randint(lo + 50, 1000),
                "num_phi": 16 * rng.randint(12, 32), "num_branches": 8}
    if kind == "serving":
        nb = rng.choice([8, 32])
        return {"kind": "serving", "count": rng.randint(3, 6), "n_min": 100, "n_max": rng.randint(1000, 4000),
                "num_phi": 2 * nb * rng.randint(320 // nb, 1024 // nb), "num_branches": nb}
    if kind == "map":
        while True:
            kt, g = rng.uniform(0.1, 0.8), rng.uniform(0.0, 0.5)
            if not _singular(kt, g):
                return {"kind": "map", "kappa_tot": kt, "shear": g, "num_stars": _log_int(rng, 20, 1000),
                        "num_points": _log_int(rng, 100, 100000)}
    nb = {"small": rng.choice([1, 1, 2, 3, 4]), "middle": rng.choice([5, 8, 16, 32]), "large": rng.choice([8, 32]),
          "fp64": rng.choice([2, 4]), "aberth": rng.choice([2, 4])}[kind]
    lo, hi = {"small": (8, 400), "middle": (300, 4000), "large": (4000, 16000), "fp64": (50, 500), "aberth": (50, 400)}[kind]
    # phi steps of a branch's side; a large field's grid has about a thousand phases whatever its branches
    steps = {"small": (20, 100), "middle": (16, 48), "large": (384 // nb, 640 // nb), "fp64": (12, 24),
             "aberth": (10, 20)}[kind]
    rect = rng.random() < 0.5
    case = {"kind": "field", **_convergence(rng, rect), **rng.choice([EQUAL, SALPETER, KROUPA]),
            "rectangular": int(rect), "num_stars": _log_int(rng, lo, hi), "num_phi": 2 * nb * rng.randint(*steps),
            "num_branches": nb}
    if kind in ("small", "middle") and rng.random() < 0.3:
        case["write_mu_length_scales"] = 1
    if kind in ("small", "middle") and rng.random() < 0.3:
        case["stars"] = "given"
    if kind == "fp64":
        case["precision"] = "fp64"
    if kind == "aberth":
        case["continuation"] = "aberth"
    return case


def _star_seed(seed, i=0):
    return 1 + (seed * 9176 + i * 131) % 2000000000


def _given_stars(case, seed):
    """A caller's star field: uniform positions in the field's rectangle or
    disc, masses of a Salpeter-like power law with mean about one."""
    rng = np.random.default_rng(seed)
    n, ks = case["num_stars"], case["kappa_star"]
    m = (0.25 ** -1.35 + rng.random(n) * (8.0 ** -1.35 - 0.25 ** -1.35)) ** (-1 / 1.35)
    m /= m.mean()
    if case.get("rectangular"):
        ax = 1 / abs(1 - case["kappa_tot"] + case["shear"])
        ay = 1 / abs(1 - case["kappa_tot"] - case["shear"])
        half = math.sqrt(math.pi * n / (4 * ks))
        corner = complex(half * math.sqrt(ax / ay), half * math.sqrt(ay / ax))
        x, y = rng.uniform(-corner.real, corner.real, n), rng.uniform(-corner.imag, corner.imag, n)
    else:
        radius = math.sqrt(n / ks)
        corner = complex(radius, 0.0)
        r, t = radius * np.sqrt(rng.random(n)), rng.uniform(0, 2 * math.pi, n)
        x, y = r * np.cos(t), r * np.sin(t)
    return np.stack([x, y, m], axis=1), corner


def _params(case):
    return {k: case[k] for k in PARAMS if k in case}


def _field_sets(case, seed):
    """The parameter sets of a batch or of a request stream."""
    rng = np.random.default_rng(seed)
    out = []
    while len(out) < case["count"]:
        serving = case["kind"] == "serving"
        ks, g = float(rng.uniform(0.1, 0.6)), float(rng.uniform(0.0, 0.5))
        kt = ks if serving else ks / (1 - float(rng.uniform(0.0, 0.3)))
        if _singular(kt, g):
            continue
        lo, hi = case["n_min"], case["n_max"]
        # sizes spread evenly over the range (its logarithm for requests) whatever the seed, so that every seed
        # is as much work; the fields themselves come from the seed
        u = (len(out) + 0.5) / case["count"]
        n = int(round(lo * (hi / lo) ** u)) if serving else int(round(lo + (hi - lo) * u))
        out.append(dict(kappa_tot=kt, kappa_star=ks, shear=g, rectangular=0, num_stars=n, num_phi=case["num_phi"],
                        num_branches=case["num_branches"], random_seed=_star_seed(seed, len(out)),
                        **(SALPETER if serving else EQUAL)))
    return out


def _disc_radius(case):
    return math.sqrt(case["num_stars"] / 0.35)


def _map_inputs(case, seed):
    """Stars, points and phases of a map case: points all over the disc, a few
    outside the tree's root box."""
    stars, corner = _given_stars({**case, "kappa_star": 0.35}, seed)
    rng = np.random.default_rng([seed, 1])
    radius = _disc_radius(case)
    z = rng.uniform(-radius, radius, case["num_points"]) + 1j * rng.uniform(-radius, radius, case["num_points"])
    z[::97] *= 3
    return stars, corner, z, rng.uniform(0, 2 * math.pi, case["num_points"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return {"kind": kind, "fields": [CCF(**p) for p in _field_sets(case, seed)]}
    if kind == "serving":
        return {"kind": kind, "server": Server(slots=4, hbm_budget=60e9), "requests": _field_sets(case, seed)}
    if kind == "map":
        stars, corner, z, phi = _map_inputs(case, seed)
        c = CCF(kappa_tot=case["kappa_tot"], shear=case["shear"], num_phi=2, num_branches=1)
        c.set_stars(stars, 0, corner)
        if not c.run(-1):
            raise RuntimeError(c.last_error())
        return {"kind": kind, "ccf": c, "z": z, "phi": phi}
    c = CCF(random_seed=_star_seed(seed), **_params(case))
    state = {"kind": kind, "ccf": c, "given": None, "buffers": None}
    if case.get("stars") == "given":
        state["given"] = (*_given_stars(case, seed), case.get("rectangular", 0))
    else:
        # page-locked result arrays that the program keeps between runs
        roots = derive_params(**_params(case))["num_roots"]
        shape = (roots * c.num_branches, c.num_phi // c.num_branches + 1)
        state["buffers"] = {"ccs": pinned_empty(shape, np.complex128), "caustics": pinned_empty(shape, np.complex128),
                            "errs": pinned_empty(shape, np.float64)}
        if case.get("write_mu_length_scales"):
            state["buffers"]["mu_length_scales"] = pinned_empty(shape, np.float64)
    return state


def _outputs(r):
    return {k: r[k] for k in ("ccs", "caustics", "mu_length_scales") if r[k] is not None}


def run(state):
    kind = state["kind"]
    if kind == "batch":
        if not run_batch(state["fields"], -1):
            raise RuntimeError(state["fields"][0].last_error())
        return [_outputs(f.results(stars=False)) for f in state["fields"]]
    if kind == "serving":
        s = state["server"]
        ids = [s.submit(**p) for p in state["requests"]]
        out = []
        for i in ids:
            if s.wait(i) != 0:
                raise RuntimeError("request failed")
            out.append(_outputs(s.field(i).results(stars=False)))
            s.release(i)
        return out
    c = state["ccf"]
    if kind == "map":
        return c.eval_points(state["z"], state["phi"])
    if state["given"] is not None:
        stars, corner, rectangular = state["given"]
        c.set_stars(stars, rectangular, corner)
    if not c.run(-1):
        raise RuntimeError(c.last_error())
    return _outputs(c.results(stars=False, out=state["buffers"]))


def _field_work(p):
    """Bytes: the stars in, 16 bytes per root and caustic point out (8 per length scale).  Flops: one evaluation
    of f, f' and the lens map per point (40 per star of a leaf's near list of ~16, 16 per term of two expansions
    of order ~23: about 1000), and one pass of reciprocal sums over every root's pairs at one centre (10 each)."""
    n = p["num_stars"]
    roots = 2 * n + (60 if p.get("rectangular") else 0)
    points = roots * (p["num_phi"] + p["num_branches"])
    size = 40 if p.get("write_mu_length_scales") else 32
    return {"bytes": 24 * n + size * points, "flops": 1000 * points + 10 * roots * (roots + n)}


def work(case):
    kind = case["kind"]
    if kind == "map":
        # z, phi in; f, f', w, bound and scale out; the evaluation and the f' terms of a point
        return {"bytes": (24 + 64) * case["num_points"], "flops": 1400 * case["num_points"]}
    sets = _field_sets(case, 0) if kind in ("batch", "serving") else [_params(case)]
    each = [_field_work(p) for p in sets]
    return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}


def exact(case, seed):
    """The map's values by direct sums over every star in FP64.  The roots of a
    field have no such value: which root a row holds is the solver's choice, and
    f itself is the tree's expansion of order ~23."""
    if case["kind"] != "map":
        return None
    stars, corner, z, phi = _map_inputs(case, seed)
    zi, m = stars[:, 0] + 1j * stars[:, 1], stars[:, 2]
    kt, g, ks = case["kappa_tot"], case["shear"], m.sum() / abs(corner) ** 2
    a = 1 - kt + ks
    s = np.zeros((3, z.size), np.complex128)
    for i0 in range(0, z.size, 4096):
        inv = 1 / (z[i0:i0 + 4096, None] - zi[None, :])
        t = m * inv
        for k in range(3):
            s[k, i0:i0 + 4096] = t.sum(axis=1)
            t = t * inv
    f = g + s[1] - a * np.exp(-1j * phi)
    af = np.abs(f)
    dw = np.conj(g + s[1])
    cct = -2j * np.conj(dw) * np.conj(-2 * s[2])
    ct = a * cct + dw * np.conj(cct)
    return {"f": f, "df": -2 * s[2], "w": (1 - kt) * z + g * np.conj(z) - np.conj(s[0]) + ks * z,
            "err": np.maximum(np.abs(af * (af + 2 * a)), np.abs(af * (af - 2 * a))), "mu_length": 1 / (2 * np.abs(ct))}
