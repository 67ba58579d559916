"""The tracker's packed evaluator (two near stars and two polynomials side by
side) at the edges of its forms: odd and even near lists, one star, full and
nearly full lists (32 stars in one leaf), deeper trees, and the smooth-mass
forms with and without the series folded into the leaves.

Tracked columns are matched as sets against the full Aberth continuation,
whose evaluation is not packed: both converge each root to the zeros of one f
to a step below 1e-9 theta_star quadratically, so they agree within the 1e-11
theta_star of the other tracker tests (which compare the caustics too).  A run
that writes length scales takes the scalar evaluator; its roots are the packed
one's to the same tolerance.
"""
import numpy as np
import pytest

from ccf_gb300 import CCF, run_batch
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def run(cfg, **extra):
    c = CCF(**cfg, **extra)
    assert c.run(-1), c.last_error()
    return c.results()


@pytest.mark.parametrize("rectangular", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 15, 16, 31, 32, 33, 65, 301])
def test_packed_evaluator_finds_the_full_sum_zeros(n, rectangular):
    cfg = dict(kappa_tot=0.35, kappa_star=0.3, shear=0.15, mass_function="uniform", m_lower=0.5, m_upper=2.0,
               rectangular=rectangular, num_stars=n, num_phi=96, num_branches=2, random_seed=100 + n)
    t = run(cfg)
    a = run(cfg, continuation="aberth")
    m = run(cfg, write_mu_length_scales=1)
    assert t["info"]["unconverged"] == 0 and t["info"]["has_nan"] == 0
    for r in (a, m):
        d = O.match_sets(t["ccs"], r["ccs"], 2)
        assert d["non_finite"] == 0 and d["non_bijective_cols"] == 0
        assert d["max_dist"] <= 1e-11
    assert np.max(t["errs"]) <= 1e-9


@pytest.mark.parametrize("n, rectangular, num_phi, nb", [
    (4096, 1, 32, 2),     # the far launch from its smallest field on, roots that leave the box among the items
    (4501, 1, 24, 1),     # an odd number of stars, long rows
    (4501, 0, 24, 1),     # a disc: few roots off the box
    (150, 1, 24, 2),      # coarse steps: rows tracked again, their off-box roots handed over
    (17, 1, 40, 1),       # more solo roots than items
])
def test_roots_off_the_box_find_the_full_sum_zeros(n, rectangular, num_phi, nb):
    cfg = dict(kappa_tot=0.45, kappa_star=0.4, shear=0.3, mass_function="equal", rectangular=rectangular, num_stars=n,
               num_phi=num_phi, num_branches=nb, random_seed=7 + n)
    t = run(cfg)
    a = run(cfg, continuation="aberth")
    d = O.match_sets(t["ccs"], a["ccs"], nb)
    assert d["non_finite"] == 0 and d["non_bijective_cols"] == 0
    assert d["max_dist"] <= 1e-11


@pytest.mark.parametrize("precision, mu", [("fp64", 0), ("fp64", 1), ("mixed", 1)])
@pytest.mark.parametrize("n, rectangular, num_phi, nb", [
    (1, 0, 6, 1),         # fewer points than one warp
    (9, 0, 64, 2),        # rows of less than a CTA
    (33, 1, 94, 1),       # roots off the box, a ragged last warp
    (150, 1, 24, 2),      # coarse steps: rows tracked again and re-run
])
def test_outputs_formed_after_the_tracking(monkeypatch, n, rectangular, num_phi, nb, precision, mu):
    """The launch that forms FP64 outputs and length scales reaches every
    point: the caustics are the oracle's lens map of the stored roots (FP64 on
    both sides, the same tree and expansions: 1e-11 of the map's size, the
    multipole evaluation's rounding), and the same bits come out with the
    outputs in host memory and one group of centres at a time."""
    monkeypatch.setenv("CCF_GB300_CHUNK_BYTES", "1")
    field = dict(kappa_tot=0.45, kappa_star=0.4, shear=0.3, mass_function="equal", rectangular=rectangular,
                 num_stars=n, random_seed=40 + n)
    cfg = dict(field, num_phi=num_phi, num_branches=nb, precision=precision, write_mu_length_scales=mu)
    a = run(cfg)
    z = a["ccs"].ravel()
    w = O.eval_field(z, **field)["w"]
    assert np.all(np.abs(a["caustics"].ravel() - w) <= 1e-11 * (1 + np.abs(w) + np.abs(z)))
    if mu:
        assert np.all(a["mu_length_scales"] > 0)
    for host in (1, 2):
        b = run(cfg, host_outputs=host)
        for k in ("ccs", "caustics", "errs") + (("mu_length_scales",) if mu else ()):
            assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("n, rectangular, num_phi, nb", [
    (1, 0, 16, 1),        # one star, fewer roots than lanes
    (3, 1, 40, 1),        # an odd near list, roots off the box
    (33, 0, 24, 3),       # groups past the last root
    (150, 1, 24, 2),      # rows tracked again and re-run
    (300, 1, 64, 8),      # a middling launch, smooth-mass series not folded into every leaf
])
def test_roots_split_over_lanes_find_the_same_zeros(n, rectangular, num_phi, nb):
    """A small launch evaluates each root with 2, 4 or 8 lanes, a launch that
    fills the GPU with one: the same field alone and in a batch of enough
    copies.  Both converge to a step below 1e-9 theta_star quadratically and
    so agree within the tracker tests' 1e-11."""
    cfg = dict(kappa_tot=0.45, kappa_star=0.4, shear=0.3, mass_function="equal", rectangular=rectangular, num_stars=n,
               num_phi=num_phi, num_branches=nb, random_seed=60 + n)
    a = run(cfg)
    items = 2 * a["info"]["centres_solved"] * ((a["info"]["num_roots"] + 31) // 32)
    for per_sm in (1, 2, 4):    # more items than that per SM: 4, 2 and 1 lanes per root
        copies = [CCF(**cfg) for _ in range(per_sm * 152 // items + 1)]
        if len(copies) == 1:
            continue
        run_batch(copies)
        d = O.match_sets(a["ccs"], copies[-1].results()["ccs"], nb)
        assert d["non_finite"] == 0 and d["non_bijective_cols"] == 0
        assert d["max_dist"] <= 1e-11


@pytest.mark.parametrize("n, rectangular, num_phi, nb", [
    (4096, 1, 16, 2),     # the smallest field whose off-box roots have a CTA of several warps each
    (4501, 1, 24, 1),     # an odd number of stars
    (4501, 0, 16, 1),     # few roots off the box
])
def test_fp64_roots_off_the_box_find_the_full_sum_zeros(n, rectangular, num_phi, nb):
    """The FP64 far launch, whose warps share a root's stars: the zeros of the
    full-sum continuation, and the oracle's lens map of them (1e-11 as in the
    tests above)."""
    field = dict(kappa_tot=0.45, kappa_star=0.4, shear=0.3, mass_function="equal", rectangular=rectangular, num_stars=n,
                 random_seed=7 + n)
    cfg = dict(field, num_phi=num_phi, num_branches=nb, precision="fp64")
    t = run(cfg)
    a = run(cfg, continuation="aberth")
    d = O.match_sets(t["ccs"], a["ccs"], nb)
    assert d["non_finite"] == 0 and d["non_bijective_cols"] == 0
    assert d["max_dist"] <= 1e-11
    h = t["info"]["root_half_length"]
    z, w = t["ccs"].ravel(), t["caustics"].ravel()
    off = np.flatnonzero(np.maximum(np.abs(z.real), np.abs(z.imag)) > h)
    assert off.size > 0 or not rectangular
    off = off[:: max(1, off.size // 200)]
    want = O.eval_field(z[off], **field)["w"]
    assert np.all(np.abs(w[off] - want) <= 1e-11 * (1 + np.abs(want) + np.abs(z[off])))


@pytest.mark.parametrize("precision, mu", [("mixed", 0), ("mixed", 1), ("fp64", 0)])
@pytest.mark.parametrize("n, num_phi, nb", [(4096, 32, 4), (9001, 16, 2)])
def test_streamed_far_launches_give_the_same_bits(monkeypatch, n, num_phi, nb, precision, mu):
    """One group of centres at a time, each with far launches of several warps
    of its own, against the whole field at once."""
    cfg = dict(kappa_tot=0.45, kappa_star=0.4, shear=0.3, mass_function="equal", rectangular=1, num_stars=n,
               num_phi=num_phi, num_branches=nb, random_seed=7 + n, precision=precision, write_mu_length_scales=mu)
    a = run(cfg)
    monkeypatch.setenv("CCF_GB300_CHUNK_BYTES", "1")
    b = run(cfg, host_outputs=2)
    for k in ("ccs", "caustics", "errs") + (("mu_length_scales",) if mu else ()):
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("n, rectangular, num_phi, nb", [(137, 0, 24, 2), (150, 1, 24, 2), (4501, 1, 24, 1)])
def test_a_batch_mate_with_length_scales_leaves_the_zeros(n, rectangular, num_phi, nb):
    """One field with length scales moves its whole batch to the scalar
    evaluator and its off-box roots to the items: the same zeros as alone."""
    cfg = dict(kappa_tot=0.45, kappa_star=0.4, shear=0.3, mass_function="equal", rectangular=rectangular, num_stars=n,
               num_phi=num_phi, num_branches=nb, random_seed=7 + n)
    mate = dict(cfg, num_stars=40, write_mu_length_scales=1)
    alone, mate_alone = run(cfg), run(mate)
    fs = [CCF(**cfg), CCF(**mate)]
    assert run_batch(fs, -1), fs[0].last_error()
    for f, want in zip(fs, (alone, mate_alone)):
        r = f.results()
        for k in ("ccs", "caustics"):
            d = O.match_sets(r[k], want[k], nb)
            assert d["non_finite"] == 0 and d["non_bijective_cols"] == 0
        assert O.match_sets(r["ccs"], want["ccs"], nb)["max_dist"] <= 1e-11
