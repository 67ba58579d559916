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

from ccf_gb300 import CCF
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
