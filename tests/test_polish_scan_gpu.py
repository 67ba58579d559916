"""The polish's scan of the 1/mu errors: sizes about its groups of 128 points (a
warp's four loads) and fields whose every point, or none, is flagged."""
import numpy as np
import pytest

from ccf_gb300 import CCF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, num_phi, nb", [(1, 2, 1), (8, 6, 1), (16, 6, 1), (16, 8, 1), (33, 62, 1), (500, 510, 1)])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_scan_sees_every_point(n, num_phi, nb, precision):
    """the largest error of the report is the largest of the stored ones"""
    c = CCF(kappa_tot=0.4, kappa_star=0.35, shear=0.2, mass_function="salpeter", m_lower=0.1, m_upper=2.0, num_stars=n,
            num_phi=num_phi, num_branches=nb, random_seed=n, precision=precision)
    assert c.run(-1), c.last_error()
    r = c.results()
    assert r["info"]["max_error"] == np.max(r["errs"])
    assert r["info"]["unconverged"] == 0 and np.min(r["errs"]) >= 0
