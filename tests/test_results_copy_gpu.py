"""Results into pageable arrays whose pages are mapped by several threads before
the copy: new arrays, used arrays, and arrays that begin and end inside a page,
whose neighbours' bytes stay as they were."""
import numpy as np
import pytest

from ccf_gb300 import CCF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("num_stars, num_phi", [(40, 16), (300, 600), (1000, 1024)])   # 0.05, 14 and 80 MB
@pytest.mark.parametrize("offset", [0, 1, 4099])
def test_results_into_pageable_arrays(num_stars, num_phi, offset):
    c = CCF(kappa_tot=0.3, kappa_star=0.3, shear=0.1, num_stars=num_stars, num_phi=num_phi, num_branches=2)
    assert c.run(-1), c.last_error()
    want = c.results(stars=False, out=c.result_buffers(pinned=True))
    out, whole = {}, {}
    for k in ("ccs", "caustics", "errs"):
        n = want[k].size
        whole[k] = np.empty(n + offset + 5, want[k].dtype)
        whole[k][:offset] = 7
        whole[k][offset + n:] = 9
        out[k] = whole[k][offset:offset + n].reshape(want[k].shape)
    for _ in range(2):                       # the pages are there the second time
        got = c.results(stars=False, out=out)
        for k in out:
            assert np.array_equal(got[k], want[k]), k
            assert np.all(whole[k][:offset] == 7) and np.all(whole[k][-5:] == 9), k
    fresh = c.results(stars=False)
    for k in out:
        assert np.array_equal(fresh[k], want[k]), k
