"""The full-sum rows cut into units over the whole GPU (rows.cu): the same bits
whatever number of CTAs takes the units and however they are cut, and the zeros
of the cluster-per-row kernel that ccf_continue_branch_noalloc keeps.  Sizes at the edges of the units: rows of one block and one unit, blocks
and chunks that end short, several tiles, more rows than fit the partial sums'
slots, steps with no root left after the first check.
"""
import ctypes

import numpy as np
import pytest

from ccf_gb300 import CCF, run_batch
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def field(n, rectangular, nb=1, num_phi=16, **kw):
    return CCF(kappa_tot=0.4, kappa_star=0.35, shear=0.2, mass_function="uniform", m_lower=0.5, m_upper=1.5,
               rectangular=rectangular, num_stars=n, num_branches=nb, num_phi=num_phi, random_seed=31 + n, **kw)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [1, 16, 127, 128, 129, 255, 512, 513, 700])
def test_rows_do_not_depend_on_the_number_of_ctas(n, precision):
    """One field alone (every CTA on its rows) and in a batch of eight (a CTA
    has about one row): the launches differ, the roots are the same bits.  Both
    have rows enough for clusters of one CTA, so the order of summation is one."""
    a = field(n, 0, nb=8, num_phi=64, continuation="aberth", precision=precision, init_cluster=1)
    assert a.run(-1), a.last_error()
    r = a.results()
    fs = [field(n, 0, nb=8, num_phi=64, continuation="aberth", precision=precision, init_cluster=1) for _ in range(8)]
    for i, f in enumerate(fs[1:]):
        f.random_seed = 500 + i
    assert run_batch(fs, -1), fs[0].last_error()
    b = fs[0].results()
    centre = 64 // 8 // 2
    assert np.array_equal(r["ccs"][:, centre], b["ccs"][:, centre])
    d = O.match_sets(r["ccs"], b["ccs"], 8)
    assert d["non_finite"] == 0 and d["non_bijective_cols"] == 0
    assert d["max_dist"] <= 1e-11
    assert r["info"]["unconverged"] == 0


@pytest.mark.parametrize("n, rectangular", [(1, 0), (100, 1), (300, 0), (520, 1)])
def test_rows_are_repeatable(n, rectangular):
    outs = []
    for _ in range(2):
        c = field(n, rectangular, nb=2, num_phi=32, continuation="aberth")
        assert c.run(-1), c.last_error()
        outs.append(c.results())
    assert np.array_equal(outs[0]["ccs"], outs[1]["ccs"])
    assert np.array_equal(outs[0]["caustics"], outs[1]["caustics"])
    assert np.array_equal(outs[0]["errs"], outs[1]["errs"])


@pytest.mark.parametrize("n, rectangular", [(1, 0), (20, 0), (129, 0), (300, 0), (520, 0)])
def test_rows_are_the_cluster_kernels(n, rectangular):
    """Branch 0, side 0 of a full-sum run, and the same steps from the same
    centre by ccf_continue_branch_noalloc."""
    import torch
    nb, num_phi = 2, 32
    half = num_phi // nb // 2
    c = field(n, rectangular, nb=nb, num_phi=num_phi, continuation="aberth")
    assert c.run(-1), c.last_error()
    r = c.results()
    R = r["info"]["num_roots"]
    start = torch.from_numpy(np.ascontiguousarray(r["ccs"].reshape(R, nb, -1)[:, 0, half]).view(np.float64).copy()).cuda()
    shape = r["ccs"].shape
    ccs = torch.zeros(shape[0] * shape[1] * 2, dtype=torch.float64, device="cuda")
    errs = torch.zeros(shape[0] * shape[1], dtype=torch.float64, device="cuda")
    f = c._L.ccf_continue_branch_noalloc
    f.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 5
    f.restype = ctypes.c_int
    assert f(c._h, 0, 0, half, start.data_ptr(), ccs.data_ptr(), errs.data_ptr(), None, None) == 0, c.last_error()
    torch.cuda.synchronize()
    z = ccs.cpu().numpy().view(np.complex128).reshape(R, nb, -1)[:, 0, :half]
    want = r["ccs"].reshape(R, nb, -1)[:, 0, :half]
    # the centre's snapshot is refreshed one sweep apart in the two, by less than the 1e-9 theta_star tolerance:
    # the sums' 1e-9 changes a converging step's end quadratically less
    assert np.max(np.abs(z - want)) <= 1e-11


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [31, 32, 33, 64, 65, 321])
def test_rows_do_not_depend_on_the_blocks(n, precision):
    """Alone a field's steps and checks go over blocks of 64 roots, in a batch
    of 40 over 128 or 256: the same bits in the solved column."""
    a = field(n, 0, nb=8, num_phi=64, continuation="aberth", precision=precision, init_cluster=1)
    assert a.run(-1), a.last_error()
    r = a.results()
    fs = [field(n, 0, nb=8, num_phi=64, continuation="aberth", precision=precision, init_cluster=1) for _ in range(40)]
    assert run_batch(fs, -1), fs[0].last_error()
    for f in (fs[0], fs[-1]):
        b = f.results()
        assert np.array_equal(r["ccs"][:, 4], b["ccs"][:, 4])
        assert O.match_sets(r["ccs"], b["ccs"], 8)["max_dist"] <= 1e-11


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n, nb", [(63, 1), (65, 4), (260, 2), (600, 1)])
def test_rows_do_not_depend_on_the_sums_tiles(n, nb, precision):
    """A row alone has sums units of half the warps, forty copies of it full
    ones: the same bits in the solved column."""
    def make():
        return field(n, 1, nb=nb, num_phi=8 * nb, continuation="aberth", precision=precision, init_cluster=1)
    a = make()
    assert a.run(-1), a.last_error()
    r = a.results()
    fs = [make() for _ in range(40)]
    assert run_batch(fs, -1), fs[0].last_error()
    b = fs[-1].results()
    assert np.array_equal(r["ccs"][:, 4], b["ccs"][:, 4])
    assert O.match_sets(r["ccs"], b["ccs"], nb)["max_dist"] <= 1e-11


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n, rectangular", [(1, 0), (40, 1), (129, 0), (520, 1), (1500, 0)])
def test_whole_sums_are_the_chunks_sums(monkeypatch, n, rectangular, precision):
    """A row whose partial sums would exceed its memory has its units add their
    chunks up, in the order in which the step adds them otherwise: the same
    bits with every sweep whole (1 byte) and with the first ones whole."""
    outs = []
    for limit in (None, "1", "60000"):
        if limit:
            monkeypatch.setenv("CCF_GB300_ROW_SUMS_BYTES", limit)
        c = field(n, rectangular, nb=2, num_phi=8, continuation="aberth", precision=precision)
        assert c.run(-1), c.last_error()
        outs.append(c.results())
    for r in outs[1:]:
        for k in ("ccs", "caustics", "errs"):
            assert np.array_equal(outs[0][k], r[k]), k


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n, shear, scale", [(60, 0.02, 1.18), (60, 0.0, 1.2), (200, 0.06, 1.2)])
def test_more_off_box_roots_than_one_pass_takes(n, shear, scale, precision):
    """A nearly square rectangle with a long Taylor series has 72 to 93 roots
    off the root box at the end of its row, more than the 64 of one pass of the
    CTA's star sums: the same bits alone (blocks of 64 roots) and in a batch of
    40 (blocks of 256)."""
    def make():
        return CCF(kappa_tot=0.45, kappa_star=0.4, shear=shear, mass_function="equal", rectangular=1, num_stars=n,
                   num_branches=4, num_phi=32, random_seed=3, safety_scale=scale, continuation="aberth", init_cluster=1,
                   precision=precision)
    a = make()
    assert a.run(-1), a.last_error()
    r = a.results()
    i = r["info"]
    z = r["ccs"].reshape(i["num_roots"], 4, -1)[:, 0, 4]
    off = np.maximum(np.abs(z.real), np.abs(z.imag)) > i["root_half_length"]
    assert np.count_nonzero(off[-256:]) > 64
    fs = [make() for _ in range(40)]
    assert run_batch(fs, -1), fs[0].last_error()
    for f in (fs[0], fs[-1]):
        b = f.results()
        for k in ("ccs", "caustics", "errs"):
            assert np.array_equal(r[k], b[k]), k
