"""Spectra with as many bins as the kernels keep in shared memory, one less and one more,
against sums taken on the host from the tree's own parents, levels and readouts.  u8/u16
sums are integers and equal; float sums differ by the order of their terms."""
import numpy as np
import pytest

import disccofan_gb300 as dcf

pytestmark = pytest.mark.gpu


def bins(n, top):
    return np.r_[np.float32(0), np.geomspace(0.5, top, n - 1).astype(np.float32)] if n > 1 else np.zeros(1, np.float32)


# (bins on attribute 18, bins on the area); 3584 was the most a launch without an opt-in held
@pytest.mark.parametrize("n1,n2", [(56, 64), (15, 239), (64, 64), (17, 241), (128, 32), (1, 4096), (4096, 1), (4095, 1)])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("pixdim", [(1.0, 1.0, 1.0), (0.5, 2.0, 1.0)])
def test_spectra_at_the_limits_of_the_bins(ctx, dtype, n1, n2, pixdim):
    rng = np.random.default_rng(8)
    img = (rng.random((160, 171)) * 250 + np.arange(171) / 3).astype(dtype)
    t = ctx.build(img, connectivity=8, tree_type="max", attribute=18, pixdim=pixdim)
    par, gv = t.parent(), t.gval()
    v1, area = t.node_attribute(18), t.node_attribute(18, area=True)
    l1, l2 = bins(n1, 40.0), bins(n2, 2e4)
    got = (t.pattern_spectrum(18, l1) if n2 == 1 else t.pattern_spectrum2d(18, l1, 0, l2)).ravel()
    r = np.flatnonzero(~np.isnan(v1))
    dh = np.where(par[r] < 0, gv[r], gv[r] - gv[np.maximum(par[r], 0)])
    assert dh.dtype == np.float32
    terms = dh.astype(np.float64) * area[r]
    find = lambda lv, v: np.maximum(np.searchsorted(lv.astype(np.float64), v, side="right") - 1, 0)
    at = find(l1, v1[r]) + n1 * (find(l2, area[r]) if n2 > 1 else 0)
    want = np.bincount(at, terms, n1 * n2)
    if dtype == np.float32:
        assert (np.abs(got - want) <= np.bincount(at, np.abs(terms), n1 * n2) * r.size * 2.0 ** -52).all()
    else:
        assert np.array_equal(got, want)
    t.close()
