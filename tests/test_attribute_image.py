"""The attribute image of trace, planar elongation and planar non-compactness
(dcf_attribute_check) measured against exact arithmetic, beside the float of the double
readout (dcf_node_attribute).

Planar nodes with unit pixels take pairs of floats over 128-bit moments (dcf_attr_eval.cuh).
Their result is within half a float ulp plus 2^-30 of the true value v.  Where the readout
rounds to the float nearest to v, the two errors differ by 2^-30 v at most, else the
readout's is the larger one: no node may be further off than its readout by more than
2^-30 v, and the image as a whole neither.  Everything else is the rounded readout bit for
bit: elongations from about 1000 on, nodes off the first slice of a volume, other pixel
sizes, sides above 65536."""
import math

import numpy as np
import pytest

import disccofan_gb300 as dcf
from test_attr_compare import smooth

pytestmark = pytest.mark.gpu


def corner(shape, at, seed):
    """A textured patch far from the origin, where the readout subtracts large sums."""
    img = np.zeros(shape, np.float32)
    patch = smooth((40, 50), seed) + 9
    img[at[0]:at[0] + 40, at[1]:at[1] + 50] = patch
    return img


IMAGES = {"noise": np.random.default_rng(1).standard_normal((90, 111)).astype(np.float32),
          "smooth": smooth((160, 201), 2),
          "corner": corner((60, 9000), (15, 8900), 7),
          "wide": np.random.default_rng(4).integers(0, 9, (2, 30000)).astype(np.uint8),
          "line": np.arange(900, dtype=np.float32)[::-1].reshape(1, 900).copy(),  # nodes of 1..900 pixels in a line
          "far line": np.arange(60000, dtype=np.uint16).reshape(1, 60000) // 67}  # the same, far from the origin


def moments(root, par, gv, w):
    n = par.size
    x, y = np.arange(n) % w, np.arange(n) // w
    sums = np.zeros((n, 6), object)
    cols = [np.ones(n, np.int64), x, y, x * x, y * y, x * y]
    node = np.where(root, np.arange(n), par)
    for k, c in enumerate(cols):
        sums[:, k] = np.bincount(node, c, n).astype(np.int64).astype(object)
    for p in np.flatnonzero(root)[np.argsort(-gv[root], kind="stable")]:  # from the top down
        if par[p] >= 0:
            sums[par[p]] += sums[p]
    return sums


def true_value(attr, n, sx, sy, sxx, syy, sxy):
    cx, cy, cxy = n * sxx - sx * sx, n * syy - sy * sy, n * sxy - sx * sy
    P = 6 * (cx + cy) + n * n
    if attr == 13:
        return P / (6 * n)
    if attr == 17:
        return P / (6 * n ** 3)
    d = math.isqrt(((cx - cy) ** 2 + 4 * cxy * cxy) << 400)  # D * 2^200
    return ((P << 200) + 6 * d) / ((P << 200) - 6 * d)


@pytest.mark.parametrize("attr", [13, 14, 17])
@pytest.mark.parametrize("name", sorted(IMAGES))
def test_no_further_from_the_true_value_than_the_readout(ctx, name, attr):
    img = IMAGES[name]
    t = ctx.build(img, connectivity=8, tree_type="max", attribute=attr)
    par, gv, val, got = t.parent(), t.gval(), t.node_attribute(attr), t.check(attr).ravel()
    t.close()
    root = ~np.isnan(val)
    assert np.array_equal(got, got[np.where(root, np.arange(par.size), par)])  # every pixel has its node's value
    sums = moments(root, par, gv, img.shape[-1])
    r = np.flatnonzero(root)
    want = np.array([true_value(attr, *sums[p]) for p in r])
    mine, readout = np.abs(got[r] - want), np.abs(val[r].astype(np.float32) - want)
    assert (mine <= readout + want * 2.0 ** -30).all()
    assert np.linalg.norm(mine) <= np.linalg.norm(readout) + np.linalg.norm(want) * 2.0 ** -30
    pairs = want < 999 if attr == 14 else np.ones(r.size, bool)
    assert (mine <= 0.5 * np.spacing(want.astype(np.float32)) + want * 2.0 ** -30)[pairs].all()
    rest = ~pairs & (want > 1001)
    assert np.array_equal(got[r][rest], val[r][rest].astype(np.float32))
    if attr == 14 and name == "line":  # both sides of the hand-over to the readout
        assert ((want > 900) & pairs).any() and rest.any()
    if name == "wide" and attr == 13:
        assert (mine < readout).any()  # the readout is further off than a float here


@pytest.mark.parametrize("attr", [13, 14, 17])
@pytest.mark.parametrize("kind", ["volume", "pixdim", "side"])
def test_everything_else_is_the_rounded_readout(ctx, kind, attr):
    img = {"volume": smooth((17, 20, 23), 5), "pixdim": IMAGES["noise"], "side": smooth((1, 65537), 6)}[kind]
    t = ctx.build(img, connectivity=6 if img.ndim == 3 else 8, tree_type="max", attribute=attr,
                  pixdim=(1.0, 1.0, 2.0) if kind == "pixdim" else (1.0, 1.0, 1.0))
    val, got, par = t.node_attribute(attr), t.check(attr).ravel(), t.parent()
    t.close()
    root = ~np.isnan(val)
    same = got == np.where(root, val, val[par]).astype(np.float32)
    if kind == "volume":  # nodes within the first slice are planar
        first = np.arange(par.size) < 20 * 23
        same |= first
        off = np.abs(got - np.where(root, val, val[par]))
        assert (off <= 1e-6 * np.abs(got)).all()
    assert same.all()
