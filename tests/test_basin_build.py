"""The basin build (csrc/dcf_basin.cu): trees from peaks, saddles and sorted chains.

On the CPU its scheme and neighbourhood code run on small random images of every
connectivity against a union-find flood.  On the GPU its parents are compared with
the merging build's (a context with DCF_BASIN_MIN above every size) at tile edges, for
every pixel type, connectivity and tree type, on flat and regular images, in batches,
and where more than one radix pass over the component numbers is needed.  Parents are
canonical, so they are equal bit for bit.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

import disccofan_gb300 as dcf

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "disccofan_gb300", "csrc")


@pytest.mark.parametrize("conn", [4, 8, 6, 26])
def test_scheme_against_flood_on_host(tmp_path, conn):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    exe = tmp_path / "around"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + CSRC, os.path.join(HERE, "around_harness.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe), str(conn), "1500", "7"], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


@pytest.fixture(scope="module")
def builds():
    """(basin build, merging build) contexts"""
    out = []
    for least in ("1", str(1 << 40)):
        os.environ["DCF_BASIN_MIN"] = least
        out.append(dcf.Context(0))
        del os.environ["DCF_BASIN_MIN"]
    yield out
    for c in out:
        c.close()


def image(shape, kind, dtype, seed):
    rng = np.random.default_rng(seed)
    n = int(np.prod(shape))
    if kind == "noise":
        a = rng.integers(0, 256 if dtype == np.uint8 else 60000, shape)
    elif kind == "few":
        a = rng.integers(0, 4, shape)
    elif kind == "flat":
        a = np.full(shape, 7)
    elif kind == "ramp":  # one long monotone path per row, ties across rows
        a = np.broadcast_to(np.arange(shape[-1]) % 251, shape)
    else:  # checker
        a = np.indices(shape).sum(0) % 2 * 9
    a = np.asarray(a, np.float64).reshape(shape)
    if dtype == np.float32 and kind == "noise":
        a = rng.permutation(n).reshape(shape) - n / 2 + 0.25
        a.reshape(-1)[:min(n, 3)] = (-np.inf, np.inf, -0.0)[:min(n, 3)]
    return a.astype(dtype)


SHAPES = [(1, 1), (1, 77), (130, 1), (31, 63), (32, 64), (33, 65), (95, 129), (300, 411), (7, 15, 15), (8, 16, 16),
          (9, 17, 17), (33, 20, 50)]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.uint32, np.float32])
@pytest.mark.parametrize("shape", SHAPES)
def test_same_parents_as_merging_build(builds, shape, dtype):
    for kind in ("noise", "few", "flat", "ramp", "checker"):
        img = image(shape, kind, dtype, 5)
        for conn in ((4, 8) if len(shape) == 2 else (6, 26)):
            for tree in ("max", "min"):
                if tree == "min" and not np.isfinite(img.astype(np.float64)).all():
                    continue
                t = [c.build(img, connectivity=conn, tree_type=tree, attribute=0) for c in builds]
                got, want = t[0].parent(), t[1].parent()
                assert np.array_equal(got, want), (kind, conn, tree)
                assert np.array_equal(t[0].node_attribute(0), t[1].node_attribute(0), equal_nan=True)
                for x in t:
                    x.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,conn", [(np.float32, 8), (np.uint8, 4), (np.uint16, 8)])
def test_batches_same_as_merging_build(builds, dtype, conn):
    rng = np.random.default_rng(3)
    shapes = [(1, 1), (1, 9), (32, 64), (33, 65), (64, 31)] + [tuple(rng.integers(1, 200, 2)) for _ in range(12)]
    cuts = [image(s, k, dtype, 11 + i) for i, s in enumerate(shapes) for k in (("noise", "few", "flat")[i % 3],)]
    cuts = [np.where(np.isfinite(c), c, 0).astype(dtype) for c in cuts]
    res = []
    for c in builds:
        b = c.batch(shapes, dtype, connectivity=conn, attribute=0)
        pix = b.concat(cuts)
        for _ in range(3):  # exact run, recorded graph, replay
            f, _ = b.run(pix, filter_attr=0, lam=9.0)
        res.append((f, b.parent()))
        b.close()
    assert np.array_equal(res[0][1], res[1][1])
    assert np.array_equal(res[0][0], res[1][0])


@pytest.mark.gpu
def test_many_components(builds):
    """White noise of 2^21 pixels: over 2^16 components, three radix passes over their numbers."""
    img = image((1400, 1500), "noise", np.uint16, 9)
    p = []
    for c in builds:
        t = c.build(img, connectivity=4, tree_type="max", attribute=0)
        p.append(t.parent())
        t.close()
    assert np.array_equal(p[0], p[1])


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("shape", [(1, 1), (1, 77), (33, 65), (300, 411), (9, 17, 17), (700, 1500)])
def test_filter_rules_along_chains_same_as_on_merged_trees(builds, shape, dtype):
    """The direct, min and subtractive rules have paths of their own for trees with a chain
    order: same images as the general path on the merging build's trees, from nothing
    removed to everything removed.  (700, 1500) has more than one group of order blocks
    only for the scans that group 512; 2^21 entries and more are covered by
    test_scans_over_groups.)"""
    for kind in ("noise", "few", "flat"):
        img = image(shape, kind, dtype, 21)
        img = np.where(np.isfinite(img.astype(np.float64)), img, 0).astype(dtype)
        for tree in ("max", "min"):
            t = [c.build(img, connectivity=4 if len(shape) == 2 else 6, tree_type=tree, attribute=18) for c in builds]
            for attr, lam in ((0, 0.0), (0, 2.0), (0, 40.0), (3, 3.0), (18, 2.0), (0, 1e12)):
                for rule in ("direct", "min", "subtractive"):
                    if dtype == np.float32 and rule == "subtractive" and img.size > 5000:
                        continue  # the float recurrence is the same code on both trees, and slow
                    for extract in (False, True):
                        got, want = (x.filter(attr, lam, rule, extract=extract) for x in t)
                        assert np.array_equal(got, want), (kind, tree, attr, lam, rule, extract)
            for x in t:
                x.close()


@pytest.mark.gpu
def test_scans_over_groups(builds):
    """2^22 pixels: more than one group in every two-level scan over the order's blocks, with
    chains that run through whole groups (a ramp) and none that do (noise)."""
    for img in (image((2048, 2200), "noise", np.uint16, 2), (np.arange(2048 * 2200) // 70).reshape(2048, 2200).astype(np.uint16)):
        t = [c.build(img, connectivity=8, tree_type="max", attribute=18) for c in builds]
        for attr in (0, 1, 3, 18):
            assert np.array_equal(t[0].node_attribute(attr), t[1].node_attribute(attr), equal_nan=True), attr
        for rule in ("direct", "min", "subtractive"):
            for lam in (30.0, 1e5):
                assert np.array_equal(t[0].filter(0, lam, rule), t[1].filter(0, lam, rule)), (rule, lam)
        for x in t:
            x.set_attribute(13)
        assert np.array_equal(t[0].node_attribute(13), t[1].node_attribute(13), equal_nan=True)
        for x in t:
            x.close()


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["pinned", "device"])
def test_image_may_be_overwritten_after_build(where):
    """A build returns only after it has read its image, from pinned host memory and from
    device memory, also when its stream has work queued before it."""
    torch = pytest.importorskip("torch")
    img = np.random.default_rng(4).integers(0, 3000, (300, 410)).astype(np.uint16)
    stream = torch.cuda.Stream()
    ctx = dcf.Context(0, stream=stream.cuda_stream)
    want = ctx.build(img, connectivity=8, tree_type="max", attribute=0).parent()
    buf = torch.from_numpy(img.view(np.int16)).clone()
    buf = buf.pin_memory() if where == "pinned" else buf.cuda()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(40_000_000)  # about 20 ms
    if where == "pinned":
        t = ctx.build(buf.numpy().view(np.uint16), connectivity=8, tree_type="max", attribute=0)
        buf.zero_()
    else:
        with torch.cuda.stream(stream):  # no order between the caller's stream and the context's
            t = ctx.build(buf.view(torch.uint16), connectivity=8, tree_type="max", attribute=0)
        with torch.cuda.stream(torch.cuda.Stream()):
            buf.zero_()
    assert np.array_equal(t.parent(), want)
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("shape,dtype", [((80, 96), np.uint8), ((300, 410), np.float32)])
def test_back_to_back_calls(builds, shape, dtype):
    """Kernels are set up while the one before them runs out: calls that follow one another
    on a stream, with buffers that alternate between different images, must not read what
    the call before left there."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(9)
    imgs = [(rng.random(shape) * 250).astype(dtype) for _ in range(3)]
    lvec = dcf.lvec_from_values([2, 4, 8, 16])

    def call(ctx, img):
        t = ctx.build(img, connectivity=8, tree_type="max", attribute=0)
        filtered = [t.filter(0, lam, rule, out=torch.empty(shape, dtype=torch.float32, device="cuda"))
                    for lam, rule in ((3.0, "direct"), (5.0, "min"), (9.0, "direct"))]
        return t, filtered, t.pattern_spectrum(0, lvec)

    basin, merging = builds
    want = [call(merging, i) for i in imgs]
    dev = [torch.from_numpy(i).cuda() for i in imgs]
    got = [(k, call(basin, dev[k])) for _ in range(20) for k in (0, 1, 2, 1)]
    for k, (t, filtered, spec) in got:
        for g, w in zip(filtered, want[k][1]):
            assert torch.equal(g, w)
        # positive terms in any order: below 123,000 x 2^-53 apart
        assert np.allclose(spec, want[k][2], rtol=1e-10, atol=0)
        assert np.array_equal(t.parent(), want[k][0].parent())


@pytest.mark.gpu
@pytest.mark.parametrize("shape,dtype", [((4096, 8192), np.uint16), ((5793, 5795), np.uint8), ((129, 509, 512), np.uint16)])
def test_large_images_same_as_merging_build(builds, shape, dtype):
    """From 2^25 pixels on the parents reach their places by way of buckets: at the bound,
    beyond it with a ragged last bucket, and in three dimensions."""
    rng = np.random.default_rng(11)
    img = (rng.integers(0, 60, shape) * 3 + np.indices(shape, sparse=True)[-1] % 67).astype(dtype)
    for tree in ("max", "min"):
        got, want = (x.build(img, connectivity=4, tree_type=tree, attribute=0) for x in builds)
        assert np.array_equal(got.parent(), want.parent())
        assert np.array_equal(got.filter(0, 9.0), want.filter(0, 9.0))


@pytest.mark.gpu
def test_more_rows_and_slices_than_a_grid_has(builds):
    """Pixels in one column or one line of slices are the same graph as in one row: the same
    parents, from tiles whose numbers go beyond 65535 rows or slices of them."""
    n = 65536 * 32 + 77
    row = (np.random.default_rng(6).integers(0, 9, n) + np.arange(n) // 50_000).astype(np.uint8)
    def parents(img, conn):
        t = builds[0].build(img, connectivity=conn, tree_type="max", attribute=0)
        p = t.parent()
        t.close()
        return p
    assert np.array_equal(parents(row.reshape(n, 1), 4), parents(row.reshape(1, n), 4))
    m = 65536 * 8 + 33
    want = parents(row[:m].reshape(1, m), 4)
    assert np.array_equal(parents(row[:m].reshape(m, 1, 1), 6), want)
    assert np.array_equal(parents(row[:m].reshape(m, 1, 1), 26), want)
    # two slices of one column each: the columns' other neighbours are m pixels apart
    two = row[:2 * (m // 2)]
    got, flat = parents(two.reshape(2, -1, 1), 6), parents(two.reshape(2, -1), 4)
    assert np.array_equal(got, flat)


@pytest.mark.gpu
def test_large_batches_same_as_single_images(builds):
    """A batch of 2^25 pixels and more writes its parents by way of buckets, over cutouts that
    share buckets and blocks; each of its cutouts alone does not."""
    shapes = [(3000, 3333), (2777, 4100), (1, 5000), (4096, 2500), (333, 444), (1501, 1999)]
    assert sum(h * w for h, w in shapes) >= 1 << 25 > max(h * w for h, w in shapes)
    rng = np.random.default_rng(12)
    cuts = [(rng.integers(0, 60, s) * 3 + np.arange(s[1]) % 67).astype(np.uint16) for s in shapes]
    b = builds[0].batch(shapes, np.uint16, connectivity=8, attribute=0)
    lv = dcf.lvec_from_values([2, 8, 32, 128, 1024])
    f, spec = b.run(b.concat(cuts), filter_attr=0, lam=9.0, spectrum=(0, lv, 0, lv), use_graph=False)
    par, f = b.split(b.parent()), b.split(f)
    for i, c in enumerate(cuts):
        t = builds[0].build(c, connectivity=8, tree_type="max", attribute=0)
        assert np.array_equal(par[i].ravel(), t.parent()), i
        assert np.array_equal(f[i], t.filter(0, 9.0)), i
        assert np.array_equal(spec[i], t.pattern_spectrum2d(0, lv, 0, lv)), i  # integers below 2^53
        t.close()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("shape", [(2, 1, 1), (2, 32, 32), (2, 32, 33), (9, 17, 17), (40, 50, 60), (1, 77), (64, 65), (300, 411)])
def test_filters_on_costly_attributes_same_as_on_merged_trees(builds, shape, dtype):
    """The sweeps along the chain order list a block's level roots before they evaluate an
    attribute other than the area, and eigenvalues are evaluated node by node before them
    (volumes, and images with pixels that are not unit squares): at the edges of a block of
    2048 positions, for every way and rule, same images as the general path."""
    volume = len(shape) == 3
    for kind in ("noise", "few", "flat"):
        img = image(shape, kind, dtype, 23)
        img = np.where(np.isfinite(img.astype(np.float64)), img, 0).astype(dtype)
        for pixdim in ((1.0, 1.0, 1.0), (1.0, 2.0, 1.0)):
            t = [c.build(img, connectivity=6 if volume else 4, tree_type="max", attribute=14, pixdim=pixdim) for c in builds]
            for attr in (14, 16, 13) + ((15,) if volume else ()):
                lams = np.nanquantile(t[1].node_attribute(attr), [0.3, 0.9])
                for lam in (float(lams[0]), float(lams[1]), 1e12):
                    for rule in ("direct", "min", "subtractive"):
                        if dtype == np.float32 and rule == "subtractive":
                            continue  # the float recurrence is the same code on both trees
                        got, want = (x.filter(attr, lam, rule) for x in t)
                        assert np.array_equal(got, want), (kind, pixdim, attr, lam, rule)
            for x in t:
                x.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,flat", [(np.float32, 15), (np.float32, 100), (np.uint16, 60), (np.uint32, 40), (np.uint32, 60)])
def test_direct_rule_of_one_long_path(builds, dtype, flat):
    """A raster ramp is one path of N / flat nodes with areas N - k * flat: the direct rule goes
    by nodes where these are few and along the chain order where they are more than 2^16."""
    shape = (1800, 1901)
    n = shape[0] * shape[1]
    img = (np.arange(n) // flat).reshape(shape).astype(dtype)
    t = builds[0].build(img, connectivity=4, tree_type="max", attribute=0)
    assert t.info()["nodes"] == -(-n // flat)
    for lam in (1, flat + 1, 5 * flat, 70_001, n // 2, n, n + 1):
        kept = (n - lam) // flat if lam <= n else -1  # the highest surviving level
        want = np.minimum(img, kept) if kept >= 0 else np.zeros(shape)
        assert np.array_equal(t.filter(0, float(lam)), want.astype(np.float32)), lam
    t.close()


@pytest.mark.gpu
def test_many_contexts_at_once():
    """Eight threads build on contexts of their own: the component rounds are a cooperative
    kernel each, whose blocks wait for one another while the others' kernels run."""
    import threading

    imgs = [image((700 + 37 * k, 1500), "noise", np.float32 if k % 2 else np.uint16, 30 + k) for k in range(8)]
    imgs = [np.where(np.isfinite(i.astype(np.float64)), i, 0).astype(i.dtype) for i in imgs]
    ctx = dcf.Context(0)
    want = []
    for img in imgs:
        t = ctx.build(img, connectivity=8, tree_type="max", attribute=0)
        want.append((t.parent(), t.filter(0, 30.0)))
        t.close()
    ctx.close()
    bad = []

    def work(k):
        try:
            c = dcf.Context(0)
            for r in range(12):
                t = c.build(imgs[k], connectivity=8, tree_type="max", attribute=0)
                if not np.array_equal(t.filter(0, 30.0), want[k][1]) or (r % 4 == 0 and not np.array_equal(t.parent(), want[k][0])):
                    bad.append((k, r))
                t.close()
            c.close()
        except Exception as e:  # reported below, in the test's own thread
            bad.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
