"""GPU tests of the error paths the C ABI promises in place of the reference's
check_alloc -> MPI_Abort (src/sources/checks.c:4-24).

* Bounded device loops.  Every tree-merge loop has an iteration limit; when it runs
  out the kernel sets an error bit and returns (no trap, no hang), and the next
  synchronising call reports DCF_ERR_TIMEOUT.  The test lowers the limit with the
  context's DCF_MERGE_BOUND knob so that an ordinary build runs out, then checks the
  status and that the device stays usable.
* Allocation failures.  The context's DCF_FAIL_ALLOC = k knob makes its k-th device
  allocation report out-of-memory; every k up to the number of allocations a build,
  filter and spectrum make must give DCF_ERR_NOMEM, and the same context must then
  build correctly.
Both knobs are read when a context is created.
"""
import numpy as np
import pytest

import disccofan_gb300 as dcf
from oracle import oracle

pytestmark = pytest.mark.gpu

TIMEOUT, NOMEM = 4, 2


def _torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def knob_ctx(monkeypatch, name, value):
    monkeypatch.setenv(name, str(value))
    ctx = dcf.Context(0)
    monkeypatch.delenv(name)
    return ctx


def image(seed=3, shape=(200, 230)):
    rng = np.random.default_rng(seed)
    return rng.integers(0, 5000, shape).astype(np.uint16)


def check_against_oracle(t, img, conn, tree):
    port = oracle.Port()
    port.load(img.astype(np.float32), conn, tree)
    port.prepare(0)
    assert np.array_equal(t.parent(), port.parent())
    assert np.array_equal(t.filter(0, 50.0), port.filter(0, 50.0, 0))


@pytest.mark.parametrize("conn,shape", [(8, (200, 230)), (4, (130, 300)), (6, (20, 40, 50))])
def test_merge_loop_limit_reports_timeout(monkeypatch, conn, shape):
    _torch()
    img = image(shape=shape)
    ctx = knob_ctx(monkeypatch, "DCF_MERGE_BOUND", 2)
    with pytest.raises(dcf.DcfError) as e:
        t = ctx.build(img, connectivity=conn, tree_type="max", attribute=0)
        t.parent()
    assert e.value.status == TIMEOUT
    ctx.close()
    # the device and a fresh context are unaffected
    ok = dcf.Context(0)
    check_against_oracle(ok.build(img, connectivity=conn, tree_type="max", attribute=0), img, conn, "max")
    ok.close()


def test_merge_loop_limit_reports_timeout_in_batches(monkeypatch):
    _torch()
    shapes = [(90, 70), (64, 130), (150, 40)]
    rng = np.random.default_rng(8)
    cuts = [rng.standard_normal(s).astype(np.float32) for s in shapes]
    ctx = knob_ctx(monkeypatch, "DCF_MERGE_BOUND", 2)
    b = ctx.batch(shapes, np.float32, connectivity=8, attribute=13)
    with pytest.raises(dcf.DcfError) as e:
        b.run(b.concat(cuts), filter_attr=0, lam=10.0, use_graph=False)
    assert e.value.status == TIMEOUT
    b.close()
    ctx.close()


def test_every_allocation_failure_reports_nomem(monkeypatch):
    _torch()
    img = image(shape=(150, 170))
    lv1 = dcf.lvec_from_values([1.5, 2, 4, 8])
    lv2 = dcf.lvec_from_values([4, 16, 64, 256])
    failures = 0
    for k in range(64):
        ctx = knob_ctx(monkeypatch, "DCF_FAIL_ALLOC", k)
        try:
            t = ctx.build(img, connectivity=8, tree_type="min", attribute=18)
            t.filter(0, 50.0, "subtractive")
            t.pattern_spectrum2d(18, lv1, 0, lv2)
            t.set_attribute(13)
            t.filter(14, 2.0)
        except dcf.DcfError as e:
            assert e.status == NOMEM, (k, str(e))
            failures += 1
            # one refusal only: the same context then works
            check_against_oracle(ctx.build(img, connectivity=8, tree_type="min", attribute=0), img, 8, "min")
            ctx.close()
            continue
        ctx.close()
        break
    else:
        pytest.fail("the knob never ran past the allocations of a build")
    assert failures >= 5


def test_batch_allocation_failures_report_nomem(monkeypatch):
    _torch()
    shapes = [(40, 50), (70, 33)]
    rng = np.random.default_rng(2)
    cuts = [rng.standard_normal(s).astype(np.float32) for s in shapes]
    failures = 0
    for k in range(64):
        ctx = knob_ctx(monkeypatch, "DCF_FAIL_ALLOC", k)
        b = None
        try:
            b = ctx.batch(shapes, np.float32, connectivity=8, attribute=13)
            b.run(b.concat(cuts), filter_attr=0, lam=10.0, use_graph=False)
        except dcf.DcfError as e:
            assert e.status == NOMEM, (k, str(e))
            failures += 1
            if b is not None:
                b.close()  # batches go before their context
            ctx.close()
            continue
        b.close()
        ctx.close()
        break
    else:
        pytest.fail("the knob never ran past the allocations of a batch")
    assert failures >= 5


def test_builds_on_a_full_device(monkeypatch):
    """DCF_SHORT_ALLOC = k: the context's k-th allocation finds the device full, once.
    Whichever it is, later builds and filters give the right results: the basin build's
    scratch is given back or the merging build takes over, and only a call that has
    neither way out reports the shortage."""
    _torch()
    monkeypatch.delenv("DCF_FAIL_ALLOC", raising=False)
    img = image(shape=(150, 170))
    vol = image(shape=(20, 30, 25))
    ref = dcf.Context(0)
    want = []
    for x in (img, vol):
        t = ref.build(x, connectivity=8, tree_type="min", attribute=18)
        want.append([t.parent(), t.filter(18, 2.0), t.filter(0, 50.0, "min"), t.filter(0, 50.0, "subtractive")])
        t.set_attribute(13)
        want[-1].append(t.filter(14, 2.0))
    ref.close()
    recovered = 0
    for k in range(64):
        ctx = knob_ctx(monkeypatch, "DCF_SHORT_ALLOC", k)
        short = 0
        for x, w in zip((img, vol, img, vol), (want[0], want[1]) * 2):
            try:
                t = ctx.build(x, connectivity=8, tree_type="min", attribute=18)
                got = [t.parent(), t.filter(18, 2.0), t.filter(0, 50.0, "min"), t.filter(0, 50.0, "subtractive")]
                t.set_attribute(13)
                got.append(t.filter(14, 2.0))
            except dcf.DcfError as e:
                assert e.status == NOMEM, (k, str(e))
                short += 1
                continue
            for i, (g, v) in enumerate(zip(got, w)):
                assert np.array_equal(g, v), (k, i)
        assert short <= 1, k  # one shortage, one call at most
        recovered += short == 0
        ctx.close()
    assert recovered >= 10


def test_batches_on_a_full_device(monkeypatch):
    """The same for batches: whichever allocation finds the device full, runs, graphs and
    gradients of the batch come out as they do with room, from basins or merged."""
    _torch()
    monkeypatch.delenv("DCF_FAIL_ALLOC", raising=False)
    shapes = [(40, 50), (70, 33), (128, 96)]
    rng = np.random.default_rng(2)
    cuts = [rng.standard_normal(s).astype(np.float32) for s in shapes]
    n = sum(h * w for h, w in shapes)
    lv1, lv2 = dcf.lvec_from_values([10, 1e3, 1e5]), dcf.lvec_from_values([4, 16, 64, 256])
    v, w = rng.standard_normal(n).astype(np.float32), rng.standard_normal((len(shapes), lv2.size, lv1.size))

    def calls(ctx):
        b = ctx.batch(shapes, np.float32, connectivity=8, attribute=13)
        pix, out = b.concat(cuts), []
        for graph in (False, True, True):
            out += list(b.run(pix, filter_attr=0, lam=10.0, spectrum=(13, lv1, 0, lv2), use_graph=graph))
            out += [b.adjoint(v, w), b.parent()]
        b.close()
        return out

    ref = dcf.Context(0)
    want = calls(ref)
    ref.close()
    for k in range(64):
        ctx = knob_ctx(monkeypatch, "DCF_SHORT_ALLOC", k)
        try:
            got = calls(ctx)
        except dcf.DcfError as e:  # before there is any scratch to give back
            assert e.status == NOMEM and k < 20, (k, str(e))
            ctx.close()
            continue
        for i, (g, x) in enumerate(zip(got, want)):
            if g.dtype == np.float64 or i % 4 == 2:  # sums in another order
                np.testing.assert_allclose(g, x, rtol=1e-6 if i % 4 == 2 else 1e-12, atol=1e-6 * np.abs(x).max())
            else:
                assert np.array_equal(g, x), (k, i)
        ctx.close()


@pytest.mark.parametrize("conn", [6, 26])
def test_volumes_with_more_saddles_than_the_scratch_holds(monkeypatch, conn):
    """No volume is known to have more than two saddle edges a pixel, which is what the
    scratch holds; a lower bound by knob shows that such a one would be merged, and that the
    context then takes what fits as before."""
    _torch()
    vol, few = image(shape=(20, 30, 25)), np.zeros((20, 30, 25), np.uint16)
    few[3, 4, 5] = 9
    port = oracle.Port()
    for cap in (1, 60, 1500):
        ctx = knob_ctx(monkeypatch, "DCF_EDGE_CAP", cap)
        ctx.set_profiling()
        for x, merged in ((vol, True), (few, False), (vol, True)):
            before = ctx.profile().get("tile_build", (0, 0))[1]
            t = ctx.build(x, connectivity=conn, tree_type="max", attribute=0)
            port.load(x.astype(np.float32), conn, "max")
            port.prepare(0)
            assert np.array_equal(t.parent(), port.parent())
            assert np.array_equal(t.filter(0, 50.0), port.filter(0, 50.0, 0))
            assert (ctx.profile().get("tile_build", (0, 0))[1] > before) == merged, (cap, merged)
            t.close()
        ctx.close()


def test_builds_and_attribute_passes_are_refused_under_capture():
    torch = _torch()
    stream = torch.cuda.Stream()
    ctx = dcf.Context(0, stream=stream.cuda_stream)
    img = image()
    t = ctx.build(img, connectivity=8, tree_type="max", attribute=13)
    want = t.filter(14, 2.0)
    t.set_attribute(0)
    out = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out += 1
        with pytest.raises(dcf.DcfError):
            t.set_attribute(13)
        with pytest.raises(dcf.DcfError):
            ctx.build(img, connectivity=8, tree_type="max", attribute=0)
    graph.replay()
    torch.cuda.synchronize()
    assert out.eq(1).all()
    t.set_attribute(13)
    assert np.array_equal(t.filter(14, 2.0), want)
    ctx.close()
