"""Launch configurations of the Siddon event kernels and the autotuner.

Every configuration the projector admits (block size, threads per LOR,
ray-length binning of the event order) computes the same operator: forward
projections within 1e-5 relative L2 of the FP64 oracle (and per event within
1e-5 of the one-thread walk), back projections within the 1e-4 image budget,
the adjoint identity to 1e-6.  The autotuner keeps the fastest configuration
it timed and reconstructions with it match the default one.
"""
import numpy as np
import pytest
import torch

import pyoracle as po
import pyyrtpet_b200 as yrt
from pyyrtpet_b200 import _lib as L

pytestmark = pytest.mark.gpu

SC_ARGS = (64, 4, 4, 10, 300, 256, 16, 1, 15, 2, 1)
IP_ARGS = (64, 64, 32, 128, 128, 64)


def rel_l2(a, b):
    a = np.asarray(a, np.float64).ravel()
    b = np.asarray(b, np.float64).ravel()
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def make(tof=None, precision=L.YRTB_COMPENSATED):
    sc = yrt.Scanner("t", *SC_ARGS)
    ip = yrt.ImageParams(*IP_ARGS)
    pp = yrt.ProjectorParams(sc)
    pp.precision = precision
    if tof:
        pp.addTOF(*tof)
    return sc, ip, yrt.DeviceProjector(sc, ip, pp)


def random_events(n, seed):
    rng = np.random.default_rng(seed)
    osc = po.Scanner(*SC_ARGS)
    d1 = rng.integers(0, osc.num_dets, 3 * n).astype(np.uint32)
    d2 = rng.integers(0, osc.num_dets, 3 * n).astype(np.uint32)
    bins = po.histo3d_bins(osc, d1, d2)
    ok = (bins != np.iinfo(np.uint64).max) & (d1 != d2)
    return d1[ok][:n], d2[ok][:n]


CONFIGS = [(b, t, v) for b in (128, 256) for t in (1, 2, 4)
           for v in (3, 2, 1, 0, 4, 5, 8, 9)
           if not (t > 1 and v != 0)]


@pytest.mark.parametrize("tof", [None, (214.0, 5)])
def test_every_launch_config_vs_oracle(tof):
    sc, ip, p = make(tof)
    d1, d2 = random_events(30000, 41)
    rng = np.random.default_rng(42)
    tv = rng.normal(0, 300, len(d1)).astype(np.float32) if tof else None
    img = rng.random(ip.shape, dtype=np.float32)
    y = rng.random(len(d1)).astype(np.float32)
    ev = yrt.DeviceEvents.from_arrays(d1, d2, tof=tv)
    lors, _ = po.lors_from_detpairs(po.scanner_lut(po.Scanner(*SC_ARGS)), d1, d2)
    oip = po.ImageParams(*IP_ARGS)
    pr = po.Proj(tof_fwhm_ps=tof[0] if tof else 0.0, tof_n_std=tof[1] if tof else 0)
    f64 = po.project(oip, pr, lors, image=img, tof=tv, precision="f64")
    b64 = po.project(oip, pr, lors, values=y.astype(np.float64), tof=tv,
                     forward=False, precision="f64")
    gimg = torch.from_numpy(img).cuda()
    gy = torch.from_numpy(y).cuda()
    base = None
    for block, tpl, vec in CONFIGS:
        p.set_launch(block, tpl, 3, vector_groups=vec)
        assert p.get_launch() == {"block": block, "threads_per_lor": tpl,
                                  "bucket_shift": 3, "order": 0, "tile_shift": 1,
                                  "vector_groups": vec}
        v = p.forward(gimg, ev).cpu().numpy()
        b = p.backward(gy, ev).cpu().numpy()
        # The fused EM pass in every vector mode (float4 gathers, float4 or
        # float2 reductions): the same image up to the FP32 atomics' order.
        em = p.em_step(gimg, torch.zeros(ip.shape, device="cuda"), ev).cpu().numpy()
        if base is None:
            em0 = em
        assert rel_l2(em, em0) < 1e-5, (block, tpl, vec)
        assert rel_l2(v, f64) < 1e-5, (block, tpl)
        assert rel_l2(b, b64) < 1e-4, (block, tpl)
        lhs = float(np.dot(v.astype(np.float64), y))
        rhs = float(np.sum(b.astype(np.float64) * img))
        assert abs(lhs - rhs) <= 1e-6 * abs(lhs), (block, tpl)
        if base is None:
            base = v
        else:
            # Pieces cut at voxel planes: per-event sums differ from the
            # one-thread walk only by rounding.
            d = np.abs(v.astype(np.float64) - base) / np.maximum(np.abs(base), 1e-30)
            assert d.max() < 1e-5, (block, tpl, d.max())


def test_threads_per_lor_needs_compensated_mode():
    sc, ip, p = make((214.0, 5), precision=L.YRTB_MIRROR)
    p.set_launch(128, 1, 2)
    with pytest.raises(yrt.YrtbError, match="threads_per_lor > 1"):
        p.set_launch(256, 2, 3)
    with pytest.raises(yrt.YrtbError, match="block must be"):
        p.set_launch(512, 1, 3)
    with pytest.raises(yrt.YrtbError, match="bucket_shift"):
        p.set_launch(256, 1, 9)
    with pytest.raises(yrt.YrtbError, match="order must be"):
        p.set_launch(256, 1, 3, order=3)
    with pytest.raises(yrt.YrtbError, match="tile_shift"):
        p.set_launch(256, 1, 3, order=1, tile_shift=5)
    with pytest.raises(yrt.YrtbError, match="vector_groups"):
        p.set_launch(256, 1, 3, vector_groups=16)


@pytest.mark.parametrize("shift,order,tile", [(0, 0, 1), (2, 0, 1), (5, 0, 1),
                                              (3, 1, 0), (5, 1, 2), (7, 1, 3),
                                              (4, 2, 1), (7, 2, 0)])
def test_ordering_with_bucket_shift_is_a_subset_major_permutation(shift, order, tile):
    sc, ip, p = make((214.0, 5))
    d1, d2 = random_events(50000, 43)
    tv = np.random.default_rng(44).normal(0, 300, len(d1)).astype(np.float32)
    ev = yrt.DeviceEvents.from_arrays(d1, d2, tof=tv)
    p.set_launch(256, 1, shift, order, tile)
    S = 7
    out, offs = p.order_events(ev, S)
    perm = out.perm.cpu().numpy()
    assert np.array_equal(np.sort(perm), np.arange(len(d1)))
    for s in range(S):
        assert np.all(perm[offs[s]:offs[s + 1]] % S == s)
    # Inside a subset, ray lengths are non-decreasing in buckets of 2^shift
    # of the ordering's O(1) crossing estimate, which exceeds the walk's
    # count by the planes crossed together (ties, a few per ray at most).
    cnt = p.count_crossings(out).cpu().numpy().astype(np.int64)
    for s in range(S):
        c = cnt[offs[s]:offs[s + 1]]
        below = (c[:-1] < (127 << shift) - 8) & (c[1:] < (127 << shift) - 8)
        assert np.all(np.diff(c)[below] >= -(1 << shift) - 4)


def test_autotune_keeps_fastest_and_reconstruction_matches():
    from pyyrtpet_b200 import synthetic as S
    sc = S.scanner_c1()
    ip = yrt.ImageParams(32, 32, 16, 256, 256, 128)
    e = S.generate_events(sc, 60000, 45, tof_fwhm_ps=214.0).numpy()
    outs, reports = [], []
    for tune in (False, True):
        osem = yrt.createOSEM(sc)
        osem.setImageParams(ip)
        osem.num_MLEM_iterations = 2
        osem.num_OSEM_subsets = 3
        osem.setListModeEnabled(True)
        osem.addTOF(214.0, 5)
        osem.projectorParams.precision = L.YRTB_COMPENSATED
        osem.autotune = tune
        osem.generateSensitivityImages()
        lm = yrt.ListModeLUT(sc)
        lm.bind(e["d1"], e["d2"], tof=e["tof"])
        osem.setDataInput(lm)
        outs.append(osem.reconstruct().cpu().numpy())
        reports.append(osem.lastTuneReport)
    rep = reports[1]
    assert 0 < rep["sample_events"] <= (len(e["d1"]) + 2) // 3
    # 3 bucket shifts x 3 orders x 5 vector-group modes, then 2 blocks x
    # 3 threads/LOR minus the stage-1 shape.
    assert len(rep["tried"]) == 3 * 3 * 5 + 2 * 3 - 1
    best_ms = min(ms for _, ms in rep["tried"])
    assert [c for c, ms in rep["tried"] if ms == best_ms][0] == rep["best"]
    assert rel_l2(outs[1], outs[0]) < 1e-5


def test_em_step_same_under_every_order():
    """The EM image of a subset does not depend on the order of its events
    beyond float summation order (image budget 1e-4; here far below)."""
    sc, ip, p = make((214.0, 5))
    d1, d2 = random_events(60000, 47)
    rng = np.random.default_rng(48)
    tv = rng.normal(0, 300, len(d1)).astype(np.float32)
    img = torch.from_numpy(rng.uniform(0.5, 1.5, ip.shape).astype(np.float32)).cuda()
    ev = yrt.DeviceEvents.from_arrays(d1, d2, tof=tv)
    S = 3
    ref = None
    for order, tile in [(0, 1), (1, 0), (1, 2), (2, 1)]:
        p.set_launch(256, 1, 3, order, tile)
        out, offs = p.order_events(ev, S)
        em = torch.zeros(ip.shape, device="cuda")
        p.em_step(img, em, out, rng=L.yrtb_range(int(offs[1]), 1, int(offs[2] - offs[1])))
        em = em.cpu().numpy()
        if ref is None:
            ref = em
        else:
            assert rel_l2(em, ref) < 1e-6


def test_release_cached_memory_after_ordering():
    sc, ip, p = make((214.0, 5))
    d1, d2 = random_events(20000, 49)
    tv = np.random.default_rng(50).normal(0, 300, len(d1)).astype(np.float32)
    ev = yrt.DeviceEvents.from_arrays(d1, d2, tof=tv)
    out, offs = p.order_events(ev, 2)
    yrt.release_cached_memory()
    out2, offs2 = p.order_events(ev, 2)   # the pool grows again on demand
    assert torch.equal(out.perm, out2.perm)


# Images whose size is no multiple of 4 or 2: the last group of the vector
# reductions is sent voxel by voxel.  nx = 1 puts every ray's last voxels in it.
@pytest.mark.parametrize("precision", [L.YRTB_MIRROR, L.YRTB_COMPENSATED])
@pytest.mark.parametrize("dims", [(61, 63, 31), (30, 31, 15), (1, 1, 3), (1, 5, 1), (2, 3, 1)])
def test_vector_reductions_on_ragged_images(precision, dims):
    sc = yrt.Scanner("t", *SC_ARGS)
    ip = yrt.ImageParams(*dims, 128, 128, 64)
    pp = yrt.ProjectorParams(sc)
    pp.precision = precision
    p = yrt.DeviceProjector(sc, ip, pp)
    d1, d2 = random_events(20000, 51)
    ev = yrt.DeviceEvents.from_arrays(d1, d2)
    y = torch.rand(len(d1), generator=torch.Generator("cuda").manual_seed(1), device="cuda")
    n = ip.numVoxels

    def back(groups):
        p.set_launch(256, 1, 3, vector_groups=groups)
        buf = torch.zeros(n + 8, device="cuda")  # torch's allocations are 512-byte aligned
        p.backward(y, ev, img=buf[:n])
        assert not buf[n:].any()
        return buf[:n].cpu().numpy()

    scalar = back(0)
    for groups in (2, 4, 8):
        # The same FP32 terms in two orders, at most all of them in one
        # voxel: half an ulp per addition, at random, on each side.
        assert rel_l2(back(groups), scalar) < 2 * len(d1) ** 0.5 * 2.0 ** -24


@pytest.mark.parametrize("order", [L.YRTB_ORDER_LOR, L.YRTB_ORDER_SPATIAL,
                                   L.YRTB_ORDER_SPATIAL_FINE])
def test_order_with_frames_groups_subsets_then_frames(order):
    sc, _, _ = make()
    nt, S = 5, 6
    ip = yrt.ImageParams(*IP_ARGS, nt=nt)
    p = yrt.DeviceProjector(sc, ip, yrt.ProjectorParams(sc))
    p.set_launch(256, 1, 3, order=order)
    d1, d2 = random_events(30001, 52)
    fr = np.random.default_rng(53).integers(-2, nt + 2, len(d1)).astype(np.int32)
    ev = yrt.DeviceEvents.from_arrays(d1, d2, frame=fr)
    out, offs = p.order_events(ev, S, first_global_index=4)
    perm = out.perm.cpu().numpy()
    assert np.array_equal(np.sort(perm), np.arange(len(d1)))
    of = out.frame.cpu().numpy()
    assert np.array_equal(of, fr[perm])
    for s in range(S):
        part = slice(int(offs[s]), int(offs[s + 1]))
        assert np.all((perm[part] + 4) % S == s)
        f = of[part].astype(np.int64)
        f[(f < 0) | (f >= nt)] = nt  # events without a frame come last
        assert np.all(np.diff(f) >= 0)


def test_multi_ray_order_is_by_subset_bin_and_tof():
    """The offsets of an event's extra rays follow its place in the order, so
    the order itself is part of a multi-ray result: subset, Histogram3D bin,
    TOF in steps of 16 ps, then file order."""
    sc = yrt.Scanner("t", *SC_ARGS)
    pp = yrt.ProjectorParams(sc)
    pp.numRays = 3
    pp.addTOF(214.0, 5)
    p = yrt.DeviceProjector(sc, yrt.ImageParams(*IP_ARGS), pp)
    d1, d2 = random_events(20000, 61)
    tv = np.random.default_rng(62).normal(0, 300, len(d1)).astype(np.float32)
    S = 5
    out, _ = p.order_events(yrt.DeviceEvents.from_arrays(d1, d2, tof=tv), S)
    bins = yrt.histo3d_bins(sc, d1, d2).astype(np.int64)
    q = np.clip(np.floor(tv / np.float32(16) + np.float32(128)), 0, 255).astype(np.int64)
    want = np.lexsort((np.arange(len(d1)), q, bins, np.arange(len(d1)) % S))
    assert np.array_equal(out.perm.cpu().numpy(), want)


# Launches at and around the largest of the small form, with skipped events, a
# range that strides, frames, and every array of the EM pass: the same values as
# one crossing at a time (a set launch shape).
@pytest.mark.parametrize("precision", [L.YRTB_MIRROR, L.YRTB_COMPENSATED])
@pytest.mark.parametrize("tof", [None, (214.0, 5)])
@pytest.mark.parametrize("n", [1, 33, 4001, 32768, 32769, 131072, 131073])
def test_small_launches_equal_the_set_shape(precision, tof, n):
    sc = yrt.Scanner("t", *SC_ARGS)
    ip = yrt.ImageParams(36, 41, 15, 128, 128, 64, nt=2)
    pp = yrt.ProjectorParams(sc)
    pp.precision = precision
    if tof:
        pp.addTOF(*tof)
    rng = np.random.default_rng(n)
    d1, d2 = random_events(3 * n + 8, 60)
    m = 3 * n + 2
    d1, d2 = np.resize(d1, m), np.resize(d2, m)
    d1[5 % m] = 1 << 30  # no such crystal
    f32 = lambda lo, hi: rng.uniform(lo, hi, m).astype(np.float32)
    meas = rng.integers(0, 3, m).astype(np.float32)
    ev = yrt.DeviceEvents.from_arrays(
        d1, d2, tof=f32(-300, 300) if tof else None,
        frame=rng.integers(-1, 3, m).astype(np.int32), measurement=meas, sens=f32(0.5, 1.5),
        att=f32(0.2, 1), additive=f32(0.1, 0.2))
    r = L.yrtb_range(2, 3, n)
    x = torch.from_numpy(rng.random(ip.shape, np.float32)).cuda()
    y = torch.from_numpy(f32(0, 1)).cuda()
    out = {}
    # The default shape, the EM pass's batched form with its float4, pair and
    # scalar reductions, and float4 gathers with staged reductions, which neither
    # batch nor walk in lock step.
    for shape in (None, (256, 2), (128, 8), (128, 0), (256, 5)):
        p = yrt.DeviceProjector(sc, ip, pp)
        if shape:
            p.set_launch(shape[0], 1, 3, vector_groups=shape[1])
        fwd = p.forward(x, ev, out=torch.full((m,), -3.0, device="cuda"), rng=r)
        bwd = p.backward(y, ev, rng=r)
        em, model = torch.zeros_like(x), torch.full((m,), -3.0, device="cuda")
        p.em_step(x, em, ev, rng=r, global_scale=0.7, model=model)
        out[shape] = (fwd, model, bwd, em, p.take_event_errors())
    b = out.pop((256, 5))
    for a in out.values():
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
        assert a[4] == b[4]
        for i in (2, 3):  # the same terms, added in another order
            assert rel_l2(a[i].cpu().numpy(), b[i].cpu().numpy()) < 2 * n ** 0.5 * 2.0 ** -24


def launched_blocks(call):
    """Threads per block of the kernels that call launches (captured, not run)."""
    from cuda.bindings import driver as cu

    def ok(r):
        assert r[0] == cu.CUresult.CUDA_SUCCESS, r[0]
        return r[1:]

    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        ok(cu.cuStreamBeginCapture(stream.cuda_stream,
                                   cu.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED))
        try:
            call()
        finally:
            r = cu.cuStreamEndCapture(stream.cuda_stream)
    graph = ok(r)[0]
    count = ok(cu.cuGraphGetNodes(graph))[1]
    out = []
    for node in ok(cu.cuGraphGetNodes(graph, count))[0]:
        if ok(cu.cuGraphNodeGetType(node))[0] == cu.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            out.append(int(ok(cu.cuGraphKernelNodeGetParams(node))[0].blockDimX))
    ok(cu.cuGraphDestroy(graph))
    return out


# One-warp blocks for small launches and forward projections, as long as no shape
# was set; a shape that was set is the one that runs.
@pytest.mark.parametrize("precision", [L.YRTB_MIRROR, L.YRTB_COMPENSATED])
@pytest.mark.parametrize("tof", [None, (214.0, 5)])
def test_a_set_shape_is_launched(precision, tof):
    sc, ip, p = make(tof, precision)
    d1, d2 = random_events(5000, 63)
    tv = np.zeros(len(d1), np.float32) if tof else None
    ev = yrt.DeviceEvents.from_arrays(d1, d2, tof=tv)
    x = torch.ones(ip.shape, device="cuda")
    y, img = torch.ones(len(d1), device="cuda"), torch.zeros_like(x)
    calls = [lambda: p.forward(x, ev, out=y), lambda: p.backward(y, ev, img=img),
             lambda: p.em_step(x, img, ev)]
    assert [launched_blocks(c) for c in calls] == [[32]] * 3
    for block in (128, 256):
        for groups in (0, 2, 8):
            p.set_launch(block, 1, 3, vector_groups=groups)
            assert [launched_blocks(c) for c in calls] == [[block]] * 3
    default = yrt.DeviceProjector(sc, ip, p.proj_params).get_launch()
    p.set_launch(**default)
    assert [launched_blocks(c) for c in calls] == [[default["block"]]] * 3


def test_autotune_that_fails_leaves_the_launch_shape_unset():
    sc, ip, p = make((214.0, 5))
    d1, d2 = random_events(5000, 64)
    ev = yrt.DeviceEvents.from_arrays(d1, d2, tof=np.zeros(len(d1), np.float32))
    x, y = torch.ones(ip.shape, device="cuda"), torch.ones(len(d1), device="cuda")
    img = torch.zeros_like(x)
    before = p.get_launch()

    def tune():
        # A captured event has no time: the first measurement fails.
        with pytest.raises(yrt.YrtbError):
            p.autotune(x, ev)

    try:
        launched_blocks(tune)
    except AssertionError:
        pass  # the capture may be lost with it
    try:
        p.backward(y, ev, img=img)
    except yrt.YrtbError:
        pass  # what the lost capture left for the next launch's check
    assert p.get_launch() == before
    assert launched_blocks(lambda: p.backward(y, ev, img=img)) == [32]
    p.autotune(x, ev)
    assert launched_blocks(lambda: p.backward(y, ev, img=img)) == [p.get_launch()["block"]]


def kept_after(use):
    """Bytes of device memory that use() still holds once all it made is gone."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    yrt.release_cached_memory()
    before = torch.cuda.mem_get_info()[0]
    use()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return before - torch.cuda.mem_get_info()[0]


# The library's pool keeps at most small tables of a projector that is gone.
def test_large_tables_go_with_the_projector():
    sc, ip, _ = make()
    pp = yrt.ProjectorParams(sc)
    pp.numRays = 3

    def table():
        p = yrt.DeviceProjector(sc, ip, pp)
        p.multiray_table(1 << 20)    # 32 MB: pool
        p.multiray_table(1 << 23)    # 256 MB
        p.multiray_table(1 << 23)    # large enough already
        assert torch.equal(p.multiray_offsets(5), yrt.DeviceProjector(sc, ip, pp).multiray_offsets(5))

    assert kept_after(table) <= 64 << 20


def test_stored_sensitivity_values_go_with_the_projector():
    # 33M bins: 132 MB of values between the two passes.
    sc = yrt.Scanner("t", 100, 4, 3, 10, 250, 400, 20, 1, 19, 1, 1)
    ip = yrt.ImageParams(24, 24, 12, 240.0, 240.0, 90.0)
    assert yrt.Histogram3D(sc).histoSize * 4 > 64 << 20
    pp = yrt.ProjectorParams(sc)
    pp.deterministic = True
    mu = torch.rand(ip.shape, device="cuda") * 0.01
    out = {}

    def image(name, captured):
        p = yrt.DeviceProjector(sc, ip, pp)
        img = torch.zeros(ip.shape, device="cuda")
        torch.cuda.synchronize()
        call = lambda: p.sensitivity_histo3d(img, mu=mu, mu_params=ip)
        if captured:
            # A captured call holds no such buffer: both passes walk.
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                call()
            g.replay()
        else:
            call()
            img.zero_()
            call()
        torch.cuda.synchronize()
        out[name] = img.cpu()

    assert kept_after(lambda: image("stored", False)) <= 64 << 20
    image("walked", True)
    assert float(out["stored"].norm()) > 0 and torch.equal(out["stored"], out["walked"])


def test_multi_ray_table_is_not_made_under_capture():
    sc, ip, _ = make()
    pp = yrt.ProjectorParams(sc)
    pp.numRays = 3
    p = yrt.DeviceProjector(sc, ip, pp)

    def make_table(count):
        with pytest.raises(yrt.YrtbError, match="captured"):
            p.multiray_table(count)

    assert launched_blocks(lambda: make_table(100)) == []
    p.multiray_table(100)
    assert launched_blocks(lambda: p.multiray_table(50)) == []  # large enough already
    assert launched_blocks(lambda: make_table(200)) == []
    d1, d2 = random_events(200, 65)
    ev = yrt.DeviceEvents.from_arrays(d1, d2)
    x = torch.rand(ip.shape, device="cuda")
    # The first table still serves; item 100 on derive their offsets.
    assert torch.equal(p.forward(x, ev), yrt.DeviceProjector(sc, ip, pp).forward(x, ev))
