"""The projection operator (ProjectionOper A / At) on list-mode and histogram
data, as the reference's integration helpers check it
(integration_tests/helper.py:43-89): the subsets' projections add up to the
full projection, and each operator satisfies <A x, y> = <x, A^T y>.

Tolerances: the subset sum is bit-exact here (every bin's projection is
computed the same way whatever subset it is in; the reference allows
allclose); the adjoint identity to 1e-6 relative in FP64 (the reference
allows 1e-3).  Multi-ray offsets follow an event's index in the call, as in
the reference device path, so for multi-ray only the adjoint identity holds
per subset.
"""
import numpy as np
import pytest
import torch  # noqa: F401  (CUDA context for the operator)

import pyyrtpet_b200 as yrt
from pyyrtpet_b200 import _lib as L

pytestmark = pytest.mark.gpu

SC_ARGS = ("s", 20, 4, 4, 10, 150, 64, 5, 1, 4, 2, 1)   # 64 x 5 crystals, every ring difference
IP_ARGS = (32, 32, 8, 160, 160, 20)


def _data(kind, tof):
    sc = yrt.Scanner(*SC_ARGS)
    rng = np.random.default_rng(61)
    if kind == "histogram":
        return sc, yrt.Histogram3D(sc)
    n = 20000
    d1 = rng.integers(0, sc.getNumDets(), 3 * n).astype(np.uint32)
    d2 = rng.integers(0, sc.getNumDets(), 3 * n).astype(np.uint32)
    keep = (d1 % 64) != (d2 % 64)
    lm = yrt.ListModeLUT(sc, tof, False)
    lm.allocate(n)
    lm.d1[:] = d1[keep][:n]
    lm.d2[:] = d2[keep][:n]
    if tof:
        lm.tof[:] = rng.normal(0, 150, n).astype(np.float32)
    return sc, lm


CASES = [("listmode", "Siddon", False, 1), ("listmode", "Siddon", True, 1),
         ("listmode", "DD", False, 1), ("listmode", "Siddon", False, 4),
         ("histogram", "Siddon", False, 1), ("histogram", "DD", False, 1),
         ("histogram", "Siddon", False, 4)]


@pytest.mark.parametrize("kind,projector,tof,rays", CASES)
def test_projection_oper_subsets_and_adjoint(kind, projector, tof, rays):
    sc, data = _data(kind, tof)
    ip = yrt.ImageParams(*IP_ARGS)
    kw = dict(projector=projector, num_rays=rays)
    if tof:
        kw.update(tof_width_ps=214.0, tof_n_std=5)
    rng = np.random.default_rng(62)
    x = rng.random((ip.nz, ip.ny, ip.nx)).astype(np.float32)
    y = rng.random(data.count()).astype(np.float32)
    k = yrt.ProjectionOper(sc, ip, data, **kw)
    Ax = k.A(x)
    assert Ax.shape == (data.count(),) and np.count_nonzero(Ax) > 0
    Aty = k.At(y)
    lhs = float(np.dot(Ax.astype(np.float64), y))
    rhs = float(np.sum(x.astype(np.float64) * Aty.reshape(x.shape)))
    assert abs(lhs - rhs) <= 1e-6 * abs(lhs)
    S = 4
    Ax_sub = np.zeros_like(Ax)
    for s in range(S):
        ks = yrt.ProjectionOper(sc, ip, data, idx_subset=s, num_subsets=S, **kw)
        Ax_s = ks.A(x)
        Ax_sub += Ax_s
        Aty_s = ks.At(y)
        lhs = float(np.dot(Ax_s.astype(np.float64), y))
        rhs = float(np.sum(x.astype(np.float64) * Aty_s.reshape(x.shape)))
        assert abs(lhs - rhs) <= 1e-6 * abs(lhs)
    if rays == 1:
        assert np.array_equal(Ax_sub, Ax)


@pytest.mark.parametrize("kind", ["listmode", "histogram"])
def test_operator_projector_device_reference_signatures(kind):
    # OperatorProjectorDevice with the reference's pybind signatures
    # (src/operators/OperatorProjectorDevice.cu:26-90): applyA(img, proj)
    # writes into a ProjectionList (entries of other subsets untouched),
    # applyAH(proj, img) adds into img; same values as ProjectionOper.
    sc, data = _data(kind, False)
    ip = yrt.ImageParams(*IP_ARGS)
    pp = yrt.ProjectorParams(sc)
    it = data.getBinIter(3, 1)
    op = yrt.OperatorProjectorDevice.create(pp, it, img_params=ip)
    rng = np.random.default_rng(62)
    x = torch.from_numpy(rng.random(ip.shape, dtype=np.float32)).cuda()
    pl = yrt.ProjectionListOwned(data)
    pl.allocate()
    pl.clearProjections(-1.0)
    op.applyA(x, pl)
    A = yrt.ProjectionOper(sc, ip, data, idx_subset=1, num_subsets=3)
    ref = A.A(x.cpu().numpy())
    idx = np.asarray(it.indices()) if kind == "histogram" else np.arange(1, data.count(), 3)
    got = pl.getProjectionsArray()
    assert np.array_equal(got[idx], ref[idx])
    outside = np.setdiff1d(np.arange(data.count()), idx)
    assert np.all(got[outside] == -1.0)
    y = yrt.ProjectionListOwned(data)
    y.allocate()
    y.values.copy_(torch.from_numpy(rng.random(data.count(), dtype=np.float32)))
    img = torch.zeros(ip.shape, device="cuda")
    op.applyAH(y, img)
    bp = A.At(y.getProjectionsArray())
    assert np.allclose(img.cpu().numpy(), bp, rtol=1e-5, atol=1e-6)
    with pytest.raises(RuntimeError):
        op.applyA(x, data)          # a ProjectionList receives the values


# Subsets of one or many phi, a subset with fewer phi than the others, both
# precisions and every projector (DD with a kernel that is not symmetric); the
# lists of crystal pairs are the oracle.  Values up to 1, and a large one on a
# bin that misses the grid, which must not set the scale of the others.
@pytest.mark.parametrize("projector,rays", [("S", 1), ("S", 3), ("DD", 1), ("DD+PSF", 1)])
@pytest.mark.parametrize("comp,det", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("subsets,subset", [(1, 0), (7, 6), (32, 31)])
def test_histogram_bins_equal_crystal_pairs(projector, rays, comp, det, subsets, subset):
    sc = yrt.Scanner("t", 40, 4, 4, 10, 100, 32, 6, 1, 4, 3, 1)
    ip = yrt.ImageParams(21, 18, 10, 105.0, 90.0, 40.0)
    pp = yrt.ProjectorParams(sc)
    pp.setProjector(projector[:2] if projector != "S" else "S")
    if projector == "DD+PSF":
        k = np.roll(np.exp(-0.5 * ((np.arange(17) - 8) * 0.6 / 1.7) ** 2), 1)
        pp.setProjPsf(30.0, 0.6, np.stack([k, k[::-1] ** 2]).astype(np.float32))
    pp.numRays = rays
    pp.precision = L.YRTB_COMPENSATED if comp else L.YRTB_MIRROR
    pp.deterministic = det
    h = yrt.Histogram3D(sc)
    it = h.getBinIter(subsets, subset)
    rng = np.random.default_rng(subsets)
    x = torch.from_numpy(rng.random(ip.shape, np.float32)).cuda()
    w = torch.from_numpy(rng.random(h.histoSize, np.float32)).cuda()
    p = yrt.DeviceProjector(sc, ip, pp)
    bins = it.indices()
    ev = yrt.DeviceEvents.from_arrays(*yrt.histo3d_detpairs(sc, bins))
    idx = torch.from_numpy(bins).cuda()
    want = torch.full((h.histoSize,), -7.0, device="cuda")
    want[idx] = p.forward(x, ev)
    miss = torch.nonzero(want[idx] == 0).reshape(-1)
    if miss.numel():
        w[idx[miss[0]]] = 1e12
    want_img = p.backward(w[idx].contiguous(), ev)
    assert float(want_img.max()) > 0
    op = yrt.OperatorProjectorDevice.create(pp, it, img_params=ip)
    got = yrt.ProjectionList(h)
    got.values = torch.full((h.histoSize,), -7.0, device="cuda")
    op.applyA(x, got)
    assert torch.equal(got.values, want)
    img = torch.zeros(ip.shape, device="cuda")
    got.values = w.clone()
    op.applyAH(got, img)
    if det:
        assert torch.equal(img, want_img)  # fixed-point sums: any order
    else:
        # Positive terms in another order: each of the up to n additions
        # rounds by half an ulp, at random (sqrt(n)) rather than all one way.
        n = len(bins)
        assert float((img - want_img).norm() / want_img.norm()) < n ** 0.5 * 2.0 ** -24 + 1e-6
    assert torch.equal(got.values, w)


def test_histogram_bins_refuse_what_crystal_pairs_refuse():
    sc = yrt.Scanner("t", 40, 4, 4, 10, 100, 32, 6, 1, 4, 3, 1)
    ip = yrt.ImageParams(8, 8, 4, 80.0, 80.0, 40.0)
    h = yrt.Histogram3D(sc)
    pp = yrt.ProjectorParams(sc)
    pp.addTOF(214.0, 5)
    op = yrt.OperatorProjectorDevice.create(pp, h.getBinIter(2, 0), img_params=ip)
    vals = yrt.ProjectionList(h)
    vals.allocate()
    with pytest.raises(RuntimeError, match="requires per-event TOF values"):
        op.applyA(torch.zeros(ip.shape, device="cuda"), vals)
    with pytest.raises(RuntimeError, match="requires per-event TOF values"):
        op.applyAH(vals, torch.zeros(ip.shape, device="cuda"))


# Rows of a multiple of 4 voxels take the float4 form of the distance-driven
# walk; images that start between 16-byte boundaries take the scalar one.
@pytest.mark.parametrize("dims,lengths,mrd", [((40, 36, 12), (160.0, 150.0, 40.0), 4),
                                              ((8, 9, 30), (150.0, 150.0, 60.0), 4),
                                              ((4, 4, 3), (200.0, 200.0, 12.0), 0)])
def test_dd_psf_histogram_quads_equal_scalar(dims, lengths, mrd):
    sc = yrt.Scanner("t", 40, 4, 4, 10, 100, 48, 6, 1, mrd, 3, 1)
    ip = yrt.ImageParams(*dims, *lengths)
    pp = yrt.ProjectorParams(sc)
    pp.setProjector("DD")
    pp.precision = L.YRTB_COMPENSATED
    k = np.exp(-0.5 * ((np.arange(17) - 8) * 0.6 / 1.7) ** 2)
    taps = np.stack([k, np.roll(k, 1)]) / (k.sum() * 0.6)  # the second row is not symmetric
    pp.setProjPsf(30.0, 0.6, taps.astype(np.float32))
    p = yrt.DeviceProjector(sc, ip, pp)
    h = yrt.Histogram3D(sc)
    rng = np.random.default_rng(dims[0])
    meas = torch.from_numpy(rng.poisson(1.0, h.histoSize).astype(np.float32)).cuda()
    n = ip.numVoxels
    x = torch.from_numpy(0.2 + rng.random(n + 1, np.float32)).cuda()

    def em(first):
        img = torch.empty(n + 1, device="cuda")[first:first + n].copy_(x[:n])
        buf = torch.zeros(n + 9, device="cuda")
        p.em_step_histo3d(img, buf[first:first + n], meas, 3, 1)
        assert not buf[first + n:].any() and not buf[:first].any()
        return buf[first:first + n].double()

    quads, scalar = em(0), em(1)
    assert float(scalar.norm()) > 0
    # The weights differ by the rounding of tap coordinates counted from
    # another voxel (2 ulp of up to 18 taps, 0.25 of a tap's weight each).
    assert float((quads - scalar).norm() / scalar.norm()) < 3e-6


# An EM ratio that overflows reaches the voxels its line crosses, as in the
# scalar form, not the rest of their float4 groups.
@pytest.mark.parametrize("ratio", [np.inf, np.nan])
def test_dd_psf_histogram_quads_keep_infinite_ratios_on_their_lines(ratio):
    sc = yrt.Scanner("t", 40, 4, 4, 10, 100, 48, 6, 1, 4, 3, 1)
    ip = yrt.ImageParams(40, 36, 12, 160.0, 150.0, 40.0)
    pp = yrt.ProjectorParams(sc)
    pp.setProjector("DD")
    pp.precision = L.YRTB_COMPENSATED
    k = np.exp(-0.5 * ((np.arange(9) - 4) * 0.6 / 1.2) ** 2)
    pp.setProjPsf(300.0, 0.6, (k / (k.sum() * 0.6)).astype(np.float32)[None])
    p = yrt.DeviceProjector(sc, ip, pp)
    h = yrt.Histogram3D(sc)
    n = ip.numVoxels
    x = torch.full((n + 1,), 1e-30, device="cuda")
    for b in range(7, h.histoSize, h.histoSize // 40):  # lines along both axes
        meas = torch.zeros(h.histoSize, device="cuda")

        def em(m, first):  # first = 1: the scalar form
            meas[b] = m
            buf = torch.zeros(n + 1, device="cuda")
            p.em_step_histo3d(x[first:first + n], buf[first:first + n], meas, 1, 0)
            return buf[first:first + n]

        # 1e38 / 1e-28 overflows.
        m = 1e38 if np.isinf(ratio) else np.nan
        bad = ~em(m, 0).isfinite()
        assert torch.equal(bad, ~em(m, 1).isfinite())
        # The whole line (and voxels that its rows end in with weight 0).
        assert bool(bad[em(1.0, 1) != 0].all()) and not bad.all()


def test_dd_psf_weights_are_as_exact_as_their_arithmetic():
    # Lines along x, so that a footprint's edges are FP32 numbers known here, on
    # voxels whose edges are whole: what rounds is the integral of the kernel
    # (4 mm FWHM, taps of 0.5 mm) over each voxel.
    sc = yrt.Scanner("t", 8, 2, 1, 10, 200, 16, 1, 1, 0, 1, 1)
    ip = yrt.ImageParams(4, 48, 1, 4.0, 48.0, 8.0)
    pp = yrt.ProjectorParams(sc)
    pp.setProjector("DD")
    pp.precision = L.YRTB_COMPENSATED
    half, step = 11, 0.5
    g = np.exp(-0.5 * (np.arange(-half, half + 1) * step * 2.3548 / 4.0) ** 2)
    taps = (g / (g.sum() * step)).astype(np.float32)
    pp.setProjPsf(1e9, step, taps[None])
    p = yrt.DeviceProjector(sc, ip, pp)
    n = 4000
    y = np.random.default_rng(71).uniform(-20, 20, n).astype(np.float32)
    lor, orient = np.zeros((n, 6), np.float32), np.zeros((n, 6), np.float32)
    lor[:, 0], lor[:, 3], lor[:, 1], lor[:, 4] = 200, -200, y, y
    orient[:, 0], orient[:, 3] = 1, -1
    ev = yrt.DeviceEvents.from_arrays(lor=lor, orient=orient)
    offs, wts, cnt = (t.cpu().numpy() for t in p.trace_walks(ev, cap=256))
    near, far = (y - np.float32(0.5)).astype(np.float64), (y + np.float32(0.5)).astype(np.float64)

    def integral(x):  # of the taps' polygon from far left to x mm from the centre
        v = np.concatenate([[0, 0], taps.astype(np.float64), [0]])
        whole = np.concatenate([[0, 0], np.cumsum((v[2:] + v[1:-1]) * step / 2)])
        u = np.clip(x / step, -half - 1, half + 1)
        i = np.minimum(np.floor(u).astype(int), half) + half + 2
        t = u - (i - half - 2)
        return whole[i] + step * (v[i] * t + (v[np.minimum(i + 1, len(v) - 1)] - v[i]) * t * t / 2)

    on = np.arange(offs.shape[1])[None] < cnt[:, None]
    assert on.sum(1).min() > 40
    edge = (offs // 4 - 24).astype(np.float64)
    want = (integral(edge + 1 - near[:, None]) - integral(edge - far[:, None]))[on]
    got = (wts.astype(np.float64) * (far - near)[:, None])[on]  # rows 1 mm long, one plane
    assert want.max() > 0.2
    # About four roundings of a weight (its parts, their sum, the row's factor):
    # half an ulp at random, 2^-25 to 2^-24 of it.
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < 2 * 2.0 ** -24.5 / 3 ** 0.5
