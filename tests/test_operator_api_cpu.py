"""Host-side checks of the OperatorProjectorDevice mirror (no GPU needed):
the arguments it cannot honour raise instead of being dropped."""
import pytest
import torch

import pyyrtpet_b200 as yrt
from pyyrtpet_b200 import _lib as L


def test_create_rejects_constraints_and_memory_budget():
    sc = yrt.Scanner("s", 20, 4, 4, 10, 150, 64, 5, 1, 4, 2, 1)
    pp = yrt.ProjectorParams(sc)
    h = yrt.Histogram3D(sc)
    it = h.getBinIter(1, 0)
    op = yrt.OperatorProjectorDevice.create(pp, it)
    assert op.getBinIter() is it
    with pytest.raises(RuntimeError, match="constraints"):
        yrt.OperatorProjectorDevice.create(pp, it, constraints=[object()])
    with pytest.raises(RuntimeError, match="mem_available"):
        yrt.OperatorProjectorDevice.create(pp, it, mem_available=1 << 30)


def test_projection_list_requires_allocation():
    sc = yrt.Scanner("s", 20, 4, 4, 10, 150, 64, 5, 1, 4, 2, 1)
    pl = yrt.ProjectionListOwned(yrt.Histogram3D(sc))
    with pytest.raises(RuntimeError, match="not allocated"):
        pl.getProjectionValue(0)


class FakeCuda:
    """Stands in for a CUDA tensor: what the argument checks look at."""

    is_cuda, requires_grad = True, False

    def __init__(self, n, device="cuda:0", dtype=torch.float32, contiguous=True):
        self.n, self.device, self.dtype, self.c = n, torch.device(device), dtype, contiguous

    def numel(self):
        return self.n

    def dim(self):
        return 1

    def is_contiguous(self):
        return self.c

    def contiguous(self):
        return self

    def data_ptr(self):
        return 1 << 20


class FakeLib:
    """Library that must not be given a pointer."""

    def __init__(self, real):
        self.yrtb_histo3d_dims = real.yrtb_histo3d_dims

    def yrtb_projector_get_image_layout(self, h, out):
        return 0

    def __getattr__(self, name):
        raise AssertionError(f"{name} was called")


def _projector_without_gpu(monkeypatch):
    sc = yrt.Scanner("s", 20, 4, 4, 10, 150, 64, 5, 1, 4, 2, 1)
    p = yrt.DeviceProjector.__new__(yrt.DeviceProjector)
    p.h, p.scanner, p.img_params = None, sc, yrt.ImageParams(4, 4, 4, 8, 8, 8)
    p.proj_params = yrt.ProjectorParams(sc)
    h = yrt.Histogram3D(sc)
    fake = FakeLib(L.lib())
    monkeypatch.setattr(L, "lib", lambda: fake)
    monkeypatch.setattr("pyyrtpet_b200.core._stream", lambda: None)
    return p, h


# The kernels write and read a value per bin of the histogram through the
# pointer they are given.
@pytest.mark.parametrize("bad,match", [
    (dict(n=-1), "bin values, expected"), (dict(n=1), "bin values, expected"),
    (dict(device="cuda:1"), "cuda:1"), (dict(dtype=torch.float64), "contiguous float32"),
    (dict(contiguous=False), "contiguous float32"),
])
def test_histogram_projection_checks_the_values(monkeypatch, bad, match):
    p, h = _projector_without_gpu(monkeypatch)
    img = FakeCuda(64)
    values = FakeCuda(**{"n": h.histoSize, **bad, **({"n": h.histoSize + bad["n"]} if "n" in bad
                                                     else {})})
    with pytest.raises(RuntimeError, match=match):
        p.forward_histo3d(img, values)
    with pytest.raises(RuntimeError, match=match):
        p.backward_histo3d(values, img)
    with pytest.raises(RuntimeError, match="contiguous float32"):
        p.forward_histo3d(img, torch.zeros(h.histoSize))  # host memory


def test_operator_lists_the_bins_of_values_on_another_device(monkeypatch):
    p, h = _projector_without_gpu(monkeypatch)
    op = yrt.OperatorProjectorDevice(p.proj_params, h.getBinIter(2, 0), p.img_params)
    op._proj = p
    h.scanner = p.scanner

    def events(data):
        raise RuntimeError("listed")

    monkeypatch.setattr(op, "_events", events)
    monkeypatch.setattr(op, "_check_image", lambda img, proj: None)
    vals = yrt.ProjectionList(h)
    vals.values = FakeCuda(h.histoSize, device="cuda:1")
    with pytest.raises(RuntimeError, match="listed"):
        op.applyA(FakeCuda(64), vals)
    with pytest.raises(RuntimeError, match="listed"):
        op.applyAH(vals, FakeCuda(64))
    vals.values = FakeCuda(h.histoSize)
    with pytest.raises(AssertionError, match="yrtb_forward_histo3d was called"):
        op.applyA(FakeCuda(64), vals)
