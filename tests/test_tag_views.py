"""tag_cells on tensors that are not the plain case: the copies it makes of strided views must live until the kernel
has been launched, and the kernel writes tags of the level's shape on the state's device, whatever tags the caller holds."""
import ctypes
import types
import weakref

import pytest
import torch

from hydroexa_gb300 import capi, solver
from hydroexa_gb300.level import Geometry
from hydroexa_gb300.params import PhysicsParameters

NX, NY = 37, 21
TH = PhysicsParameters(h_grad_thresh=[3.0], umag_grad_thresh=[8.0], z_grad_thresh=[2.5])


def cropped(a, dtype=torch.float64):
    """The values of ``a`` as the inner part of a padded tensor, as a level's valid cells lie in their ghosts."""
    big = torch.full((a.shape[0], a.shape[1] + 2, a.shape[2] + 6), 7.0, dtype=dtype, device=a.device)
    big[:, 1:-1, 2:-4] = a
    return big[:, 1:-1, 2:-4]


@pytest.fixture
def call(monkeypatch):
    """tag_cells on host tensors with the library call replaced by one that looks at what it is handed."""
    seen = types.SimpleNamespace(tensors=[], devices=set(), arrays=None)
    real = solver.array4

    def array4(t, *a):
        seen.tensors.append(weakref.ref(t))
        seen.devices.add(t.device.type)
        return real(t, *a)

    def tag(method, U, T, tags, *rest):
        assert all(r() is not None for r in seen.tensors), "a tensor was freed before the launch"
        assert len(seen.devices) == 1, "tensors of different devices"
        seen.arrays = [x._obj for x in (U, T, tags)]
        a = seen.arrays[2]
        assert (a.lo[0], a.lo[1], a.hi[0], a.hi[1]) == (0, 0, NX - 1, NY - 1), "tags of another shape"
        ctypes.memset(seen.arrays[2].p, 1, NX * NY)
        return 0

    monkeypatch.setattr(solver, "array4", array4)
    monkeypatch.setattr(capi, "lib", lambda: types.SimpleNamespace(hx_tag_level_f64=tag, hx_tag_level_f32=tag))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: types.SimpleNamespace(cuda_stream=0))

    def run(tags, U, T):
        solver.HydrostaticRoe().tag_cells(tags, U, T, Geometry(NX, NY, 0.1, 0.13), 0, 0.0, TH)
        return seen
    return run


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_copies_of_views_live_until_the_launch(call, dtype):
    U, T = (torch.rand((k, NY, NX), dtype=dtype) for k in (3, 2))
    tags = torch.zeros((NY, NX), dtype=torch.int8)
    call(tags, cropped(U, dtype), cropped(T, dtype))
    assert (tags == 1).all()


def test_tags_of_another_device_are_copied(call):
    """Meta tensors stand for the other device: they have no data to copy, so an attempt to copy them raises."""
    U, T = (torch.rand((k, NY, NX), dtype=torch.float64) for k in (3, 2))
    with pytest.raises(NotImplementedError):
        call(torch.zeros((NY, NX), dtype=torch.int8, device="meta"), U, T)


@pytest.mark.parametrize("shape", [(NY, NX), (1, NY, NX), (1, 1, NY, NX), (NY + 1, NX), (NY, NX + 3), (2, NY, NX), (NY, 1), (NX * NY,)])
@pytest.mark.parametrize("dtype", [torch.int8, torch.int32])
def test_tags_have_the_level_shape(call, shape, dtype):
    U, T = (torch.rand((k, NY, NX), dtype=torch.float64) for k in (3, 2))
    tags = torch.zeros(shape, dtype=dtype)
    if shape[-2:] == (NY, NX) and tags.numel() == NY * NX:
        call(tags, U, T)
        assert (tags == 1).all()
    else:
        with pytest.raises(RuntimeError):
            call(tags, U, T)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.int8, torch.int32])
def test_host_tags_are_written_back(cuda, hxlib, dtype):
    g = torch.Generator(device="cuda").manual_seed(4)
    U, T = (torch.rand((k, NY, NX), dtype=torch.float64, device=cuda, generator=g) for k in (3, 2))
    a, b = torch.zeros((NY, NX), dtype=torch.int8, device=cuda), torch.zeros((NY, NX), dtype=dtype)
    a[3, 4] = b[3, 4] = 5  # what was tagged stays tagged
    for tags in (a, b):
        solver.HydrostaticRoe().tag_cells(tags, U, T, Geometry(NX, NY, 0.1, 0.13), 0, 0.0, TH)
    assert torch.equal(a.cpu(), b.to(torch.int8)) and 0 < int((a == 2).sum()) < NX * NY


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_views_give_the_tags_of_their_copies(cuda, hxlib, dtype):
    g = torch.Generator(device="cuda").manual_seed(3)
    U, T = (torch.rand((k, NY, NX), dtype=dtype, device=cuda, generator=g) for k in (3, 2))
    out = []
    for u, t in ((U, T), (cropped(U, dtype), cropped(T, dtype)), (U.transpose(1, 2).contiguous().transpose(1, 2), T)):
        tags = torch.zeros((NY, NX), dtype=torch.int8, device=cuda)
        solver.HydrostaticRoe().tag_cells(tags, u, t, Geometry(NX, NY, 0.1, 0.13), 0, 0.0, TH)
        out.append(tags.cpu())
    assert 0 < int((out[0] == 2).sum()) < NX * NY
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
