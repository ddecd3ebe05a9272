"""Arrays in device memory: converted in place by uploads and downloads, and
read by the flux call through tensor maps where their alignment allows it."""
import numpy as np
import pytest

from raishinsource_b200 import RgError, config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,offset", [(dict(nr=41, nth=23, nph=13), 0), (dict(nr=40, nth=24, nph=16), 1),
                                       (dict(nr=48, nth=40), 0), (dict(nr=48, nth=40, precision="mixed"), 1)])
def test_device_upload_and_download_equal_host(gpu_ctx, kw, offset):
    """Any double alignment (offset doubles into an allocation), odd extents,
    slabs stored as one plane and the mixed layout."""
    import torch
    r = gpu_ctx.admit(dict(config.torus(**kw), guard=1))
    r.ic_torus(seed=9)
    u = r.prims()
    buf = torch.zeros(u.size + offset, dtype=torch.float64, device="cuda")
    buf[offset:] = torch.from_numpy(u.ravel())
    torch.cuda.synchronize()
    r.step(1)
    r.upload_prims_ptr(buf.data_ptr() + 8 * offset, t0=0.5)
    out = torch.full_like(buf, float("nan"))
    torch.cuda.synchronize()  # the download runs on the context's stream, which does not wait for torch's
    r.download_prims_ptr(out.data_ptr() + 8 * offset)
    assert np.array_equal(out[offset:].cpu().numpy(), u.ravel())
    r.step(1)
    a = r.prims()
    r.upload_prims(u, t0=0.5)
    r.step(1)
    assert np.array_equal(a, r.prims())
    assert r.stats()["time"] > 0.5
    r.release()


@pytest.mark.parametrize("where", ["pinned", "device"])
def test_upload_has_read_the_array_when_it_returns(gpu_ctx, where):
    """A 3D run (no uniformity check to wait for), with steps queued ahead of
    the upload: the array is overwritten as soon as the call returns."""
    import torch
    r = gpu_ctx.admit(dict(config.torus(nr=96, nth=64, nph=48), guard=1))
    r.ic_torus(seed=9)
    u = torch.from_numpy(r.prims())
    buf = u.clone().pin_memory() if where == "pinned" else u.cuda()
    torch.cuda.synchronize()
    r.step(20)
    r.upload_prims_ptr(buf.data_ptr(), t0=0.0)
    buf.fill_(-7.0)
    assert np.array_equal(r.prims(), u.numpy())
    r.release()


def test_device_upload_refuses_a_slab_that_is_not_uniform(gpu_ctx):
    import torch
    r = gpu_ctx.admit(dict(config.torus(nr=48, nth=40), guard=1))
    r.ic_torus(seed=9)
    u = torch.from_numpy(r.prims()).cuda()
    u[3, 1, 5, 0] += 1e-13  # one cell of one phi plane
    torch.cuda.synchronize()
    with pytest.raises(RgError) as e:
        r.upload_prims_ptr(u.data_ptr())
    assert e.value.code == 1
    r.release()


@pytest.mark.parametrize("nr,nth,nph,offset", [(64, 24, 17, 0), (64, 24, 17, 1), (41, 24, 17, 0)])
def test_static_fluxes_whatever_the_alignment(gpu_ctx, nr, nth, nph, offset):
    """Staged (16-byte aligned, imax a multiple of 4) or direct, the fluxes are
    rg_calflx's to rounding."""
    import torch
    r = gpu_ctx.admit(dict(config.torus(nr=nr, nth=nth, nph=nph), guard=1))
    r.ic_torus(seed=9)
    u = r.prims()
    n = u.size // 9
    want = r.calflx(u)
    buf = torch.zeros(9 * n + offset, dtype=torch.float64, device="cuda")
    buf[offset:] = torch.from_numpy(np.ascontiguousarray(u.reshape(n, 9).T).ravel())
    ww = torch.zeros(3, 9, *u.shape[:3], dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    r.calflx_static(buf.data_ptr() + 8 * offset, ww.data_ptr())
    got = np.moveaxis(ww.cpu().numpy(), (0, 1), (4, 3))
    m = r.nm1 - 1
    a, b = got[m:-m - 1, m:-m - 1, m:-m - 1], want[m:-m - 1, m:-m - 1, m:-m - 1]
    scale = np.abs(b).max(axis=(0, 1, 2, 4))[:, None]
    assert (np.abs(a - b).max(axis=(0, 1, 2)) / np.maximum(scale, 1e-300)).max() < 1e-12
    r.release()
