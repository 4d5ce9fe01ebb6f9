"""The scattering accumulation reads its inputs while the volume pass runs: they must be those a kernel
wrote just before the call, and the volume the one this call integrates."""
import numpy as np
import pytest

from raytracedgl1_gb300 import _native as N
from raytracedgl1_gb300.denoiser import Context, Stream, Volumetric
from raytracedgl1_gb300.scene import Scene

pytestmark = pytest.mark.gpu

INPUTS = ("MOTION", "DEPTH_WORLD", "NORMAL", "DEPTH_NDC", "SCATTER_VOLUME")


@pytest.mark.parametrize("flags", [0, N.VOLUME_EXACT_MATH])
@pytest.mark.parametrize("size", [(1920, 1080), (34, 17)])
def test_scatter_inputs_written_by_a_kernel_just_before(flags, size):
    torch = pytest.importorskip("torch")
    W, H = size
    rng = np.random.default_rng(W + flags)
    nx, ny, nz = N.VOLUME_SIZE
    p = N.VolumetricParams()
    for m in (p.invView, p.invProjection, p.volumeViewProj):
        m[:] = np.eye(4, dtype=np.float32).reshape(-1)
    p.cameraPosition[:] = (0.0, 0.0, -1.0, 0.0)
    p.volumeCameraNear, p.volumeCameraFar, p.maxHistoryLength = 0.5, 3.0, 6.0
    p.volumeEnableType, p.frameId, p.flags = N.VOLUME_ENABLE_VOLUMETRIC, 9, flags
    sc = Scene(W, H, seed=4)
    frames = []
    for f in range(2):
        bufs, _ = sc.generate(f)
        d = {k: bufs[k] for k in INPUTS[:3]}
        d["DEPTH_NDC"] = rng.uniform(0.1, 0.9, (H, W)).astype(np.float32)
        d["SCATTER_VOLUME"] = rng.uniform(0.0, 0.2, (ny * nz, nx, 4)).astype(np.float16)
        frames.append({k: torch.from_numpy(np.ascontiguousarray(v).view(np.uint8).reshape(-1)).cuda() for k, v in d.items()})
    with Context(0) as ctx:
        out = []
        for waited in (True, False):
            s = Stream(ctx, W, H, N.STORAGE_FP16)
            bound = {}
            for k in INPUTS:
                for slot in (0, 1) if s.image(k, 0).has_prev else (0,):
                    bound[k, slot] = torch.zeros_like(frames[0][k])
                    s.bind(k, slot, bound[k, slot].data_ptr())
            torch.cuda.synchronize()
            for f in range(6):
                slot = f & 1
                for k in INPUTS:
                    # an elementwise kernel, not a copy engine
                    torch.bitwise_or(frames[slot][k], 0, out=bound[(k, slot) if (k, slot) in bound else (k, 0)])
                if waited:
                    torch.cuda.synchronize()
                Volumetric(s).ProcessScattering(slot, p)
                if waited:
                    torch.cuda.synchronize()
            torch.cuda.synchronize()
            out.append([s.download(k, i) for k in ("SCATTERING", "SCATTERING_HISTORY") for i in (0, 1)])
            s.close()
        for a, b in zip(*out):
            assert np.array_equal(a, b)


# four scenes over two slots: every copy changes the bytes of every plane, in the steady state too
@pytest.mark.parametrize("storage", [N.STORAGE_FP16, N.STORAGE_REF])
@pytest.mark.parametrize("size", [(1920, 1080), (34, 17)])
def test_scatter_inputs_that_change_every_frame(storage, size):
    torch = pytest.importorskip("torch")
    W, H = size
    rng = np.random.default_rng(W + storage)
    nx, ny, nz = N.VOLUME_SIZE
    p = N.VolumetricParams()
    for m in (p.invView, p.invProjection, p.volumeViewProj):
        m[:] = np.eye(4, dtype=np.float32).reshape(-1)
    p.cameraPosition[:] = (0.0, 0.0, -1.0, 0.0)
    p.volumeCameraNear, p.volumeCameraFar, p.maxHistoryLength = 0.5, 3.0, 6.0
    p.volumeEnableType, p.frameId = N.VOLUME_ENABLE_VOLUMETRIC, 9
    frames = []
    for f in range(4):
        bufs, _ = Scene(W, H, seed=4 + f).generate(f)
        d = {k: bufs[k] for k in INPUTS[:3]}
        d["DEPTH_NDC"] = rng.uniform(0.1, 0.9, (H, W)).astype(np.float32)
        d["SCATTER_VOLUME"] = rng.uniform(0.0, 0.2, (ny * nz, nx, 4)).astype(np.float16)
        frames.append({k: torch.from_numpy(np.ascontiguousarray(v).view(np.uint8).reshape(-1)).cuda() for k, v in d.items()})
    for k in INPUTS:
        assert all(not torch.equal(frames[f][k], frames[g][k]) for f in range(4) for g in range(f)), k
    with Context(0) as ctx:
        out = []
        for waited in (True, False):
            s = Stream(ctx, W, H, storage)
            bound = {}
            for k in INPUTS:
                for slot in (0, 1) if s.image(k, 0).has_prev else (0,):
                    bound[k, slot] = torch.zeros_like(frames[0][k])
                    s.bind(k, slot, bound[k, slot].data_ptr())
            torch.cuda.synchronize()
            for f in range(8):
                slot = f & 1
                for k in INPUTS:
                    torch.bitwise_or(frames[f % 4][k], 0, out=bound[(k, slot) if (k, slot) in bound else (k, 0)])
                if waited:
                    torch.cuda.synchronize()
                Volumetric(s).ProcessScattering(slot, p)
                if waited:
                    torch.cuda.synchronize()
            torch.cuda.synchronize()
            out.append([s.download(k, i) for k in ("SCATTERING", "SCATTERING_HISTORY") for i in (0, 1)])
            s.close()
        for a, b in zip(*out):
            assert np.array_equal(a, b)
