"""ProcessScattering on values at the ends of their range: froxels and histories that overflowed binary16,
and a history reset over a bright history, in all three forms of the accumulation."""
import numpy as np
import pytest

import oracle
from raytracedgl1_gb300 import _native as N
from raytracedgl1_gb300.denoiser import Context, Stream, Volumetric
from raytracedgl1_gb300.scene import Scene
from tests.test_gpu_parity import _volumetric_params, upload_frame

pytestmark = pytest.mark.gpu

# the default form, the IEEE form, the default form of a stream in the reference formats
FORMS = [("default", N.STORAGE_FP16, 0), ("exact", N.STORAGE_FP16, N.VOLUME_EXACT_MATH), ("ref", N.STORAGE_REF, 0)]
QUANTUM = 2.0 ** -9   # two binary16 quanta, as in the parity tests


def scattering(form, size, volume, previous, p):
    """(SCATTERING of the GPU, of the oracle) as floats: one frame over `previous`"""
    _, storage, flags = form
    W, H = size
    with Context(0) as ctx:
        s, o = Stream(ctx, W, H, storage), oracle.OracleStream(W, H, oracle.MODE_F32)
        upload_frame(s, o, {"SCATTER_VOLUME": volume.astype(np.float16).view(np.uint16)}, 0)
        rng = np.random.default_rng(3)
        upload_frame(s, o, {"SCATTERING": previous.astype(np.float16).view(np.uint16),
                            "SCATTERING_HISTORY": rng.uniform(1, 5, (H, W)).astype(np.float16).view(np.uint16)}, 1)
        sc = Scene(W, H, seed=W)
        for f in (1, 0):
            bufs, _ = sc.generate(f)
            upload_frame(s, o, {k: bufs[k] for k in ("NORMAL", "DEPTH_WORLD", "MOTION")}, f)
        upload_frame(s, o, {"DEPTH_NDC": rng.uniform(0.1, 0.9, (H, W)).astype(np.float32)}, 0)
        p.flags = flags
        Volumetric(s).ProcessScattering(0, p)
        o.process_scattering(0, p)
        g, c = (x.copy().view(np.float16).astype(np.float32) for x in (s.download("SCATTERING", 0), o.plane("SCATTERING", 0)))
        s.close()
    return g, c


@pytest.mark.parametrize("form", FORMS, ids=[f[0] for f in FORMS])
@pytest.mark.parametrize("size", [(64, 36), (50, 23)])
@pytest.mark.parametrize("vmode", [N.VOLUME_ENABLE_SIMPLE, N.VOLUME_ENABLE_VOLUMETRIC])
def test_infinities_stay_infinities(form, size, vmode):
    """Froxels that are Inf beside each other interpolate to Inf, an Inf history mixes to Inf: the texels
    that are Inf and those that are NaN (Inf with a weight of zero) are the oracle's, the rest within
    two quanta."""
    W, H = size
    nx, ny, nz = N.VOLUME_SIZE
    rng = np.random.default_rng(W + vmode)
    vol = np.concatenate([rng.uniform(0, 0.5, (nz, ny, nx, 3)), rng.uniform(0, 0.1, (nz, ny, nx, 1))], axis=3)
    # in-scatter only: an infinite extinction would extinguish all behind it
    vol[25:, ny // 4:ny // 2, nx // 4:nx // 2, :2] = np.inf
    prev = np.concatenate([rng.uniform(0, 1, (H, W, 3)), rng.uniform(0.2, 1, (H, W, 1))], axis=2)
    prev[H // 2:H // 2 + 8, W // 2:, 1:3] = np.inf
    g, c = scattering(form, size, vol.reshape(ny * nz, nx, 4), prev, _volumetric_params(vmode, 11))
    inf, nan = np.isinf(c), np.isnan(c)
    assert inf.sum() > 50 and np.isfinite(c).mean() > 0.5
    assert np.array_equal(np.isinf(g), inf), f"{(np.isinf(g) != inf).sum()} of {inf.sum()} texels' infinities"
    assert np.array_equal(np.isnan(g), nan), f"{(np.isnan(g) != nan).sum()} texels' NaN"
    fin = np.isfinite(c)
    scale = np.max(np.where(fin, np.abs(c), 0.0), axis=-1, keepdims=True)
    err = np.where(fin, np.abs(np.where(fin, g, 0.0) - np.where(fin, c, 0.0)), 0.0)
    assert np.all(err <= QUANTUM * scale + 1e-6), f"max error {(err / (scale + 1e-6)).max():.3e} of the texel's largest channel"


@pytest.mark.parametrize("form", FORMS, ids=[f[0] for f in FORMS])
@pytest.mark.parametrize("vmode", [N.VOLUME_ENABLE_NONE, N.VOLUME_ENABLE_SIMPLE, N.VOLUME_ENABLE_VOLUMETRIC])
def test_reset_over_a_bright_history(form, vmode):
    """maxHistoryLength 0 resets the history: the mix factor is 1 and nothing of the previous frame is
    left, not even the rounding of a difference with it. Each colour channel to two binary16 quanta and
    2^-20 (SIMPLE's 1 - exp( -depth density ): a few ulp of the exponential near 1)."""
    W, H = 64, 36
    nx, ny, nz = N.VOLUME_SIZE
    rng = np.random.default_rng(vmode + 1)
    vol = np.concatenate([rng.uniform(0, 1e-4, (ny * nz, nx, 3)), rng.uniform(0, 0.1, (ny * nz, nx, 1))], axis=2)
    prev = np.concatenate([rng.uniform(3e4, 6e4, (H, W, 3)), rng.uniform(0.2, 1, (H, W, 1))], axis=2)
    p = _volumetric_params(vmode, 12)
    p.maxHistoryLength = 0.0
    g, c = scattering(form, (W, H), vol, prev, p)
    err = np.abs(g - c)
    assert np.all(err <= QUANTUM * np.abs(c) + 2.0 ** -20), f"max error {err.max():.3e}"
