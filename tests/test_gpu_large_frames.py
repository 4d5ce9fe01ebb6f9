"""Frames large enough for the forms that only large frames take: their planes must equal those of
the batched kernels, which have one form for every size, bit for bit."""
import numpy as np
import pytest

import oracle
from raytracedgl1_gb300 import _native as N
from raytracedgl1_gb300.denoiser import Context, Denoiser, Stream, Tonemapping
from raytracedgl1_gb300.scene import Scene
from tests import _formats as F
from tests.test_gpu_parity import run_frames

pytestmark = pytest.mark.gpu


def table_config():
    """Every frame on the batched kernels, however large."""
    cfg = N.BatchConfig()
    cfg.atrousFusionDepth, cfg.tuned = 1, 1
    for i in range(6):
        cfg.atrousBlocksPerSM[i] = 3
    return cfg


# the L2 prefetch starts at 1 500 000 pixels: just above it, with a last block of 8 that is cut, an
# odd height, rows of 4-byte texels that start 8 bytes off a 16-byte unit; and just below it
@pytest.mark.parametrize("mode_name,mode", [("ref", N.STORAGE_REF), ("fp32", N.STORAGE_FP32), ("fp16", N.STORAGE_FP16), ("bf16", N.STORAGE_BF16)])
@pytest.mark.parametrize("size", [(1502, 1001), (1502, 997)])
def test_large_frame_equals_batched(mode_name, mode, size):
    W, H = size
    with Context(0) as ctx:
        ctx.set_batch_config(mode, table_config())
        sc = Scene(W, H, seed=71)
        a, b = Stream(ctx, W, H, mode), Stream(ctx, W, H, mode)
        for f in range(3):
            fi = f & 1
            bufs, p = sc.generate(f)
            p.atrousIterations = 5
            for s in (a, b):
                for name, arr in bufs.items():
                    s.upload(name, fi, arr)
            Denoiser(a).Denoise(fi, p)
            Tonemapping(a).CalculateExposure(fi, p)
            ctx.submit_batch([(b, fi, p)])
        for name in N.FB_NAMES:
            img = a.image(name, 0)
            if img.data:
                for slot in (0, 1) if img.has_prev else (0,):
                    assert np.array_equal(a.download(name, slot), b.download(name, slot)), (name, slot)
        assert a.tonemapping()[1] == b.tonemapping()[1]
        a.close()
        b.close()


@pytest.mark.parametrize("mode_name,mode", [("ref", N.STORAGE_REF), ("fp32", N.STORAGE_FP32), ("fp16", N.STORAGE_FP16), ("bf16", N.STORAGE_BF16)])
def test_large_frame_against_the_oracle(mode_name, mode):
    """The same forms against code that shares nothing with them, to the bounds of test_end_to_end."""
    W, H = 1502, 1001
    with Context(0) as ctx:
        sc = Scene(W, H, seed=71)
        s, o = Stream(ctx, W, H, mode), oracle.OracleStream(W, H, mode)
        fi = run_frames(s, o, sc, 3)
        img = s.image("PRE_FINAL", fi)
        g = F.decode(s.download("PRE_FINAL", fi), img.format)
        c = F.decode(o.plane("PRE_FINAL", fi), img.format)
        err = F.texel_rel_err(g, c, atol=1e-4 * float(np.percentile(c, 99)))
        if mode == N.STORAGE_FP32:
            assert err.max() <= 1e-3, f"max rel err {err.max():.3e}"
        else:
            assert np.mean(err <= 1e-2) >= 0.99, f"{np.mean(err <= 1e-2):.4f} of pixels within 1e-2"
            assert F.psnr(g, c) > 50.0
        s.close()
