"""The packed colour formats' device codecs, over every code, against the oracle and the plain kernels."""
import numpy as np
import pytest

import oracle
from raytracedgl1_gb300 import _native as N
from raytracedgl1_gb300.denoiser import Context, Denoiser, Stream
from raytracedgl1_gb300.scene import Scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode_name,mode,omode", [("ref", N.STORAGE_REF, oracle.MODE_REF), ("fp32", N.STORAGE_FP32, oracle.MODE_F32)])
@pytest.mark.parametrize("albedo_from_codes", [False, True])
def test_b10g11r11_codes(mode_name, mode, omode, albedo_from_codes):
    """Sky pixels compose to albedo * throughput: every B10G11R11 code as the albedo (decode), and every
    binary16 as the throughput (encode in the reference formats: subnormals, ties, overflow, Inf, NaN,
    negative values)."""
    W, H = 256, 256
    bufs, p = Scene(W, H, seed=5).generate(0)
    i = np.arange(W * H, dtype=np.uint32).reshape(H, W)
    bufs["IS_SKY"][:] = 1
    bufs["ALBEDO"][:] = ((i % 2048) | ((i * 7 % 2048) << 11) | ((i % 1024) << 22)) if albedo_from_codes else 0x3C0 | (0x3B5 << 11) | (0x1E3 << 22)
    bufs["THROUGHPUT"][..., :3] = 0x3C00 if albedo_from_codes else np.stack([i, i * 5, i * 3], -1).astype(np.uint16)
    with Context(0) as ctx:
        s, o = Stream(ctx, W, H, mode), oracle.OracleStream(W, H, omode)
        for name, arr in bufs.items():
            s.upload(name, 0, arr)
            o.load(name, 0, arr)
        Denoiser(s).Denoise(0, p)
        o.denoise(0, p)
        g, c = s.download("PRE_FINAL", 0), o.plane("PRE_FINAL", 0)
        same = (g == c) if mode == N.STORAGE_REF else (g == c) | (np.isnan(g) & np.isnan(c))
        assert same.all(), np.argwhere(~same)[:5]
        s.close()


# one tile, cut tiles, several tiles with an odd height
@pytest.mark.parametrize("size", [(2, 1), (32, 32), (34, 33), (98, 67)])
@pytest.mark.parametrize("spread", [32, 3])
def test_shared_exponent_antifirefly_any_code(size, spread):
    """Anti-firefly in the reference formats on arbitrary codes (exponents far apart and close, unnormalised
    mantissas, zeros): the packed kernel equals the one that clamps decoded floats, bit for bit."""
    W, H = size
    rng = np.random.default_rng(W * 100 + spread)
    _, p = Scene(W, H, seed=3).generate(0)
    with Context(0) as ctx:
        a, b = Stream(ctx, W, H, N.STORAGE_REF), Stream(ctx, W, H, N.STORAGE_REF)
        for name in ("DIFF_TEMPORARY", "SPEC_ACCUM_COLOR", "INDIR_ACCUM"):
            code = rng.integers(0, 2 ** 27, (H, W), dtype=np.uint64) | (rng.integers(0, spread, (H, W), dtype=np.uint64) << 27)
            code[rng.random((H, W)) < 0.1] = 0
            for s in (a, b):
                s.upload(name, 0, code.astype(np.uint32))
        q = p.copy()
        q.flags |= N.FLAG_STAGE_DEFAULT
        a.stage(N.STAGE_ANTI_FIREFLY, 0, 0, p)
        b.stage(N.STAGE_ANTI_FIREFLY, 0, 0, q)
        for name in ("DIFF_ACCUM_COLOR", "SPEC_PING_COLOR", "INDIR_PING"):
            assert np.array_equal(a.download(name, 0), b.download(name, 0)), name
        a.close()
        b.close()
