"""Bloom at a size whose first mip has 64K texels or more, where the wide builds of the downsample and the
2x2 upsample run, in every storage mode."""
import hashlib

import numpy as np
import pytest

import oracle
from raytracedgl1_gb300 import _native as N
from raytracedgl1_gb300.denoiser import Bloom, Context, Stream
from tests import _formats as F
from tests.test_gpu_parity import BLOOM_PLANES, MODES, TOL, _encode_pre

pytestmark = pytest.mark.gpu


# SHA-256 of the eight mips, BLOOM_RESULT and FINAL in the reference formats, whose packed codes stay what
# they were (recorded from commit d03ae75 on GB300: other builds of the downsample, another codec)
RECORDED = {(802, 451): "9b74a92cb7f4fce6b705208c57d24a712271eb1e1a70e37d4d336a22db769274",
            (1366, 767): "cf42c471d9e709b6525a77afac34816cf869535afb3a6b4453253621bc07b5d1"}


@pytest.mark.parametrize("mode_name,mode", MODES)
@pytest.mark.parametrize("size", sorted(RECORDED))
def test_bloom_parity_large_levels(mode_name, mode, size):
    """The bounds of test_bloom_parity, and in the reference formats the recorded codes."""
    W, H = size
    rng = np.random.default_rng(W * 5 + H)
    with Context(0) as ctx:
        o, s = oracle.OracleStream(W, H, mode), Stream(ctx, W, H, mode)
        assert s.image("BLOOM_MIP1", 0).width * s.image("BLOOM_MIP1", 0).height >= 65536
        for name in BLOOM_PLANES:
            img = s.image(name, 0)
            if mode == N.STORAGE_REF:   # exponents up to 2^5 of the input, 2 of the rest
                top = 20 if name == "BLOOM_INPUT" else 16
                ch = [(rng.integers(0, top, (img.height, img.width)) << m) | rng.integers(0, 1 << m, (img.height, img.width)) for m in (6, 6, 5)]
                data = (ch[0] | (ch[1] << 11) | (ch[2] << 22)).astype(np.uint32)
            else:
                rgb = rng.uniform(0.0, 1.0, (img.height, img.width, 3)) ** 4 * (24.0 if name == "BLOOM_INPUT" else 2.0)
                data = _encode_pre(rgb, img.format)
            o.plane(name, 0)[...] = data
            s.upload(name, 0, data)
        Bloom(s).Apply(0, 0.7)
        o.bloom(0, 0.7)
        codes = hashlib.sha256()
        for name in BLOOM_PLANES[1:]:
            img = s.image(name, 0)
            g, c = s.download(name, 0), o.plane(name, 0)
            codes.update(g.tobytes())
            err = F.texel_rel_err(F.decode(g, img.format), F.decode(c, img.format), atol=1e-6)
            assert err.max() <= (1e-5 if img.format == F.F_RGBA32F else TOL[img.format]), f"{name}: max rel err {err.max():.3e}"
        assert mode != N.STORAGE_REF or codes.hexdigest() == RECORDED[size]
        s.close()
