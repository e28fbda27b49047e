"""The FP64 sums of an image's samples (k_accumulate) over a float's range:
the squares and conversions are put together from integers, the rest of the
range takes the double units.

One emissive quad a pixel, of radiance zero, the smallest and largest
subnormal, the smallest and largest normal and values between, infinity, one
of each sign; half of each pixel's samples pass it by.  The oracle sums the
same samples with double products, in the same order: every bit is equal.
"""
import numpy as np
import pytest

import lisa_gb300 as L
from lisa_gb300 import scenes as S

pytestmark = pytest.mark.gpu

EDGES = np.array([0x0, 0x1, 0x7fffff, 0x800000, 0x800001, 0xffffff, 0x3f800000, 0x3f7fffff, 0x3fb504f3, 0x3fb504f4,
                  0x3fffffff, 0x5f000000, 0x1f800000, 0x7f7fffff, 0x7f800000], np.uint32).view(np.float32)


@pytest.mark.parametrize("accum", [0, 1])
@pytest.mark.parametrize("spp", [1, 2, 7])
def test_sums_of_any_float(gpu, oracle, spp, accum):
    rand = np.random.default_rng(3).integers(0x00800000, 0x7f800000, 49, dtype=np.uint32).view(np.float32)
    values = np.concatenate([EDGES, rand])
    n = len(values)
    mats, v, mi = [], [], []
    for i, e in enumerate(values):
        # a quad over the left half of pixel (i % 8, i / 8) of an 8 x 8 image
        x, y = (i % 8 - 4) / 4.0, (i // 8 - 4) / 4.0
        w, h = 0.13, 0.25
        a, b, c, d = (x, y, 0), (x + w, y, 0), (x + w, y + h, 0), (x, y + h, 0)
        v += [a, b, c, a, c, d]
        mi += [i, i]
        mats.append([1, 1, 0, 1, 1, 1, 1, e, np.float32(1.0), -e])
    v = np.array(v, np.float32)
    nrm = np.tile(np.array([0, 0, 1], np.float32), (len(v), 1))
    mats = np.array(mats, np.float32)
    cam = dict(eye=(0.0, 0.0, 10.0), look_at=(0.0, 0.0, 0.0), fov=11.4)
    p = L.params_from_arrays(v, nrm, np.array(mi), mats, 8, 8, cam["eye"], cam["look_at"], cam["fov"], spp, 2)
    r = L.Renderer(p, accum_fp64=accum)
    r.render()
    _, var, mean = r.image(variance=True, fp64=True)
    with np.errstate(all="ignore"):
        s, sq, _ = oracle.Scene(v, nrm, np.array(mi, np.int32), mats, width=8, height=8, spp=spp, bounces=2,
                                **cam).render(use_bvh=True)
        s, sq = s.reshape(8, 8, 3), sq.reshape(8, 8, 3)
        seen = (s != 0).any(axis=2).sum()
        assert seen > 0.3 * n
        if accum:
            assert np.array_equal(mean, s / spp, equal_nan=True)
            ref = (sq / spp - mean * mean) * spp / (spp - 1.0) if spp > 1 else np.zeros_like(sq)
            assert np.array_equal(var, np.where(ref > 0, ref, 0.0))
        else:  # the mean is the float sum's
            ref = (sq / spp - mean * mean) * spp / (spp - 1.0) if spp > 1 else np.zeros_like(sq)
            assert np.array_equal(var, np.where(ref > 0, ref, 0.0))
