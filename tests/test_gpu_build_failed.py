"""A BVH build whose sort failed (a bounded wait ran out) ends with a status:
the kernels behind the sort, which would take indices from its output, write
nothing, and the GPU is as before."""
import ctypes as C

import numpy as np
import pytest

import lisa_gb300 as L
from lisa_gb300 import scenes

N = L._native


def test_arguments():
    lib = N.lib()
    w = C.c_uint32(7)
    assert lib.lisa_selftest_bvh_failed(10, None) == N.LISA_ERR_INVALID
    assert lib.lisa_selftest_bvh_failed(0, C.byref(w)) == N.LISA_ERR_INVALID
    assert lib.lisa_selftest_bvh_failed(65537, C.byref(w)) == N.LISA_ERR_INVALID
    assert w.value == 7


@pytest.mark.gpu
@pytest.mark.parametrize("t", [1, 2, 3, 300, 5000, 65536])
def test_later_kernels_return_at_once(gpu, t):
    w = C.c_uint32(123)
    assert N.lib().lisa_selftest_bvh_failed(t, C.byref(w)) == N.LISA_ERR_DEVICE
    assert b"wait ran out" in N.lib().lisa_last_error()
    assert w.value == 0
    sc = scenes.cornell_box(width=16, height=16, num_samples=1, num_bounces=2)
    r = L.Renderer(L.params_from_scene(sc))
    st = r.render()
    assert st.device_status == 0 and st.rays_primary == 16 * 16 and np.isfinite(r.image()).all()
