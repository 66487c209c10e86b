"""A batch's scratch starts clean whatever its memory held before: the rotate-back
reads the partials' columns beside the field of view, which no kernel writes."""
import ctypes

import numpy as np
import pytest

from geoms import product_geom
from golden import inputs as I

pytestmark = pytest.mark.gpu

TINY = dict(plane_sep=1.21875, binsize=1.21875, nrings=8, nelements=16, nangles=32, ring_radius=15.0, span=3,
            maxdel=4, subsets=4)


def dirty_device_memory():
    """Blocks of the sizes that a small context allocates, filled and freed."""
    rt = ctypes.CDLL("libcudart.so.12")
    rt.cudaMalloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t]
    rt.cudaMemset.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t]
    rt.cudaFree.argtypes = [ctypes.c_void_p]
    blocks = []
    for k in range(256):
        p = ctypes.c_void_p()
        assert rt.cudaMalloc(ctypes.byref(p), 4096 << (k % 8)) == 0
        assert rt.cudaMemset(p, 0x4b, 4096 << (k % 8)) == 0  # 1.3e7 as floats
        blocks.append(p)
    assert rt.cudaDeviceSynchronize() == 0
    for p in blocks:
        assert rt.cudaFree(p) == 0


def test_batch_on_dirty_memory():
    import hrrt_reconstruction_b200 as H
    with H.Context(product_geom(TINY)) as ctx:
        prompts, randoms, norm, atten, scatter = I.sinograms(*ctx.sino_shape)
        ctx.upload_inputs(prompts, randoms, norm, atten, scatter)
        ctx.sensitivity()
        ctx.init_image()
        ctx.osem(2)
        want = ctx.get_image()
    with H.Context(product_geom(TINY)) as ctx:
        dirty_device_memory()
        with ctx.batch(2, norm=norm, atten=atten) as b:
            for f in range(2):
                b.set_frame(f, prompts, randoms, scatter, iterations=2)
            b.run()
            for f in range(2):
                assert np.array_equal(b.get_image(f)[0].view(np.uint32), want.view(np.uint32)), f
