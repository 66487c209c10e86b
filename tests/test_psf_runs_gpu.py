"""The PSF passes for every filter half width that has a kernel of its own (1..8)
and the first that has not, on a grid whose columns no run divides: bit for
bit the single-precision oracle's convolve3d."""
import numpy as np
import pytest

from geoms import product_geom, random_image

pytestmark = pytest.mark.gpu

RAGGED = dict(nrings=27, nelements=68, nangles=96, ring_radius=62.0, plane_sep=1.21875, binsize=1.21875, span=3,
              maxdel=16, subsets=16)


@pytest.mark.parametrize("half", range(1, 10))
def test_half_widths(half):
    import hrrt_reconstruction_b200 as H
    from oracle.oracle import Oracle
    fwhm = 0.9 * half + 0.05
    O = Oracle(precision="f32", **RAGGED)
    assert O.psf_kernel(fwhm, 0.0, 0.0, pixel_size=1.21875).size == 2 * half + 1
    O.set_psf(True, fwhm, 0.0, 0.0)
    with H.Context(product_geom(RAGGED)) as ctx:
        ctx.set_psf(True, fwhm, 0.0, 0.0)
        img = random_image(ctx.image_shape, O.cylwiny(), seed=half, zvalid=O.nz)
        want, got = O.psf(img), ctx.psf(img)
        assert np.array_equal(want.view(np.uint32), got.view(np.uint32))
