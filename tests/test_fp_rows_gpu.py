"""The forward projector at the sizes where its row ring, plane runs and sample
tiles can go wrong, bit for bit against the single-precision oracle: quads
with fewer rows than the ring has slots, a column grid that no sample tile
divides (c = 74 and 34), plane runs left over from the groups of four, every
plane variant, and a NaN and infinities outside the field of view's columns
that the outside points must not pick up."""
import numpy as np
import pytest

from geoms import product_geom, random_image

pytestmark = pytest.mark.gpu

BASE = dict(plane_sep=1.21875, binsize=1.21875, subsets=16)
GEOMS = {
    "ragged9": dict(BASE, nrings=59, nelements=148, nangles=160, ring_radius=134.5, span=9, maxdel=38, subsets=10),
    "ragged3": dict(BASE, nrings=27, nelements=68, nangles=96, ring_radius=62.0, span=3, maxdel=16),
    "tiny3": dict(BASE, nrings=8, nelements=16, nangles=32, ring_radius=15.0, span=3, maxdel=4),
}


@pytest.mark.parametrize("name", sorted(GEOMS))
def test_fp_bit_identical(name):
    import hrrt_reconstruction_b200 as H
    from oracle.oracle import Oracle
    d = GEOMS[name]
    O = Oracle(precision="f32", **d)
    img = random_image((O.nx, O.nx, O.zp), O.cylwiny(), seed=3, zvalid=O.nz)
    with H.Context(product_geom(d)) as ctx:
        for planes in (0, 7, 9, 11):
            ctx.set_tuning(fp_planes=planes)
            for view in (0, 1, O.views // 2 - 1):
                want, got = O.fp_pair(img, view), ctx.fp_pair(img, view)
                assert np.array_equal(want.view(np.uint32), got.view(np.uint32)), (planes, view)
        # corner column 0 is what an outside point's address falls on
        bad = img.copy()
        bad[0, 0, :] = np.nan
        bad[0, 1, :] = np.inf
        want, got = O.fp_pair(bad, 1), ctx.fp_pair(bad, 1)
        assert np.array_equal(np.isnan(want), np.isnan(got)) and np.array_equal(np.nan_to_num(want), np.nan_to_num(got))
