"""Every run length the forward projector is built for (13, 17, 21 and 25 planes a
task) through both of its outputs: the estimate, bit for bit against the
single-precision oracle, and the ratio, as the image after one subset against
the FP64 one (1e-5, as the OSEM tests).  A plane variant takes the shortest
run that fits a CTA from its own on: a short scanner takes 13, 17 and 21, and a
tall one with many segments, which offers one variant only, takes 25."""
import numpy as np
import pytest

from geoms import product_geom, random_image
from golden import inputs as I

pytestmark = pytest.mark.gpu

BASE = dict(plane_sep=1.21875, binsize=1.21875)
GEOMS = {
    "short": dict(BASE, nrings=27, nelements=68, nangles=96, ring_radius=62.0, span=3, maxdel=16, subsets=16),
    "tall": dict(BASE, nrings=208, nelements=32, nangles=32, ring_radius=120.0, span=13, maxdel=207, subsets=8),
}


@pytest.mark.parametrize("name,variants", [("short", (7, 9, 11)), ("tall", (9,))])
def test_runs(name, variants):
    import hrrt_reconstruction_b200 as H
    from oracle.oracle import Oracle
    d = GEOMS[name]
    F, O = Oracle(precision="f32", **d), Oracle(precision="f64", **d)
    img = random_image((F.nx, F.nx, F.zp), F.cylwiny(), seed=5, zvalid=F.nz)
    prompts, randoms, norm, atten, scatter = I.sinograms(O.P, O.views, O.nx)
    p, a, m = O.prep(prompts, randoms, norm, atten, scatter)
    nf, want = O.sensitivity(m), O.init_image()
    s = int(O.order()[0])
    O.osem_subset(want, nf[s], p, a, s)
    with H.Context(product_geom(d)) as ctx:
        ctx.upload_inputs(prompts, randoms, norm, atten, scatter)
        ctx.sensitivity()
        ctx.set_norm_zero_mask(np.ones_like(ctx.norm_zero_mask()))
        for planes in variants:
            ctx.set_tuning(fp_planes=planes)
            for view in (1, O.views // 2 - 1):
                assert np.array_equal(F.fp_pair(img, view).view(np.uint32), ctx.fp_pair(img, view).view(np.uint32))
        ctx.upload_inputs(prompts, randoms, norm, atten, scatter)
        ctx.sensitivity()
        for planes in variants:
            ctx.set_tuning(fp_planes=planes)
            ctx.init_image()
            ctx.osem_subsets(0, 1)
            got = ctx.get_image_xyz().astype(np.float64)
            assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want), planes
