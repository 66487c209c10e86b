"""The back projector's row groups at the sizes where they can go wrong, against
the FP64 oracle: a centre row inside a group (c = 74 and 34), plane runs that
do not fill a warp's tile, steep segments whose adjacent rows are more than a
plane apart (evaluated row by row), and the device entry point on an output
that is only 4-byte aligned.  Tolerance: the projector tests' 2e-6 (float32
sums of at most 2 * 45 interpolations against doubles)."""
import ctypes

import numpy as np
import pytest

from geoms import product_geom, random_rows

pytestmark = pytest.mark.gpu

BASE = dict(plane_sep=1.21875, binsize=1.21875, subsets=16)
GEOMS = {
    "ragged9": dict(BASE, nrings=59, nelements=148, nangles=160, ring_radius=134.5, span=9, maxdel=38, subsets=10),
    "ragged3": dict(BASE, nrings=27, nelements=68, nangles=96, ring_radius=62.0, span=3, maxdel=16),
    "steep3": dict(BASE, nrings=24, nelements=64, nangles=96, ring_radius=34.0, span=3, maxdel=13),
}


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("name", sorted(GEOMS))
def test_row_groups(name):
    import torch

    import hrrt_reconstruction_b200 as H
    from oracle.oracle import Oracle
    d = GEOMS[name]
    O = Oracle(precision="f64", **d)
    with H.Context(product_geom(d)) as ctx:
        for view in (0, ctx.info.nviews // 4 + 1):
            rows = random_rows(ctx.rows_shape, seed=view)
            want = O.bp_pair(rows, view)
            got = ctx.bp_pair(rows, view)
            assert rel_l2(got, want) <= 2e-6, (view, rel_l2(got, want))
            assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
            # the device entry point, output at an odd multiple of 4 bytes
            d_in = torch.from_numpy(rows).cuda()
            n = int(np.prod(ctx.image_shape))
            d_out = torch.empty(n + 1, device="cuda")
            torch.cuda.synchronize()
            rc = H.lib.hrrt_bp_pair_noalloc(ctx._h, ctypes.c_void_p(d_in.data_ptr()), view,
                                            ctypes.c_void_p(d_out[1:].data_ptr()), None)
            torch.cuda.synchronize()
            assert rc == 0
            assert rel_l2(d_out[1:].cpu().numpy().reshape(ctx.image_shape), got) <= 1e-6
