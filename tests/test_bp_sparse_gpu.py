"""The back projector on rows that are zero but for a few large bins, voxel by
voxel against the FP64 oracle.  Every term of a voxel's sum is a plane times a
weight of at least zero, so nothing cancels and each voxel keeps its relative
accuracy however large its neighbours are: at most 4 * groups + 4 roundings of
2^-24 each (two fused adds per segment side, the weight 1 - f, the centre
segment and the sum of the two partials)."""
import ctypes

import numpy as np
import pytest

from geoms import ALL, product_geom

pytestmark = pytest.mark.gpu

BASE = dict(plane_sep=1.21875, binsize=1.21875, subsets=16)
GEOMS = {
    "small3": ALL["small3"],
    "ragged9": dict(BASE, nrings=59, nelements=148, nangles=160, ring_radius=134.5, span=9, maxdel=38, subsets=10),
    "ragged3": dict(BASE, nrings=27, nelements=68, nangles=96, ring_radius=62.0, span=3, maxdel=16),
    "steep3": dict(BASE, nrings=24, nelements=64, nangles=96, ring_radius=34.0, span=3, maxdel=13),
}


def device_bp(ctx, rows, view):
    """hrrt_bp_pair_noalloc on device buffers."""
    import torch

    import hrrt_reconstruction_b200 as H
    d_in = torch.from_numpy(rows).cuda()
    d_out = torch.empty(int(np.prod(ctx.image_shape)), device="cuda")
    torch.cuda.synchronize()
    assert H.lib.hrrt_bp_pair_noalloc(ctx._h, ctypes.c_void_p(d_in.data_ptr()), view,
                                      ctypes.c_void_p(d_out.data_ptr()), None) == 0
    torch.cuda.synchronize()
    return d_out.cpu().numpy().reshape(ctx.image_shape)


@pytest.mark.parametrize("name", sorted(GEOMS))
def test_sparse_rows(name):
    import hrrt_reconstruction_b200 as H
    from oracle.oracle import Oracle
    d = GEOMS[name]
    O = Oracle(precision="f64", **d)
    groups = (d["maxdel"] - (d["span"] - 1) // 2) // d["span"]
    bar = (4 * groups + 4) * 2.0 ** -24
    with H.Context(product_geom(d)) as ctx:
        for view, hot in ((0, 100.0), (ctx.info.nviews // 4 + 1, 1e4)):
            rng = np.random.default_rng(view + 1)
            rows = np.where(rng.random(ctx.rows_shape) < 0.01, hot * rng.random(ctx.rows_shape), 0.0)
            rows = rows.astype(np.float32)
            want = O.bp_pair(rows, view)
            for got in (ctx.bp_pair(rows, view), device_bp(ctx, rows, view)):
                # the oracle's sums are incremental: its own cancellation of the large bins, in doubles
                assert np.all(np.abs(got - want) <= bar * np.abs(want) + hot * 1e-13), \
                    (view, float(np.max(np.abs(got - want) / np.maximum(np.abs(want), hot * 1e-9))))


@pytest.mark.parametrize("name", sorted(GEOMS))
def test_infinite_bin(name):
    """An infinite bin gives infinity, not NaN, wherever it has a weight."""
    import hrrt_reconstruction_b200 as H
    with H.Context(product_geom(GEOMS[name])) as ctx:
        shape = ctx.rows_shape
        rng = np.random.default_rng(7)
        for view in (0, 5):
            at = tuple(int(rng.integers(n // 3, 2 * n // 3)) for n in shape)
            rows = np.zeros(shape, np.float32)
            rows[at] = 1.0
            weight = ctx.bp_pair(rows, view)
            assert (weight > 0).any()
            rows[at] = np.inf
            for got in (ctx.bp_pair(rows, view), device_bp(ctx, rows, view)):
                assert np.isposinf(got[weight > 0]).all(), int((~np.isposinf(got[weight > 0])).sum())
