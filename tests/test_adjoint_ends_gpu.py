"""The exact adjoint's end planes, as a gather by table and (where a plane would
take more than four of them) entry by entry, against the FP64 oracle's
transpose; tolerance of the adjoint tests, 1e-6."""
import numpy as np
import pytest

from geoms import product_geom, random_rows

pytestmark = pytest.mark.gpu

BASE = dict(plane_sep=1.21875, binsize=1.21875, subsets=16)
# name -> (geometry, whether its end planes gather by table)
GEOMS = {
    "ragged9": (dict(BASE, nrings=59, nelements=148, nangles=160, ring_radius=134.5, span=9, maxdel=38, subsets=10), True),
    "ragged3": (dict(BASE, nrings=27, nelements=68, nangles=96, ring_radius=62.0, span=3, maxdel=16), False),
    "ragged7": (dict(BASE, nrings=28, nelements=68, nangles=96, ring_radius=62.0, span=7, maxdel=17), True),
    "steep9": (dict(BASE, nrings=32, nelements=64, nangles=96, ring_radius=34.0, span=9, maxdel=22), False),
}


def gathers(d):
    """At least 6 end planes an end, of which at most 4 consecutive ones reach
    an output plane, and no end's outputs span 24 planes (rows 1 .. c-1 and
    their mirrors)."""
    import hrrt_reconstruction_b200 as H
    zi = H.geometry_table(product_geom(d), "flookup_zzi")
    zs, N = d["span"] - 1, d["nelements"]
    if zs < 6:
        return False
    zi = zi.reshape(N, -1, 2, zs)
    rows = zi[[y for y in range(1, N) if y != N // 2]].reshape(-1, zs)
    for r in rows:
        if r.max() + 1 - r.min() >= 24:
            return False
        for z in range(r.min(), r.max() + 2):
            i = np.flatnonzero((r == z) | (r + 1 == z))
            if i.size and i[-1] - i[0] + 1 > 4:
                return False
    return True


@pytest.mark.parametrize("name", sorted(GEOMS))
def test_adjoint_end_planes(name):
    import hrrt_reconstruction_b200 as H
    from oracle.oracle import Oracle
    d, table = GEOMS[name]
    assert gathers(d) == table
    O = Oracle(precision="f64", **d)
    with H.Context(product_geom(d)) as ctx:
        for view in (0, 3, ctx.info.nviews // 2 - 1):
            rows = random_rows(ctx.rows_shape, seed=view + 1)
            want, got = O.fp_adjoint(rows, view), ctx.bp_pair(rows, view, mode=H.BP_ADJOINT)
            e = np.linalg.norm(got.astype(np.float64) - want) / np.linalg.norm(want)
            assert e <= 1e-6, (view, e)
