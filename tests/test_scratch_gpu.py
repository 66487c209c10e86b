"""hrrt_rotate_add takes a whole image, outside the field of view as well, through
scratch that the back projection's partials lie in.  What it leaves there must
not reach a later result: each equals a fresh context's, bit for bit."""
import numpy as np
import pytest

from geoms import ALL, product_geom, random_rows
from golden import inputs as I

pytestmark = pytest.mark.gpu


def bits(a):
    return np.asarray(a, np.float32).view(np.uint32)


def study(ctx, bp):
    prompts, randoms, norm, atten, scatter = I.sinograms(*ctx.sino_shape)
    ctx.set_backprojector(bp)
    ctx.upload_inputs(prompts, randoms, norm, atten, scatter)
    ctx.sensitivity()
    ctx.init_image()
    ctx.osem(1)
    return ctx.get_image()


@pytest.mark.parametrize("bp", [0, 1])
@pytest.mark.parametrize("name", ["small3", "small9"])
def test_after_rotate_add(name, bp):
    import hrrt_reconstruction_b200 as H
    with H.Context(product_geom(ALL[name])) as ctx:
        rows = random_rows(ctx.rows_shape, seed=2)
        want_bp, want = ctx.bp_pair(rows, 3, mode=bp), study(ctx, bp)
    with H.Context(product_geom(ALL[name])) as ctx:
        foreign = np.full(ctx.image_shape, 1e3, np.float32)
        ctx.rotate_add(foreign, 1, np.zeros_like(foreign))
        assert np.array_equal(bits(ctx.bp_pair(rows, 3, mode=bp)), bits(want_bp))
        ctx.rotate_add(foreign, 1, np.zeros_like(foreign))
        assert np.array_equal(bits(study(ctx, bp)), bits(want))
