"""A context's calls share scratch: what one call leaves there -- in the columns
outside the field of view above all, which no projector writes -- must not
reach the next call's result.  Every result equals a fresh context's, bit for
bit."""
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
def test_after_foreign_images(name, bp):
    import hrrt_reconstruction_b200 as H
    with H.Context(product_geom(ALL[name])) as ctx:
        rows = random_rows(ctx.rows_shape, seed=2)
        want_bp, want = ctx.bp_pair(rows, 3, mode=bp), study(ctx, bp)
    with H.Context(product_geom(ALL[name])) as ctx:
        foreign = np.full(ctx.image_shape, 1e3, np.float32)  # everywhere, outside the field of view as well
        ctx.rotate_add(foreign, 1, np.zeros_like(foreign))
        ctx.fp_pair(foreign, 1)
        assert np.array_equal(bits(ctx.bp_pair(rows, 3, mode=bp)), bits(want_bp))
        ctx.rotate_add(foreign, 1, np.zeros_like(foreign))
        assert np.array_equal(bits(study(ctx, bp)), bits(want))


@pytest.mark.parametrize("name", ["small3", "small9"])
def test_reconstruct_twice(name):
    import hrrt_reconstruction_b200 as H
    with H.Context(product_geom(ALL[name])) as ctx:
        prompts, randoms, norm, atten, scatter = I.sinograms(*ctx.sino_shape)
        first, _ = ctx.reconstruct(prompts, randoms, norm, atten, scatter, iterations=2)
        again, _ = ctx.reconstruct(prompts, randoms, norm, atten, scatter, iterations=2)
        assert np.array_equal(bits(first), bits(again))
