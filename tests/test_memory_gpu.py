"""The forward projector's rotated rows take memory that nothing else waits for: a
context without inputs does not hold them, and where the device has no room for
a buffer of their own (before or after it was taken) every call still works, with
the same results, in the partials' memory."""
import numpy as np
import pytest

from geoms import ALL, product_geom, random_image, random_rows
from golden import inputs as I

pytestmark = pytest.mark.gpu

BASE = dict(plane_sep=1.21875, binsize=1.21875)
# few subsets: 40 view pairs in one, whose rows take 0.6 GB beside 0.9 GB of partials
GEOM = dict(BASE, nrings=59, nelements=148, nangles=160, ring_radius=134.5, span=9, maxdel=38, subsets=2)
MB = 1 << 20


def free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


class Filled:
    """The device filled up to `leave` bytes."""

    def __init__(self, leave):
        import torch
        torch.cuda.empty_cache()
        self.block = torch.empty(max(0, (free() - leave) // (2 * MB)) * 2 * MB, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *a):
        import torch
        del self.block
        torch.cuda.empty_cache()


def work(ctx, inputs, img, rows):
    """One of every call that uses the rotated rows or the partials."""
    out = [ctx.fp_pair(img, 3), ctx.bp_pair(rows, 3)]
    ctx.upload_inputs(*inputs)
    ctx.sensitivity()
    ctx.init_image()
    ctx.osem(1)
    out.append(ctx.get_image())
    out.append(ctx.forward_project(img))
    out.append(ctx.bp_pair(rows, 2))
    ctx.osem(1)
    out.append(ctx.get_image())
    return out


def same(a, b):
    return all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b))


def test_rows_without_room():
    import hrrt_reconstruction_b200 as H
    H.Context(product_geom(ALL["small3"])).close()  # module load and the driver's own buffers
    before = free()
    with H.Context(product_geom(GEOM)) as ctx:
        i = ctx.info
        created = before - free()
        inputs = I.sinograms(*ctx.sino_shape)
        cyl = [(0, 0) if abs(x - 74) > 60 else (40, 108) for x in range(i.nx)]
        img = random_image(ctx.image_shape, np.array(cyl), seed=4, zvalid=i.nz)
        rows = random_rows(ctx.rows_shape, seed=6)
        want = work(ctx, inputs, img, rows)
        held = before - free()
    partials = 8 * i.nx * i.ny * i.zp * (i.sviews // 2)
    rows_bytes = held - created  # at least: inputs and staging besides
    assert created <= partials + 384 * MB, (created // MB, partials // MB)
    assert rows_bytes > 512 * MB
    with Filled(held - 400 * MB):
        with H.Context(product_geom(GEOM)) as ctx:
            assert same(work(ctx, inputs, img, rows), want)


def test_rows_given_back():
    """A buffer taken while there was room makes way for a later call's."""
    import hrrt_reconstruction_b200 as H
    with H.Context(product_geom(GEOM)) as ctx:
        inputs = I.sinograms(*ctx.sino_shape)
        want = [ctx.reconstruct(*inputs, iterations=1)[0]]
    with H.Context(product_geom(GEOM)) as ctx:
        ctx.upload_inputs(*inputs)
        with Filled(64 * MB):  # the reconstruction's staging takes 0.4 GB
            got = [ctx.reconstruct(*inputs, iterations=1)[0]]
        assert same(got, want)


def test_batch_without_room():
    import hrrt_reconstruction_b200 as H
    with H.Context(product_geom(GEOM)) as ctx:
        prompts, randoms, norm, atten, scatter = I.sinograms(*ctx.sino_shape)

        def run():
            with ctx.batch(1, norm=norm, atten=atten, storage=H.STORE_16) as b:
                b.set_frame(0, prompts, randoms, scatter, iterations=2)
                b.run()
                return [b.get_image(0)[0]]

        before = free()
        want = run()
        b = ctx.batch(1, norm=norm, atten=atten, storage=H.STORE_16)
        need = before - free()
        b.close()
        with Filled(need - 300 * MB):
            assert same(run(), want)
