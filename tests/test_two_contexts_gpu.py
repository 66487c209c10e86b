"""Two contexts of different geometry on one GPU, each driven by a thread of its
own: the projectors' shared-memory sizes differ, and neither context's launches
may depend on what the other set last.  Each image equals the one the context
gives alone."""
import threading

import numpy as np
import pytest

from geoms import ALL, product_geom
from golden import inputs as I

pytestmark = pytest.mark.gpu

ITERATIONS = 40


def loaded(H, name, bp):
    ctx = H.Context(product_geom(ALL[name]))
    prompts, randoms, norm, atten, scatter = I.sinograms(*ctx.sino_shape)
    ctx.set_backprojector(bp)
    ctx.upload_inputs(prompts, randoms, norm, atten, scatter)
    ctx.sensitivity()
    return ctx


def image(ctx):
    ctx.init_image()
    ctx.osem(ITERATIONS)
    return ctx.get_image()


@pytest.mark.parametrize("bp", [0, 1])
def test_two_threads(bp):
    import hrrt_reconstruction_b200 as H
    ctxs = [loaded(H, name, bp) for name in ("small3", "small9")]
    try:
        alone = [image(c) for c in ctxs]
        got, errors = [None, None], []
        start = threading.Barrier(2)

        def work(i):
            try:
                start.wait()
                got[i] = image(ctxs[i])
            except Exception as e:  # noqa: BLE001 (reported below)
                errors.append((i, str(e)))

        ts = [threading.Thread(target=work, args=(i,)) for i in range(2)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert not errors, errors
        for g, w in zip(got, alone):
            assert np.array_equal(g.view(np.uint32), w.view(np.uint32))
    finally:
        for c in ctxs:
            c.close()
