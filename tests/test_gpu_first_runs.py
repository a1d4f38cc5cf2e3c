"""The first run of a new handle, over and over in device memory that other handles and fills left dirty: what
creation uploads (tube order, source tables, maps, descriptors) is in place when the first kernel reads it."""
import numpy as np
import pytest

import vocalsim_b200 as V
from vocalsim_b200 import synthetic as S

pytestmark = pytest.mark.gpu
STEP_SHAPE = {0: 7, 1: 21}           # single-step kernels of the two arithmetics


def batch(tubes, kw):
    return V.Batch([V.params(**kw) for _ in tubes], [V.Geometry(*t) for t in tubes])


def dirty_memory():
    """Device memory of several allocation sizes filled with -1 and given back to the driver."""
    import torch
    junk = [torch.full((1 << k,), -1, dtype=torch.int32, device="cuda") for k in (6, 10, 16, 20, 24)]
    torch.cuda.synchronize()
    del junk
    torch.cuda.empty_cache()


KINDS = {"gauss": {}, "sine": dict(source_type=0, mouth_radiation_cond=1), "fine": dict(srate_mul=30),
         "two_mass": dict(source_type=2, tmm_ps_pa=800.0), "two_mass_f64": dict(source_type=2, tmm_ps_pa=800.0, tmm_f64=1)}


@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("kind", KINDS)
def test_first_run_of_every_new_batch_equals_the_step_kernels(kind, fast, cuda_ok):
    kw = dict(KINDS[kind], cross_sectional_shape=2, fast_math=fast)
    sizes = (1, 2, 7, 33, 96) if kind in ("gauss", "sine") else (1, 3)
    steps, want = 40, {}
    for n in sizes:
        tubes = [S.batch_tube((5 * k + n) % 256)[:2] for k in range(n)]
        b = batch(tubes, kw)
        b.set_tile(STEP_SHAPE[fast])
        want[n] = (tubes, b.run(steps))
        b.close()
    for turn in range(6):
        for n in sizes if turn % 2 else reversed(sizes):
            tubes, trace = want[n]
            dirty_memory()
            b = batch(tubes, kw)
            got = b.run(steps)
            b.close()
            np.testing.assert_array_equal(got, trace)


@pytest.mark.parametrize("fast", [0, 1])
def test_first_gradient_of_every_new_batch_is_the_same(fast, cuda_ok):
    tubes = [S.batch_tube(k)[:2] for k in range(3)]
    seed = np.random.default_rng(2).standard_normal((3, 70)).astype(np.float32)
    want = None
    for _ in range(6):
        dirty_memory()
        b = batch(tubes, dict(cross_sectional_shape=2, fast_math=fast))
        trace = b.forward_ckpt(70, 32)
        maps, gz = b.adjoint(seed)
        again = b.run(5)             # continues on the descriptors that the adjoint restored
        b.close()
        got = [trace, again, gz] + [g for m in maps for g in m]
        want = want or got
        for x, y in zip(got, want):
            np.testing.assert_array_equal(x, y)
