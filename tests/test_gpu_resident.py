"""The resident kernel (vs_resident.cu, the cluster shape): a whole run of
every tube on its own cluster, against the step kernels, value for value."""
import numpy as np
import pytest

import vocalsim_b200 as V
from vocalsim_b200 import synthetic as S

pytestmark = pytest.mark.gpu
CLUSTER = len(V.tile_shapes()) - 1


def tube(length, area):
    """One section; the frame's width follows the length, its height the area."""
    return np.array([length], np.float32), np.array([area], np.float32)


# (steps of the runs, tubes, parameters): one row per CTA and several, tiles of 64 columns with one
# column over and one short, more tubes than clusters resident at once, one step, odd run lengths
CASES = {
    "narrow": ((1, 2, 97), [tube(1.2, 0.2)], dict(cross_sectional_shape=1)),
    "flat": ((130, 1), [tube(17.5, 0.05)], dict(cross_sectional_shape=1)),
    "tile_edges": ((60, 61), [tube(x, 3.0) for x in (7.52, 7.59, 7.67, 7.75)], dict(cross_sectional_shape=1)),
    "sine_mouth": ((201,), [S.vowel_tube(k) for k in range(3)],
                   dict(cross_sectional_shape=2, source_type=0, mouth_radiation_cond=1)),
    "eigen_2d": ((150,), [S.vowel_tube(5)], dict(cross_sectional_shape=2, engine=2, fdtd_solver_type=0)),
    "voiced": ((1, 120, 33), [S.vowel_tube(k) for k in range(2)],
               dict(cross_sectional_shape=2, source_type=2, tmm_ps_pa=800.0)),
    "voiced_f64": ((2, 201), [S.vowel_tube(3)],
                   dict(cross_sectional_shape=2, source_type=2, tmm_ps_pa=800.0, tmm_f64=1)),
    "many": ((33, 40), [S.batch_tube(k)[:2] for k in range(90)], dict(cross_sectional_shape=2)),
    "fine": ((64,), [S.batch_tube(k)[:2] for k in range(2)], dict(cross_sectional_shape=2, srate_mul=30)),
}


def run(case, fast, shape):
    runs, tubes, kw = CASES[case]
    kw = dict(kw, fast_math=fast)
    b = V.Batch([V.params(**kw) for _ in tubes], [V.Geometry(*t) for t in tubes])
    if shape is not None:
        b.set_tile(shape)
    out = [b.run(n) for n in runs]
    return out, [b.fields(i) for i in (0, len(tubes) - 1)]


@pytest.mark.parametrize("fast", [1, 0])
@pytest.mark.parametrize("case", CASES)
def test_resident_equals_the_step_kernels(case, fast, cuda_ok):
    a, fa = run(case, fast, CLUSTER)
    r, fr = run(case, fast, 21 if fast else 7)
    for x, y in zip(a, r):
        np.testing.assert_array_equal(x, y)
    for x, y in zip(fa, fr):
        for u, v in zip(x, y):
            np.testing.assert_array_equal(u, v)


@pytest.mark.parametrize("kw", [{}, dict(source_type=2, tmm_ps_pa=800.0, tmm_f64=1)])
@pytest.mark.parametrize("fast", [1, 0])
def test_resident_history_gives_the_step_kernels_gradients(fast, kw, cuda_ok):
    """The adjoint's recomputation on the resident kernel: the same states, so the same gradients."""
    tubes = [S.batch_tube(k)[:2] for k in range(3)]
    rng = np.random.default_rng(5)
    seed = rng.standard_normal((3, 300)).astype(np.float32)
    res = []
    for shape in (CLUSTER, 21 if fast else 7):
        b = V.Batch([V.params(cross_sectional_shape=2, fast_math=fast, **kw) for _ in tubes],
                    [V.Geometry(*t) for t in tubes])
        b.set_tile(shape)
        tr = b.forward_ckpt(300, 128)
        maps, gz = b.adjoint(seed)
        res.append((tr, np.concatenate([g.ravel() for m in maps for g in m]), gz))
    for x, y in zip(*res):
        np.testing.assert_array_equal(x, y)
