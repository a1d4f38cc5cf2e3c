"""Gradients of one handle whose launch shape changes between them: the states are recomputed by the kernel of the
shape in use (one or two steps a launch, or a segment on the resident kernel), and the gradients are the same."""
import numpy as np
import pytest

import vocalsim_b200 as V
from kernel_names import launched
from vocalsim_b200 import synthetic as S

pytestmark = pytest.mark.gpu
SHAPES = range(len(V.tile_shapes()))
CLUSTER = SHAPES[-1]
TWO_STEP = next(k for k in SHAPES if V.tile_shape_steps(k) == 2)


def test_recomputation_follows_the_shape(cuda_ok):
    n, steps = 3, 192
    b = V.Batch([V.params(cross_sectional_shape=2, fast_math=1) for _ in range(n)],
                [V.Geometry(*S.batch_tube(k)[:2]) for k in range(n)])
    seed = np.random.default_rng(4).standard_normal((n, steps)).astype(np.float32)
    want, out = None, []
    for shape, every, part in ((CLUSTER, 64, "resident_kernel"), (TWO_STEP, 64, "quad2"), (CLUSTER, 64, "resident_kernel"),
                               (TWO_STEP, 48, "quad2"), (TWO_STEP, 63, None), (CLUSTER, 50, "resident_kernel")):
        b.set_tile(shape)
        b.forward_ckpt(steps, every)
        names = launched(lambda: out.append(b.adjoint(seed)), ("resident_kernel", "quad", "::strip_kernel"))
        if part and names:
            history = {k for k in names if "adjoint" not in k and any(s in k for s in ("resident_", "quad", "strip_"))}
            assert all(part in k for k in history), names
        maps, gz = out[-1]
        got = [gz] + [g for m in maps for g in m]
        want = want or got
        for x, y in zip(got, want):
            np.testing.assert_array_equal(x, y)
    b.close()
