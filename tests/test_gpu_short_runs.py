"""Runs of a few steps on a handle's default choice: a batch that fills the GPU takes the step kernels for them,
in between longer runs on the resident kernel, with the same values; a chosen shape is kept whatever the length."""
import numpy as np
import pytest

import vocalsim_b200 as V
from kernel_names import launched
from vocalsim_b200 import synthetic as S

pytestmark = pytest.mark.gpu
CLUSTER = len(V.tile_shapes()) - 1


def batch(n, **kw):
    return V.Batch([V.params(cross_sectional_shape=2, **kw) for _ in range(n)],
                   [V.Geometry(*S.batch_tube(k)[:2]) for k in range(n)])


@pytest.mark.parametrize("kw", [{}, dict(source_type=2, tmm_ps_pa=800.0)], ids=["table", "two_mass"])
@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("n", [8, 9, 39, 40])
def test_mixed_lengths_equal_the_resident_kernel(n, fast, kw, cuda_ok):
    a, b = batch(n, fast_math=fast, **kw), batch(n, fast_math=fast, **kw)
    b.set_tile(CLUSTER)
    for steps in (1, 2, 37, 4, 3, 1, 5, 64, 4, 130, 2, 1):
        np.testing.assert_array_equal(a.run(steps), b.run(steps))
    for i in (0, n - 1):
        for x, y in zip(a.fields(i), b.fields(i)):
            np.testing.assert_array_equal(x, y)
    a.close()
    b.close()


@pytest.mark.parametrize("n, few", [(8, 0), (9, 1), (40, 4)])
def test_which_kernel_runs(n, few, cuda_ok):
    def resident(steps):
        names = launched(lambda: b.run(steps), ("resident_kernel", "quad", "strip_kernel"))
        if names is None:
            pytest.skip("the profiler records no kernels here")
        return any("resident_kernel" in k for k in names)

    b = batch(n, fast_math=1)
    b.run(5)
    assert [resident(k) for k in (1, 2, 4, 5, 6)] == [k > few for k in (1, 2, 4, 5, 6)]
    b.set_tile(CLUSTER)
    assert all(resident(k) for k in (1, 2, 4, 5))
    b.set_tile(-1)
    assert resident(1) == (few < 1)
    b.close()
