"""A wait of the resident kernel that runs out: the poll limit of one makes the tiles' wait for the two-mass flow
give up in its first steps, while the clusters' exchanges are under way.  The call reports VS_ERR_TIMEOUT, the
CTAs leave after what was sent to them has landed, and the next call with the default limit is right again."""
import numpy as np
import pytest

import vocalsim_b200 as V
from vocalsim_b200 import abi
from vocalsim_b200 import synthetic as S

pytestmark = pytest.mark.gpu
CLUSTER = len(V.tile_shapes()) - 1
MODELS = [dict(tmm_f64=0), dict(tmm_f64=1)]


def batch(n, **kw):
    kw = dict(cross_sectional_shape=2, source_type=2, tmm_ps_pa=800.0, **kw)
    b = V.Batch([V.params(**kw) for _ in range(n)], [V.Geometry(*S.batch_tube(k)[:2]) for k in range(n)])
    b.set_tile(CLUSTER)
    return b


def times_out(call):
    with pytest.raises(V.VsError) as e:
        call()
    assert e.value.status == abi.VS_ERR_TIMEOUT


@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("model", MODELS, ids=["float", "double"])
@pytest.mark.parametrize("n", [1, 20])
def test_run_reports_the_timeout_and_the_next_run_is_clean(n, model, fast, cuda_ok):
    b = batch(n, fast_math=fast, **model)
    want = b.run(200)
    for _ in range(3):
        b.reset()
        b.set_wait_limit(1)
        times_out(lambda: b.run(300))
        b.set_wait_limit(0)
        b.reset()
        np.testing.assert_array_equal(b.run(200), want)
    b.close()
