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


@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("model", MODELS, ids=["float", "double"])
def test_checkpointed_forward_reports_the_timeout(model, fast, cuda_ok):
    b = batch(3, fast_math=fast, **model)
    seed = np.ones((3, 300), np.float32)
    b.set_wait_limit(1)
    times_out(lambda: b.forward_ckpt(300, 64))
    with pytest.raises(V.VsError) as e:              # its checkpoints are not states
        b.adjoint(seed)
    assert e.value.status == abi.VS_ERR_INVALID_ARG
    b.set_wait_limit(0)
    trace = b.forward_ckpt(300, 64)
    b.reset()
    np.testing.assert_array_equal(b.run(300), trace)
    b.close()


@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("model", MODELS, ids=["float", "double"])
def test_adjoint_reports_the_timeout(model, fast, cuda_ok):
    """Several segments: the status of the first recomputed one is kept over those that follow."""
    b = batch(3, fast_math=fast, **model)
    seed = np.random.default_rng(1).standard_normal((3, 200)).astype(np.float32)
    b.forward_ckpt(200, 64)
    want, want_z = b.adjoint(seed)
    b.set_wait_limit(1)
    times_out(lambda: b.adjoint(seed))
    b.set_wait_limit(0)
    with pytest.raises(V.VsError) as e:
        b.adjoint(seed)
    assert e.value.status == abi.VS_ERR_INVALID_ARG
    b.forward_ckpt(200, 64)
    got, got_z = b.adjoint(seed)
    np.testing.assert_array_equal(got_z, want_z)
    for x, y in zip(got, want):
        for u, v in zip(x, y):
            np.testing.assert_array_equal(u, v)
    b.close()
