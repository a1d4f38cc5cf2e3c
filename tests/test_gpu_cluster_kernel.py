"""The shared-memory cluster kernel (vs_cluster.cu) on the frames it is left with: those the resident kernel's plan
refuses, here by their width (more than 1025 columns, or 961 with the two-mass source).  Values against the step
kernels and the FP32 oracle; the profiler and the shape's limits say which kernel ran."""
import numpy as np
import pytest

import oracle as O
import vocalsim_b200 as V
from kernel_names import launched

pytestmark = pytest.mark.gpu
CLUSTER = len(V.tile_shapes()) - 1
TWO_MASS = dict(source_type=2, tmm_ps_pa=800.0)


def tube(length, *areas):
    return np.full(len(areas), length / len(areas), np.float32), np.array(areas, np.float32)


LONG = [tube(80.0, 1.5, 3.0, 0.8), tube(90.0, 2.5)]
# parameters, tubes: single, a batch of uneven tubes, and a frame only the two-mass source's warp keeps out
CASES = {"one": ({}, LONG[:1]), "one_sine_mouth": (dict(source_type=0, mouth_radiation_cond=1), LONG[:1]),
         "eigen": (dict(engine=2), LONG[1:]), "two": ({}, LONG), "two_mass": (TWO_MASS, LONG),
         "two_mass_f64": (dict(TWO_MASS, tmm_f64=1), LONG[:1]), "two_mass_edge": (TWO_MASS, [tube(72.5, 2.0)])}


KERNELS = ("cluster_kernel", "resident_kernel", "quad", "strip_kernel")


def run(case, fast, shape, runs=(1, 130, 169)):
    kw, tubes = CASES[case]
    b = V.Batch([V.params(fast_math=fast, **kw) for _ in tubes], [V.Geometry(*t) for t in tubes])
    b.set_tile(shape)
    trace = np.concatenate([b.run(n) for n in runs], axis=1)
    fields = [f for i in range(len(tubes)) for f in b.fields(i)]
    names = launched(lambda: b.run(20), KERNELS)
    width = [d["frame_w"] for d in b.dims]
    b.close()
    return trace, fields, names, width


@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("case", CASES)
def test_wide_frames_equal_the_step_kernels(case, fast, cuda_ok):
    trace, fields, names, width = run(case, fast, CLUSTER)
    assert min(width) > (961 if case == "two_mass_edge" else 1025)
    if names:
        assert any("cluster_kernel" in k for k in names) and not any("resident_kernel" in k for k in names)
    want, want_fields, names, _ = run(case, fast, 21 if fast else 7)
    assert not any("cluster_kernel" in k for k in names or ())
    np.testing.assert_array_equal(trace, want)
    for x, y in zip(fields, want_fields):
        np.testing.assert_array_equal(x, y)
    if not fast:
        kw, tubes = CASES[case]
        for k, t in enumerate(tubes):
            np.testing.assert_array_equal(trace[k], O.run(O.params(**kw), O.Geometry(*t), trace.shape[1], "f32"))


def test_frames_in_reach_run_on_the_resident_kernel(cuda_ok):
    """The widest frames either source's plan takes, and the default of one wide tube."""
    for kw, length, kernel in (({}, 75.0, "resident_kernel"), (TWO_MASS, 70.0, "resident_kernel"), ({}, 80.0, "cluster_kernel")):
        s = V.Solver(V.params(**kw), V.Geometry(*tube(length, 2.0)))
        got = s.run(60)
        names = launched(lambda: s.run(20), KERNELS)
        assert not names or any(kernel in k for k in names), (s.dims["frame_w"], kernel)
        np.testing.assert_array_equal(got, O.run(O.params(**kw), O.Geometry(*tube(length, 2.0)), 60, "f32"))
        s.close()


def test_the_plan_refuses_wide_frames(cuda_ok):
    """Only the shared-memory kernel is limited to 64 tubes: a wide batch of 65 has no cluster shape."""
    for length, taken in ((80.0, False), (20.0, True)):
        b = V.Batch([V.params() for _ in range(65)], [V.Geometry(*tube(length, 2.0)) for _ in range(65)])
        if taken:
            b.set_tile(CLUSTER)
        else:
            with pytest.raises(V.VsError):
                b.set_tile(CLUSTER)
        b.close()
