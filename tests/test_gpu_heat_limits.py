"""The heat stepper at the limits of its inputs: sources that are not finite on heat-sinked faces
(held voxels take no source)."""
import numpy as np
import pytest

import heatcases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(37, 20, 18), (33, 16, 17), (6, 5, 530), (800, 4, 3)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("steps", [3, 6])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 3e38])
def test_source_on_sinked_faces_is_ignored(shape, steps, bad, oracle_lib):
    """A heat-sinked voxel is held at its temperature whatever its source: the run with `bad` there is
    the run with no source there, bit for bit."""
    from mcmatlab_b200 import native
    case = heatcases.shaped(shape, seed=7, heatSinked=1, nt=steps)
    face = np.ones(shape, bool)
    face[1:-1, 1:-1, 1:-1] = False
    runs = []
    for q in (0.0, bad):
        hp = dict(case["hp"])
        Q = np.array(hp["dTdt_abs"], order="F", copy=True)
        Q[face] = q
        hp["dTdt_abs"] = Q
        runs.append(native.heat_forward(case["T0"], case["Omega0"], hp, *shape))
    for a, b in zip(*runs):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(runs[1][0][face], case["T0"][face])
