"""Coded-row passes of the heat stepper against the FP64 oracle where they can go wrong: lines
shorter than a chunk, at and just past the chunk (16 rows) and block-class edges, padding lines and
columns, heat-sinked faces, no damage, and grids whose media vary voxel by voxel (more row
coefficients than the code tables hold, which step with the TMA-staged passes). The tolerances are
those of the streamed stepper's tests: the FP32 state stays within 1e-5 of FP64 over tens of steps."""
import numpy as np
import pytest

import heatcases
from test_gpu_heat_stream import _check

pytestmark = pytest.mark.gpu

SHAPES = [(2, 3, 2), (3, 2, 5), (4, 33, 2), (5, 16, 17), (16, 17, 16), (17, 15, 33), (33, 32, 31), (128, 5, 6), (129, 4, 7),
          (320, 4, 3), (321, 3, 4), (512, 3, 2), (6, 128, 5), (5, 129, 6), (4, 209, 3), (3, 321, 4), (2, 512, 3),
          (7, 5, 128), (6, 7, 129), (5, 3, 208), (4, 3, 320), (3, 4, 321), (3, 2, 512)]


@pytest.mark.parametrize("hs", [0, 1])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_row_passes_at_edges(shape, hs, oracle_lib):
    _check(heatcases.shaped(shape, seed=sum(shape), heatSinked=hs, lightsOn=shape[0] % 2 == 1, nt=6,
                            with_damage=shape[1] % 2 == 1, dt_factor=1.5), oracle_lib)


@pytest.mark.parametrize("nM,hs", [(3, 0), (24, 0), (24, 1)])
def test_media_varying_by_voxel(nM, hs, oracle_lib):
    """nM = 3 fits the code tables, nM = 24 does not."""
    from mcmatlab_b200 import mexargs, prep
    case = heatcases.shaped((40, 33, 21), seed=nM, heatSinked=hs, nt=8)
    rng = np.random.default_rng(nM)
    M1 = rng.integers(1, nM + 1, case["n"]).astype(np.uint8)
    TC, VHC = rng.uniform(0.002, 0.006, nM), rng.uniform(3.0, 4.2, nM)
    c, Q = prep.calc_dTdt_arrays(VHC, TC, 0.02, 0.02, 0.02, 40.0 * rng.random(case["n"]), 1.0, M1)
    A, E = np.where(np.arange(nM) % 2, 7.6e66, 0.0), np.where(np.arange(nM) % 2, 4.48e5, 0.0)
    hp = case["hp"]
    case["hp"] = mexargs.heat_mex_params(M1, A, E, c, Q, True, hs, hp["tempSensorCornerIdxs"].ravel(),
                                         hp["tempSensorInterpWeights"], True, 8, 0.02)
    _check(case, oracle_lib)
