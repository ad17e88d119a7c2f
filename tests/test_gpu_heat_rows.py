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


LONG = [(513, 5, 4), (700, 3, 5), (4, 513, 5), (5, 640, 4), (3, 1000, 4), (5, 4, 513), (6, 5, 641), (4, 3, 1024)]


@pytest.mark.parametrize("shape", LONG, ids=lambda s: "x".join(map(str, s)))
def test_long_axes(shape, oracle_lib):
    """Axes over 512 voxels (32 rows per lane), heat-sinked faces on the odd ones."""
    _check(heatcases.shaped(shape, seed=sum(shape), heatSinked=sum(shape) % 2, nt=5, dt_factor=15.0), oracle_lib)


def _many_media(case, nM, dt, steps, hs=0):
    """`case` with media varying voxel by voxel."""
    from mcmatlab_b200 import mexargs, prep
    rng = np.random.default_rng(nM)
    M1 = rng.integers(1, nM + 1, case["n"]).astype(np.uint8)
    c, Q = prep.calc_dTdt_arrays(rng.uniform(3.0, 4.2, nM), rng.uniform(0.002, 0.006, nM), 0.02, 0.02, 0.02,
                                 40.0 * rng.random(case["n"]), 1.0, M1)
    hp = case["hp"]
    hp = mexargs.heat_mex_params(M1, np.full(nM, 7.6e66), np.full(nM, 4.48e5), c, Q, True, hs, hp["tempSensorCornerIdxs"].ravel(),
                                 hp["tempSensorInterpWeights"], True, steps, dt)
    return dict(case, hp=hp)


def test_long_axis_of_many_media(oracle_lib):
    """Too many row coefficients for the code tables on a grid the staged passes do not take either."""
    _check(_many_media(heatcases.shaped((9, 7, 530), seed=5, nt=6), 24, 0.02, 6), oracle_lib)


def test_long_state_outgrows_its_codes(oracle_lib):
    """A resident state on a long axis whose codes fit at a small time step and not at a large one goes
    on as a factored state, with its temperatures and damage, and back to small steps."""
    from mcmatlab_b200 import native
    from oracle import orc
    base = heatcases.shaped((8, 9, 600), seed=6, nt=4)
    calls = [_many_media(base, 3, dt, 4)["hp"] for dt in (1e-6, 2.0, 1e-6)]
    T, O = base["T0"], base["Omega0"]
    st = native.HeatState(T, O, calls[0], *base["n"])
    try:
        for hp in calls:
            st.step(hp)
            T, O, _, _ = orc.oracle_heat(T.astype(np.float32), O.astype(np.float32), hp, *base["n"])
        Tg, Og = st.read()
    finally:
        st.close()
    assert np.max(np.abs(Tg - T) / np.abs(T)) <= 3e-5  # 1e-5 per call
    assert np.max(np.abs(Og - O)) <= 1e-4 * np.max(O)
