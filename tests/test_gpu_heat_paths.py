"""Each of the heat stepper's three paths against the FP64 oracle, on calls that take it:

* the TMA-staged passes: calls of fewer than four steps, and grids whose row coefficients do not fit the
  code tables (counted here as the stepper counts them), with and without the 16-step graph,
* the coded-row passes: up to 796 voxels along x and 1024 along y and z,
* the factored stepper: longer x axes, and long axes whose row coefficients do not fit.

Bounds of the stepper's other tests: 1e-5 of T, 1e-4 of the damage gained."""
import numpy as np
import pytest

import heatcases
from test_gpu_heat_limits import row_codes
from test_gpu_heat_stream import SHAPES, _check

pytestmark = pytest.mark.gpu


def mixed(shape, steps, nM=24, hs=0, lights=True, damage=True, seed=3):
    """A case with sensors whose medium changes from voxel to voxel; its row codes do not fit."""
    from mcmatlab_b200 import mexargs, prep
    case = heatcases.shaped(shape, seed=seed, heatSinked=hs, nt=steps, with_damage=damage)
    rng = np.random.default_rng(seed)
    M1 = rng.integers(1, nM + 1, shape).astype(np.uint8)
    c, Q = prep.calc_dTdt_arrays(rng.uniform(3.0, 4.2, nM), rng.uniform(0.002, 0.006, nM), 0.02, 0.02, 0.02,
                                 40.0 * rng.random(shape), 1.0, M1)
    A, E = np.where(np.arange(nM) % 2, 7.6e66, 0.0), np.where(np.arange(nM) % 2, 4.48e5, 0.0)
    hp = case["hp"]
    hp = mexargs.heat_mex_params(M1, A, E, c, Q, True, hs, hp["tempSensorCornerIdxs"].ravel(), hp["tempSensorInterpWeights"],
                                 lights, steps, 0.02)
    assert max(row_codes(hp)) > 255
    return dict(case, hp=hp)


def kernels(call):
    """Names of the kernels that `call` launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return " ".join({e.name for e in p.events()})


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_staged_line_classes_in_short_calls(shape, oracle_lib):
    _check(heatcases.shaped(shape, seed=sum(shape), nt=3), oracle_lib)


@pytest.mark.parametrize("hs,lights", [(1, True), (1, False), (0, False)])
def test_staged_sink_and_light_in_short_calls(hs, lights, oracle_lib):
    _check(heatcases.shaped((44, 36, 28), seed=9, heatSinked=hs, lightsOn=lights, nt=3), oracle_lib)


@pytest.mark.parametrize("dtf", [1.5, 15.0, 400.0])
def test_staged_large_time_steps_in_short_calls(dtf, oracle_lib):
    _check(heatcases.shaped((70, 40, 30), seed=13, nt=3, dt_factor=dtf), oracle_lib)


@pytest.mark.parametrize("shape,steps,hs,lights", [
    ((100, 20, 18), 17, 0, True), ((200, 12, 10), 8, 1, True), ((300, 9, 8), 8, 0, False), ((400, 8, 9), 6, 1, False),
    ((20, 60, 18), 33, 0, True), ((16, 190, 8), 8, 1, True), ((17, 350, 8), 6, 0, True),
    ((14, 20, 100), 16, 1, False), ((12, 10, 250), 8, 0, True), ((10, 12, 400), 6, 1, True)],
    ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else None)
def test_staged_passes_of_uncoded_media(shape, steps, hs, lights, oracle_lib):
    """16, 17 and 33 steps run one or two graphs of 16 and what is left."""
    _check(mixed(shape, steps, hs=hs, lights=lights, damage=steps % 2 == 0), oracle_lib)


@pytest.mark.parametrize("nx", [796, 797])
@pytest.mark.parametrize("hs", [0, 1])
def test_longest_coded_x_axis_and_the_next(nx, hs, oracle_lib):
    """The X pass holds 32 lines of 796 voxels in shared memory; one more takes the factored stepper."""
    _check(heatcases.shaped((nx, 7, 6), seed=nx, heatSinked=hs, nt=5), oracle_lib)


@pytest.mark.parametrize("shape", [(530, 16, 12), (12, 530, 9), (9, 7, 530), (800, 6, 5), (6, 9, 1030)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("steps,hs", [(6, 0), (18, 1)])
def test_factored_stepper_of_uncoded_media(shape, steps, hs, oracle_lib):
    _check(mixed(shape, steps, hs=hs), oracle_lib)


PATHS = [
    ("staged, few steps", lambda: heatcases.shaped((60, 40, 30), nt=3), "sx_kernel", "rows_x_kernel"),
    ("staged, uncoded", lambda: mixed((60, 40, 30), 5), "sx_kernel", "rows_x_kernel"),
    ("coded", lambda: heatcases.shaped((60, 40, 30), nt=4), "rows_x_kernel", "sx_kernel"),
    ("coded, long", lambda: heatcases.shaped((796, 6, 5), nt=2), "rows_x_kernel", "pass_x_kernel"),
    ("factored, long x", lambda: heatcases.shaped((797, 6, 5), nt=4), "pass_x_kernel", "rows_x_kernel"),
    ("factored, uncoded", lambda: mixed((530, 16, 12), 4), "pass_x_kernel", "rows_x_kernel"),
]


@pytest.mark.parametrize("make,runs,not_runs", [p[1:] for p in PATHS], ids=[p[0] for p in PATHS])
def test_which_path_runs(make, runs, not_runs):
    from mcmatlab_b200 import native
    case = make()
    names = kernels(lambda: native.heat_forward(case["T0"], case["Omega0"], case["hp"], *case["n"]))
    if "kernel" not in names:
        pytest.skip("the profiler records no kernels here")
    assert runs in names and not_runs not in names, names
