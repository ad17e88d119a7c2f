"""The heat stepper at the limits of its inputs: sources that are not finite on heat-sinked faces
(held voxels take no source), line matrices far from diagonal dominance (pivots that settle slowly),
contexts of several threads that step grids of one launch class at the same time, and media whose row
coefficients do not fit the code tables."""
import ctypes
import threading
import time

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


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("H", [60.0, 300.0, 1000.0])
def test_uniform_heating_of_a_stiff_line(axis, H):
    """An insulated block of one medium under a uniform source warms up uniformly, by dt Q per step,
    whatever its couplings. With a coupling of H = dt/2 c the pivots settle over about 10 sqrt(H) rows
    and a pivot error is amplified H-fold: FP32 pivots rounded from converged FP64 ones leave at most
    1.5e-6 of the rise (FP32 line solves emulated on the CPU for these H), pivots frozen at the first two
    that round alike 1.2e-5 at H = 300 and 5e-5 at H = 1000. Bound: 5e-6."""
    from mcmatlab_b200 import mexargs, native
    shape = [5, 5, 5]
    shape[axis] = 500
    dt, Q, steps = 0.1, 250.0, 4
    c = np.full((1, 1, 3), 0.5, np.float32)
    c[0, 0, axis] = 2 * H / dt
    T0 = np.full(shape, 20.0, np.float32, order="F")
    hp = mexargs.heat_mex_params(np.ones(shape, np.uint8), [0.0], [0.0], c, np.full(shape, Q, np.float32), True, 0, None,
                                 None, True, steps, dt)
    T, _, _, _ = native.heat_forward(T0, None, hp, *shape)
    rise = steps * dt * Q
    assert np.max(np.abs(T.astype(np.float64) - 20.0 - rise)) <= 5e-6 * rise


@pytest.mark.parametrize("steps", [3, 4])
def test_threads_share_a_launch_class(steps, oracle_lib):
    """Two contexts, one per thread, step grids whose passes are the same kernels with different amounts
    of shared memory. Every call succeeds and gives what it gives alone."""
    from mcmatlab_b200 import abi, native
    lib = native.lib()
    fp = ctypes.POINTER(ctypes.c_float)
    cases = [heatcases.shaped(s, seed=3, nt=steps, with_damage=False) for s in ((126, 40, 40), (18, 40, 40))]
    alone = [native.heat_forward(c["T0"], None, c["hp"], *c["n"])[0] for c in cases]
    errors = []

    def work(k):
        ctx = ctypes.c_void_p()
        assert lib.mcb_ctx_create(0, ctypes.byref(ctx)) == 0
        try:
            hb = abi.HeatParamBuffers(*cases[k]["n"], cases[k]["hp"])
            T0 = np.ascontiguousarray(cases[k]["T0"].reshape(-1, order="F"))
            sens = np.zeros(max(hb.nS * (steps + 1), 1))
            mx = np.zeros(hb.nM, np.float32)
            for rep in range(400):
                T = T0.copy()
                st = lib.mcb_heat_forward(ctx, ctypes.byref(hb.params), T.ctypes.data_as(fp), ctypes.cast(None, fp),
                                          sens.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), mx.ctypes.data_as(fp))
                if st != 0:
                    errors.append((k, rep, lib.mcb_last_error(ctx).decode()))
                    return
                if not np.array_equal(T.reshape(cases[k]["n"], order="F"), alone[k]):
                    errors.append((k, rep, "differs"))
                    return
        finally:
            lib.mcb_ctx_destroy(ctx)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def voxelwise(shape, nM, steps, dt_factor=1.5, seed=1, hs=0):
    """A case whose medium changes from voxel to voxel."""
    from mcmatlab_b200 import mexargs, prep
    rng = np.random.default_rng(seed)
    M1 = rng.integers(1, nM + 1, shape).astype(np.uint8)
    TC, VHC, d = rng.uniform(0.002, 0.006, nM), rng.uniform(3.0, 4.2, nM), 0.01
    c, Q = prep.calc_dTdt_arrays(VHC, TC, d, d, d, 40.0 * rng.random(shape), 1.0, M1)
    dt = dt_factor * float(np.min(VHC / TC)) * d * d / 6
    A, E = np.where(np.arange(nM) % 2, 7.6e66, 0.0), np.where(np.arange(nM) % 2, 4.48e5, 0.0)
    hp = mexargs.heat_mex_params(M1, A, E, c, Q, True, hs, None, None, True, steps, dt)
    T0 = np.asfortranarray((50 + 10 * rng.random(shape)).astype(np.float32))
    return dict(T0=T0, Omega0=np.zeros(shape, np.float32, order="F"), hp=hp, n=shape)


def row_codes(hp):
    """Row coefficients along x, y and z and of the y and z faces as the stepper codes them: distinct media of
    a row and its neighbours, with its FP32 inverse pivot along the lines. More than 255 along an axis do not
    fit."""
    M = np.asarray(hp["M"]).astype(np.int64)
    H = np.float32(hp["dt"] / 2) * np.asarray(hp["dTdtperdeltaT"], np.float32)  # [own, neighbour, axis]
    sinked = np.zeros(M.shape, bool)
    if hp["heatBoundaryType"]:
        sinked[:] = True
        sinked[1:-1, 1:-1, 1:-1] = False
    out = []
    for ax in range(3):
        m, sk = np.moveaxis(M, ax, 0), np.moveaxis(sinked, ax, 0)
        n, keys = m.shape[0], []
        ib, cp = np.zeros(m.shape[1:]), np.zeros(m.shape[1:])
        for i in range(n):
            a = np.where(sk[i], 0, H[m[i], m[max(i - 1, 0)], ax] if i else 0).astype(np.float64)
            c = np.where(sk[i], 0, H[m[i], m[min(i + 1, n - 1)], ax] if i < n - 1 else 0).astype(np.float64)
            ib = 1 / (1 + a + c - a * cp * ib)
            cp = c
            prev = np.where(sk[i] | (i == 0), 0, 256 + m[max(i - 1, 0)])
            nxt = np.where(sk[i] | (i == n - 1), 0, 256 + m[min(i + 1, n - 1)])
            key = (((prev << 9) | nxt) << 8 | m[i]) << 32 | ib.astype(np.float32).view(np.uint32).astype(np.int64)
            keys.append(np.unique(key[~sk[i]] if ax < 2 else key))
        out.append(np.unique(np.concatenate(keys)).size)
    key = M.copy()
    for ax in (1, 2):
        for side in (-1, 1):
            nb = 256 + np.roll(M, -side, ax)
            edge = [slice(None)] * 3
            edge[ax] = 0 if side < 0 else -1
            nb[tuple(edge)] = 0
            key = key << 9 | nb
    out.append(np.unique(key[~sinked]).size)
    return out


def test_row_code_overflow_is_cheap():
    """Four steps on a resident state whose row coefficients overflow the code tables find that out in less
    than the time of a call of three (which does not try): the bound leaves room for a few fold, the full
    search of every failing row was about 15-fold."""
    from mcmatlab_b200 import native
    case = voxelwise((100, 100, 100), 24, 4)
    assert max(row_codes(case["hp"])) > 255
    best = {}
    for steps in (3, 4):
        hp = dict(case["hp"], steps=float(steps))
        st = native.HeatState(case["T0"], case["Omega0"], hp, *case["n"])
        try:
            for _ in range(8):
                t = time.perf_counter()
                st.step(hp)
                best[steps] = min(best.get(steps, 1.0), time.perf_counter() - t)
        finally:
            st.close()
    assert best[4] <= 3 * best[3], best


def test_state_whose_codes_fit_at_some_steps_only(oracle_lib):
    """A resident state steps with codes, without (twice: the second call does not try), with codes at
    the first time step again, and with codes at the time step that overflowed but other coefficients."""
    from mcmatlab_b200 import native
    from oracle import orc
    shape = (40, 37, 100)
    case = voxelwise(shape, 2, 5)
    small, large = (dict(case["hp"], dt=dt) for dt in (1e-6, 0.5))
    weak = dict(large, dTdtperdeltaT=np.float32(1e-6) * large["dTdtperdeltaT"])
    assert max(row_codes(small)) <= 255 and max(row_codes(weak)) <= 255 and max(row_codes(large)) > 255
    T, O = case["T0"].astype(np.float64), case["Omega0"].astype(np.float64)
    st = native.HeatState(case["T0"], case["Omega0"], small, *shape)
    try:
        for hp in (small, large, large, small, weak):
            st.step(hp)
            T, O, _, _ = orc.oracle_heat(T.astype(np.float32), O.astype(np.float32), hp, *shape)
        Tg, _ = st.read()
    finally:
        st.close()
    assert np.max(np.abs(Tg - T) / np.abs(T)) <= 5e-5  # 1e-5 per call, as the stepper's other tests


def test_long_state_whose_codes_fit_at_first(oracle_lib):
    """The same on an axis over 512, where a state whose codes do not fit goes on as a factored one: with
    its temperatures, and with its damage to the bit (no medium adds any here)."""
    from mcmatlab_b200 import native
    from oracle import orc
    shape = (8, 9, 600)
    case = voxelwise(shape, 2, 4)
    O0 = np.asfortranarray(np.random.default_rng(5).random(shape).astype(np.float32))
    none = np.zeros((2, 1))
    calls = [dict(case["hp"], dt=dt, A=none, E=none) for dt in (1e-6, 2.0, 2.0, 1e-6)]
    assert max(row_codes(calls[0])) <= 255 < max(row_codes(calls[1]))
    T = case["T0"].astype(np.float64)
    st = native.HeatState(case["T0"], O0, calls[0], *shape)
    try:
        for k, hp in enumerate(calls):
            st.step(hp)
            T, _, _, _ = orc.oracle_heat(T.astype(np.float32), None, hp, *shape)
            Tg, Og = st.read()
            assert np.max(np.abs(Tg - T) / np.abs(T)) <= 1e-5 * (k + 1)
            np.testing.assert_array_equal(Og, O0)
    finally:
        st.close()


def test_long_calls_in_turn_share_one_block(oracle_lib):
    """Whole calls on one context, some with codes that fit and some without, with and without damage: each
    equals the oracle, and what the context holds for them afterwards is one factored state (66 bytes per
    voxel; the bound leaves room for the allocator's pages), not a streamed one beside it."""
    import torch
    from mcmatlab_b200 import abi, native
    from oracle import orc
    lib, fp = native.lib(), ctypes.POINTER(ctypes.c_float)
    shape = (64, 60, 700)

    def call(ctx, case, hp, damage):
        hb = abi.HeatParamBuffers(*case["n"], hp)
        T = np.ascontiguousarray(case["T0"].reshape(-1, order="F")).copy()
        O = np.zeros(T.size, np.float32)
        mx = np.zeros(hb.nM, np.float32)
        st = lib.mcb_heat_forward(ctx, ctypes.byref(hb.params), T.ctypes.data_as(fp),
                                  O.ctypes.data_as(fp) if damage else ctypes.cast(None, fp),
                                  ctypes.cast(None, ctypes.POINTER(ctypes.c_double)), mx.ctypes.data_as(fp))
        assert st == 0, lib.mcb_last_error(ctx).decode()
        return T.reshape(case["n"], order="F"), O.reshape(case["n"], order="F")

    ctx = ctypes.c_void_p()
    assert lib.mcb_ctx_create(0, ctypes.byref(ctx)) == 0
    try:
        small, case = voxelwise((16, 8, 520), 2, 3), voxelwise(shape, 2, 3)
        for dt in (1e-6, 2.0):  # loads the kernels
            call(ctx, small, dict(small["hp"], dt=dt), True)
        free = torch.cuda.mem_get_info(0)[0]
        for dt, damage in ((2.0, True), (1e-6, True), (2.0, True), (1e-6, False), (2.0, False)):
            hp = dict(case["hp"], dt=dt)
            T, O = call(ctx, case, hp, damage)
            To, Oo, _, _ = orc.oracle_heat(case["T0"], np.zeros(shape, np.float32) if damage else None, hp, *shape)
            assert np.max(np.abs(T - To) / np.abs(To)) <= 1e-5
            if damage:
                assert np.max(np.abs(O - Oo)) <= 1e-4 * np.max(Oo)
        held = free - torch.cuda.mem_get_info(0)[0]
        assert held <= 72 * np.prod(shape) + (8 << 20), held / np.prod(shape)
    finally:
        lib.mcb_ctx_destroy(ctx)


def test_adjoint_gives_large_states_back():
    """After an adjoint on 8.4 million voxels the context holds its work memory (ten grids and the pool's eighth:
    45 bytes per voxel) and not the two states beside it (another 90)."""
    import torch
    from mcmatlab_b200 import abi, native
    lib, fp = native.lib(), ctypes.POINTER(ctypes.c_float)

    def call(ctx, shape):
        case = voxelwise(shape, 2, 2)
        hb = abi.HeatParamBuffers(*shape, case["hp"])
        T = np.ascontiguousarray(case["T0"].reshape(-1, order="F"))
        w = np.zeros(T.size, np.float32)
        w[T.size // 2:T.size // 2 + 9] = 1.0
        obj, g = abi.mcb_heat_objective(), abi.mcb_heat_grad()
        obj.damageWeight, obj.peakWeight = w.ctypes.data_as(fp), ctypes.cast(None, fp)
        dT = np.zeros(T.size, np.float32)
        g.dJ_dT0 = dT.ctypes.data_as(fp)
        assert lib.mcb_heat_adjoint(ctx, ctypes.byref(hb.params), T.ctypes.data_as(fp), ctypes.byref(obj), 0, ctypes.byref(g)) == 0
        return dT

    ctx = ctypes.c_void_p()
    assert lib.mcb_ctx_create(0, ctypes.byref(ctx)) == 0
    try:
        small = call(ctx, (30, 28, 24))
        free = torch.cuda.mem_get_info(0)[0]
        shape = (256, 256, 128)
        big = call(ctx, shape)
        held = free - torch.cuda.mem_get_info(0)[0]
        assert held <= 50 * np.prod(shape), held / np.prod(shape)
        np.testing.assert_allclose(call(ctx, shape), big, rtol=1e-4, atol=1e-6 * np.abs(big).max())
        np.testing.assert_allclose(call(ctx, (30, 28, 24)), small, rtol=1e-4, atol=1e-6 * np.abs(small).max())
    finally:
        lib.mcb_ctx_destroy(ctx)
