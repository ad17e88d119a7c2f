"""The transport's launch parameters are what runs: a context takes them from the tuning file, for every
value of their range, and the results do not depend on them."""
import ctypes

import numpy as np
import pytest

from mcmatlab_b200 import configs, mexargs

pytestmark = pytest.mark.gpu


def test_scatter_group_of_the_tuning_file_is_used(tmp_path, monkeypatch):
    """Groups of 8, 16 and 32 of a full warp's lanes: waiting for all 32 leaves most lanes of a warp idle, so the
    kernel takes at least a tenth longer than with 8 (a group capped at 8 takes the same time)."""
    import torch
    from mcmatlab_b200 import abi, native
    lib = native.lib()
    mc_in = mexargs.prepare_mc(configs.standard_tissue_cube(n=60, nPhotons=4e5, seed=5))
    mb = abi.McModelBuffers(mc_in)
    cls = int(lib.mcb_mc_size_class(ctypes.byref(mb.model), 0, 0))
    path = tmp_path / "tune.txt"
    monkeypatch.setenv("MCB_TUNE_FILE", str(path))
    ms, out = {}, {}
    for group in (8, 16, 32):
        path.write_text("%s\t%d\t12\t%d\n" % (torch.cuda.get_device_name(0), cls, group))
        ctx = ctypes.c_void_p()
        assert lib.mcb_ctx_create(0, ctypes.byref(ctx)) == 0
        try:
            for _ in range(5):
                rb = abi.McResultBuffers(mc_in)
                assert lib.mcb_mc_run(ctx, ctypes.byref(mb.model), ctypes.byref(rb.result)) == 0
                ms[group] = min(ms.get(group, np.inf), rb.result.kernelMs)
            out[group] = rb.outputs()
        finally:
            lib.mcb_ctx_destroy(ctx)
    assert ms[32] >= 1.1 * ms[8], ms
    for group in (16, 32):
        assert out[group]["propagationSteps"] == out[8]["propagationSteps"]
        np.testing.assert_allclose(out[group]["NFR"], out[8]["NFR"], rtol=1e-6, atol=1e-9 * float(out[8]["NFR"].max()))
