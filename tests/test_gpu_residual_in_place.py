"""fvm_residual whose result replaces its primitives, in each form of the divergence.  Needs a B200."""
import ctypes as ct

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("mesh", ["channel", "box"])
def test_result_may_replace_primitives(mesh, variant):
    """dudt == prims: bitwise the result of a call with its own output, also where the kernel that stores
    dudt evaluates the facets itself (variant 1)."""
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    from fvm_solver_b200 import _lib, workloads as W
    from fvm_solver_b200.autotune import set_variant
    eq = (W.channel_cylinder(n_cells=30_000) if mesh == "channel" else W.taylor_green(12)).equation()
    prims = eq.cells.get_values()[0].contiguous()
    set_variant("div_stage", variant)
    try:
        eq.reset_gradients()
        want = eq.forward(prims).clone()
        for _ in range(5):
            eq.reset_gradients()
            x = prims.clone()
            _lib.check(eq.lib.fvm_residual(ct.byref(eq.dev.struct), ct.byref(eq.phys), x.data_ptr(), eq.grads.data_ptr(),
                                           eq.has_grads.data_ptr(), x.data_ptr(), ct.byref(eq.work.struct),
                                           _lib.stream_ptr()), "fvm_residual")
            assert torch.equal(x, want)
    finally:
        set_variant("div_stage", 0)
