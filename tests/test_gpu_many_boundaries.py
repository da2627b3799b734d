"""A batch whose boundary facets alone fill much of a wave of blocks: each copy of a case steps
bitwise as the case alone (both sides of the cell kernel's grid rule).  Needs a B200."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [2, 200])
def test_many_boundary_blocks(copies):
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    from fvm_solver_b200 import batched as B, workloads as W
    p = W.ensemble_params(0)
    p["n_cells"] = 2100
    c = W.channel_cylinder(device="cuda", solver_name="AB3", solver_extra="SSP_RK3", cfl=0.3, **p)
    part = B.build_case_tables(c)
    one = B.BatchedFVM([part], c.cfg, device="cuda")
    many = B.BatchedFVM([part] * copies, c.cfg, device="cuda")
    one.t_solver.step(4)
    many.t_solver.step(4)
    for k in range(copies):
        assert torch.equal(many.case_state(k), one.case_state(0)), f"copy {k}"
