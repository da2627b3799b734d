"""Meshes whose row tables take a large share of the device's memory.  Needs a B200."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", ["channel", "box"])
def test_large_tables_run_from_the_rows(mesh, monkeypatch):
    """Past the share the tiled copies are left out, and a step's result stays the same bit for bit."""
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    from fvm_solver_b200 import equation, workloads as W
    out = {}
    for share in (equation.TILED_SHARE, 1e-9):
        monkeypatch.setattr(equation, "TILED_SHARE", share)
        case = W.channel_cylinder(n_cells=1500) if mesh == "channel" else W.taylor_green(4)
        case.cfg.solver_name, case.cfg.solver_extra = "Butcher", "RK4"
        eq = case.equation()
        rows, tiles = (sum(getattr(eq.dev.t, f).numel() for f in fs if hasattr(eq.dev.t, f))
                       for fs in (("cell_rec", "div_rec", "face_rec"), ("cell_tiles", "div_tiles", "face_tiles")))
        assert tiles == 0 if share < 1e-6 else 0.5 * rows < tiles <= 1.5 * rows
        eq.t_solver.step(2)
        out[share] = eq.cells.state.clone()
    a, b = out.values()
    assert torch.equal(a, b)
