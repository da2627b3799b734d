"""The boundary blocks of the cell kernel at the edges of what the mesh tables may hold.  Needs a B200."""
import dataclasses

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["reversed", "shuffled"])
def test_boundary_facets_in_any_order(order):
    """A batch's residual does not depend on the order of its boundary facets (bitwise: each facet's value
    comes from its own cell and its case's characteristic mean, whose order is kept)."""
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    from fvm_solver_b200 import batched as B, workloads as W
    from fvm_solver_b200.corrector import ResidualEval
    cases = [W.channel_cylinder(n_cells=n, solver_name="Butcher", solver_extra="SSP_RK3") for n in (1500, 2011, 1777)]
    for c in cases:
        c.cfg.cfl = None
    b = B.BatchedFVM([B.build_case_tables(c) for c in cases], cases[0].cfg)
    U = b.cells.state.clone()
    want = ResidualEval(b)(U, torch.empty_like(U)).clone()
    kt, ca, _ = B.concat_tables(b.parts)
    n = kt.n_bc
    p = torch.arange(n).flip(0) if order == "reversed" else torch.randperm(n, generator=torch.Generator().manual_seed(0))
    at = torch.empty_like(p)
    at[p] = torch.arange(n)                              # new index of each facet
    moved = {f: getattr(kt, f)[p] for f in ("bc_face", "bc_side", "bc_cell", "bc_kind", "bc_b", "bc_l", "bc_ga",
                                            "bc_gb", "bc_char")}
    cols = kt.g_cols.long()
    moved["g_cols"] = torch.where(cols >= kt.n_cells, kt.n_cells + at[(cols - kt.n_cells).clamp(min=0)], cols).int()
    moved["fbc"] = torch.where(kt.fbc >= 0, at[kt.fbc.long().clamp(min=0)].int(), kt.fbc)
    b.dev = B.BatchedDeviceMesh(dataclasses.replace(kt, **moved), dict(ca, bc_case=ca["bc_case"][p]), b.device)
    assert torch.equal(ResidualEval(b)(U, torch.empty_like(U)), want)
