"""Tiled tables: their content against the row records (CPU) and the launches that read them against
the row launches (GPU, bitwise: same terms in the same order)."""
import pytest
import torch

from fvm_solver_b200 import workloads as W
from fvm_solver_b200.tables import tiled_records

MESHES = {"channel": lambda: W.channel_cylinder(n_cells=1500), "channel_odd": lambda: W.channel_cylinder(n_cells=2011),
          "box": lambda: W.taylor_green(4), "sphere": lambda: W.sphere(3000)}


def _untile(t, n, quads):
    return t.view(-1, quads, 32, 4).permute(0, 2, 1, 3).reshape(-1, 4 * quads)[:n]


@pytest.mark.parametrize("name", sorted(MESHES))
def test_tiles_hold_the_rows(name):
    kt = MESHES[name]().tables().kernel
    rec = kt.records()
    t = tiled_records(kt.dim, kt.kg, kt.kf, rec)
    dim, N, F = kt.dim, kt.n_cells, kt.n_facets
    ints = lambda x: x.contiguous().view(torch.int32).long()
    assert torch.equal(_untile(t["cell_tiles"], N, 5 if dim == 2 else 8).view(torch.int32), rec["cell_rec"].view(torch.int32))
    f = _untile(t["face_tiles"], F, 3 if dim == 2 else 4)
    assert torch.equal(f.view(torch.int32), rec["face_rec"][:, :4 + 4 * dim].contiguous().view(torch.int32))
    if dim == 2:
        d = _untile(t["div_tiles"], N, 1)
        ids, vol = ints(d[:, :3]), d[:, 3]
    else:
        d = t["div_tiles"]
        ids, vol = ints(d[:, :128].reshape(-1, 4)[:N]), d[:, 128:].reshape(-1)[:N]
    assert torch.equal(torch.where(ids < 0, -vol[:, None], vol[:, None]), kt.f_vals.t())
    assert torch.equal(ids & 0x7fffffff, kt.f_cols.t().long())


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(MESHES))
@pytest.mark.parametrize("solver", ["Butcher/RK4", "RK3_SSP4/"])
def test_tiled_launches_equal_rows(name, solver):
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    out = {}
    for tiles in (True, False):
        case = MESHES[name]()
        case.cfg.solver_name, case.cfg.solver_extra = solver.split("/")
        eq = case.equation()
        if not tiles:
            eq.dev.struct.cell_tiles = eq.dev.struct.face_tiles = eq.dev.struct.div_tiles = None
        prims = eq.cells.get_values()[0].contiguous()
        r = [eq.forward(prims).clone(), eq.forward(prims * 1.01).clone(), eq.grads.clone()]
        eq.reset_gradients()
        eq.t_solver.step(3)
        out[tiles] = r + [eq.cells.state.clone(), eq.t_solver.dt.clone(), eq.grads.clone()]
    for a, b in zip(out[True][:5], out[False][:5]):
        if a.numel() > 1 or not solver.startswith("RK3_SSP4"):
            assert torch.equal(a, b)
        else:                                       # adaptive dt: FP64 atomics in any order
            assert float((a - b).abs() / b) < 1e-6


@pytest.mark.gpu
def test_tiled_batch_equals_rows_with_mask():
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    from fvm_solver_b200 import batched as B
    cases = [W.channel_cylinder(n_cells=n, solver_name="Butcher", solver_extra="SSP_RK3") for n in (1500, 2011, 1777)]
    for c in cases:
        c.cfg.cfl = None
    parts = [B.build_case_tables(c) for c in cases]
    out = {}
    for tiles in (True, False):
        b = B.BatchedFVM(parts, cases[0].cfg)
        if not tiles:
            b.dev.struct.cell_tiles = b.dev.struct.face_tiles = b.dev.struct.div_tiles = None
        b.t_solver.update_cfl_dt(0.5)
        b.t_solver.step(2)
        b.use_case_mask(True)
        b.active.copy_(torch.tensor([1, 0, 1], dtype=torch.uint8))
        b.t_solver.step(2)
        out[tiles] = (b.cells.state.clone(), b.grads.clone())
    assert all(torch.equal(x, y) for x, y in zip(out[True], out[False]))
