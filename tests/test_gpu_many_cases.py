"""CFL time steps and conservation sums of batches on both sides of 256 cases (one pass of the last block,
or blocks of their own).  Needs a B200."""
import ctypes as ct

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 256, 257, 300])
def test_reductions_of_many_cases(copies):
    """Each copy of a case gets the case's own values: the maximum exactly, the FP64 sums to 1e-12 of the
    largest (their order differs)."""
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    from fvm_solver_b200 import _lib, batched as B, workloads as W
    c = W.channel_cylinder(n_cells=600, solver_name="Butcher", solver_extra="SSP_RK3")
    c.cfg.cfl = None
    part = B.build_case_tables(c)
    out = []
    for n in (1, copies):
        b = B.BatchedFVM([part] * n, c.cfg)
        dt, S = torch.zeros(n, device="cuda"), torch.zeros(n, b.n_comp, dtype=torch.float64, device="cuda")
        for _ in range(2):                               # the second call finds the first one's sums cleared
            _lib.check(b.lib.fvm_cfl_dt(ct.byref(b.dev.struct), ct.byref(b.phys), b.cells.state.data_ptr(), 0.3,
                                        dt.data_ptr(), ct.byref(b.work.struct), _lib.stream_ptr()), "fvm_cfl_dt")
            _lib.check(b.lib.fvm_conservation(ct.byref(b.dev.struct), b.cells.state.data_ptr(), S.data_ptr(),
                                              ct.byref(b.work.struct), _lib.stream_ptr()), "fvm_conservation")
        out.append((dt, S))
    (dt1, S1), (dt, S) = out
    assert float(dt1) > 0 and torch.equal(dt, dt1.expand(copies))
    assert float((S - S1).abs().max()) < 1e-12 * float(S1.abs().max())
