"""ELL products with more than five slots, on both sides of each rule that picks their kernel (slots 6 / 7,
8 / 9 and 12 / 13, whole groups of eight columns), against FP64.  Needs a B200.  Tolerance:
at most 16 products summed in fp32, 1e-6 of the sum of magnitudes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [6, 7, 8, 9, 12, 13])
@pytest.mark.parametrize("M", [257, 1_100_001])
def test_wide_products(K, M):
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    from fvm_solver_b200 import _lib
    lib, N, s = _lib.load(), 3001, _lib.stream_ptr()
    g = torch.Generator(device="cuda").manual_seed(100 * K + M % 97)
    vals = torch.randn(K, M, device="cuda", generator=g)
    cols = torch.randint(0, N, (K, M), device="cuda", generator=g, dtype=torch.int32)
    bias = torch.randn(M, device="cuda", generator=g)
    for B, ld, b in [(1, 1, None), (1, 2, bias), (2, 2, bias), (7, 7, None), (8, 9, bias), (9, 9, None), (16, 16, None)]:
        X = torch.randn(N, ld, device="cuda", generator=g)[:, :B]
        Y = torch.full((M, B), float("nan"), device="cuda")
        if B == 1:
            rc = lib.fvm_ell_spmv(vals.data_ptr(), cols.data_ptr(), M, K, X.data_ptr(), ld, _lib.ptr(b), Y.data_ptr(), 1, s)
        else:
            rc = lib.fvm_ell_spmm(vals.data_ptr(), cols.data_ptr(), M, K, X.data_ptr(), ld, B, _lib.ptr(b), Y.data_ptr(), B, s)
        assert rc == 0
        want = torch.zeros(M, B, device="cuda", dtype=torch.float64) + (0.0 if b is None else b.double()[:, None])
        size = want.abs()
        for k in range(K):
            t = vals[k][:, None].double() * X.double()[cols[k].long()]
            want += t
            size += t.abs()
        assert float(((Y.double() - want).abs() / size).max()) < 1e-6, (B, ld)
