"""ELL products over the forms their kernels are chosen by (slots, columns, rows, strides, alignment,
bias) against FP64.  Needs a B200.  Tolerance: K <= 16 products summed in fp32, 1e-6 of the sum of
magnitudes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operator(M, N, K, seed):
    from fvm_solver_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(seed)
    vals = torch.randn(K, M, device="cuda", generator=g)
    cols = torch.randint(0, N, (K, M), device="cuda", generator=g, dtype=torch.int32)
    cols[:, -1] = N - 1                                   # the operand's last row
    return _lib.load(), vals, cols


@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 7, 16])
@pytest.mark.parametrize("M", [1, 255, 4097, 700_001])
def test_products(K, M):
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    from fvm_solver_b200 import _lib
    N = 3001
    lib, vals, cols = _operator(M, N, K, 100 * K + M % 97)
    g = torch.Generator(device="cuda").manual_seed(K)
    bias = torch.randn(M, device="cuda", generator=g)
    s = _lib.stream_ptr()
    for B, ld, off, with_bias in [(1, 1, 0, True), (1, 3, 1, False), (2, 2, 0, False), (4, 4, 0, True), (5, 5, 0, False),
                                  (5, 5, 1, True), (5, 5, 3, True), (5, 7, 2, False), (8, 8, 0, True), (9, 9, 0, False)]:
        store = torch.randn(N * ld + off, device="cuda", generator=g)
        X = store[off:off + N * ld].view(N, ld)[:, :B]
        Y = torch.full((M, B), float("nan"), device="cuda")
        b = bias.data_ptr() if with_bias else None
        if B == 1:
            rc = lib.fvm_ell_spmv(vals.data_ptr(), cols.data_ptr(), M, K, X.data_ptr(), ld, b, Y.data_ptr(), 1, s)
        else:
            rc = lib.fvm_ell_spmm(vals.data_ptr(), cols.data_ptr(), M, K, X.data_ptr(), ld, B, b, Y.data_ptr(), B, s)
        assert rc == 0
        want, size = torch.zeros(M, B, device="cuda", dtype=torch.float64), torch.zeros(M, B, device="cuda", dtype=torch.float64)
        for k in range(K):
            t = vals[k][:, None].double() * X.double()[cols[k].long()]
            want += t
            size += t.abs()
        if with_bias:
            want += bias[:, None].double()
            size += bias[:, None].double().abs()
        assert float(((Y.double() - want).abs() / size).max()) < 1e-6, (B, ld, off)
