"""The corrector's layer kernels at tile edges: forward forms against GEMM + gather kernels (bitwise),
the backward kernels against FP64 products of the same operands.  Needs a B200.

Tolerances: products of bf16 values are exact in fp32 and at most 128 (rows: a few thousand) of them are
summed in fp32, so rel-L2 <= 1e-5 against FP64; SiLU' uses the fast exponential (2 ulp of its argument's
range, below 1e-6), so dZ rounds to the same bf16 up to rare ties (rel-L2 <= 1e-4) and a column sum
agrees with a running fp32 sum of the recomputed terms to 1e-5 of the sum of magnitudes.
"""
import ctypes as ct

import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")


def _rand(*shape, seed, scale=1.0, bf=False):
    t = scale * torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))
    return t.to(torch.bfloat16) if bf else t


def _nbr(N, KN, seed):
    """Symmetric adjacency: a ring with offsets, some links missing."""
    g = np.random.default_rng(seed)
    n = np.full((N, KN), -1, np.int32)
    used = np.zeros(N, int)
    for off in range(1, KN + 1):
        for i in g.permutation(N)[: max(1, N // 2)]:
            j = (i + off * 3) % N
            if j != i and used[i] < KN and used[j] < KN:
                n[i, used[i]], n[j, used[j]] = j, i
                used[i] += 1
                used[j] += 1
    return torch.from_numpy(n).cuda()


@pytest.mark.parametrize("N,KN,O", [(1, 1, 1), (127, 3, 4), (128, 4, 5), (129, 8, 8), (1000, 5, 3)])
def test_forward_forms(N, KN, O):
    from fvm_solver_b200 import _lib
    lib, s = _lib.load(), _lib.stream_ptr()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    X, Win, bias = _rand(N, 64, seed=1, bf=True), _rand(64, 64, seed=2, scale=0.1, bf=True), _rand(64, seed=3)
    want, zw = torch.empty(N, 64, device="cuda"), torch.empty(N, 64, device="cuda")
    _lib.check(lib.fvm_gemm_bf16(X.data_ptr(), 64, Win.data_ptr(), 64, N, 64, 64, 1, bias.data_ptr(), None, 0,
                                 want.data_ptr(), None, 64, zw.data_ptr(), 1, err.data_ptr(), s), "gemm")
    h, z = torch.full_like(want, float("nan")), torch.full_like(want, float("nan"))
    _lib.check(lib.fvm_in_layer(X.data_ptr(), N, Win.data_ptr(), bias.data_ptr(), h.data_ptr(), z.data_ptr(),
                                err.data_ptr(), s), "in_layer")
    assert torch.equal(h, want) and torch.equal(z, zw)
    nbr, Wt = _nbr(N, KN, 4), _rand(64, 128, seed=5, scale=0.1, bf=True)
    Wo, bo = _rand(O, 64, seed=6), _rand(O, seed=7)
    A = torch.empty(N, 128, dtype=torch.bfloat16, device="cuda")
    _lib.check(lib.fvm_mp_gather_f32(h.data_ptr(), nbr.data_ptr(), N, KN, A.data_ptr(), s), "gather")
    _lib.check(lib.fvm_gemm_bf16(A.data_ptr(), 128, Wt.data_ptr(), 128, N, 64, 128, 1, bias.data_ptr(), h.data_ptr(),
                                 64, want.data_ptr(), None, 64, zw.data_ptr(), 1, err.data_ptr(), s), "gemm")
    out_w = torch.empty(N, O, device="cuda")
    _lib.check(lib.fvm_decoder_f32(want.data_ptr(), Wo.data_ptr(), bo.data_ptr(), N, O, out_w.data_ptr(), s), "dec")
    h2, z2, out = torch.full_like(want, float("nan")), torch.full_like(want, float("nan")), torch.empty_like(out_w)
    A2 = torch.zeros_like(A)
    _lib.check(lib.fvm_mp_layer_train(h.data_ptr(), nbr.data_ptr(), N, KN, Wt.data_ptr(), bias.data_ptr(),
                                      h2.data_ptr(), z2.data_ptr(), A2.data_ptr(), Wo.data_ptr(), bo.data_ptr(), O,
                                      out.data_ptr(), err.data_ptr(), s), "layer")
    assert torch.equal(A2, A) and torch.equal(z2, zw) and torch.equal(h2, want) and torch.equal(out, out_w)
    assert int(err.item()) == 0


@pytest.mark.parametrize("N,KN,O", [(1, 1, 1), (127, 3, 4), (129, 4, 5), (700, 8, 8), (40_001, 3, 4), (100_001, 4, 5)])
def test_backward_kernels(N, KN, O):
    from fvm_solver_b200 import _lib
    lib, s = _lib.load(), _lib.stream_ptr()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    h, Wo, dout, Z1, Z0 = (_rand(N, 64, seed=1).abs(), _rand(O, 64, seed=2), _rand(N, O, seed=3).abs() + 0.1,
                           _rand(N, 64, seed=4), _rand(N, 64, seed=5))
    A, Wt, X = _rand(N, 128, seed=6, bf=True), _rand(64, 128, seed=7, scale=0.1, bf=True), _rand(N, 64, seed=8, bf=True)
    WT, nbr = Wt.t().contiguous(), _nbr(N, KN, 9)
    sums = torch.full((O + 3, _lib.FVM_BACK_SET), float("nan"), device="cuda")
    f = lambda *sh: torch.full(sh, float("nan"), device="cuda")
    dh, dh0, dA, dZ = f(N, 64), f(N, 64), f(N, 128), torch.empty(N, 64, dtype=torch.bfloat16, device="cuda")
    dZ0, dW, dWin = torch.empty_like(dZ), torch.zeros(64, 128, device="cuda"), torch.zeros(64, 64, device="cuda")
    P = lambda t: t.data_ptr()
    dec, b1, b0 = P(sums[2]), P(sums[1]), P(sums[0])
    _lib.check(lib.fvm_back_top(P(h), P(Wo), P(dout), P(Z1), N, O, P(dh), P(dZ), dec, b1, s), "top")
    _lib.check(lib.fvm_back_decoder(P(h), P(dout), N, O, dec, s), "decoder")
    _lib.check(lib.fvm_back_layer(P(dZ), P(A), P(WT), P(nbr), KN, N, P(dA), P(dW), P(err), s), "layer")
    _lib.check(lib.fvm_back_gather(P(dA), P(nbr), N, KN, P(dh), P(Z1), b1, P(Z0), P(dh0), P(dZ0), b0, s), "gather")
    _lib.check(lib.fvm_back_layer(P(dZ0), P(X), None, None, 0, N, None, P(dWin), P(err), s), "input layer")
    _lib.check(lib.fvm_back_bias(P(dh0), P(Z0), N, b0, s), "bias")
    db = torch.zeros(2, 64, device="cuda")
    dWo, dbo = torch.zeros(O, 64, device="cuda"), torch.zeros(O, device="cuda")
    dst = [db[0], db[1]] + [dWo[o] for o in range(O)] + [dbo]
    n = len(dst)
    _lib.check(lib.fvm_back_finish(n, (ct.c_void_p * n)(*[P(sums[q]) for q in range(n)]),
                                   (ct.c_void_p * n)(*[P(t) for t in dst]), (ct.c_int32 * n)(*([64] * (n - 1) + [O])), s),
               "finish")
    assert int(err.item()) == 0
    rel = lambda a, b: rel_l2(a.double().cpu().numpy(), b.double().cpu().numpy())
    grad = lambda d, z: d * torch.sigmoid(z) * (1 + z * (1 - torch.sigmoid(z)))
    # products and the gather, each from the operands its kernel read
    assert rel(dh, dout.double() @ Wo.double()) < 1e-5
    assert rel(dZ, grad(dh, Z1).to(torch.bfloat16)) < 1e-4
    want = dZ.double() @ Wt.double()
    deg = (nbr >= 0).sum(1, keepdim=True).clamp(min=1)
    want[:, 64:] /= deg
    assert rel(dA, want) < 1e-5
    assert rel(dW, dZ.double().t() @ A.double()) < 1e-5
    assert rel(dWin, dZ0.double().t() @ X.double()) < 1e-5
    m = dh.double() + dA[:, :64].double()
    for k in range(KN):
        j = nbr[:, k].long()
        m += torch.where((j >= 0)[:, None], dA[j.clamp(min=0), 64:].double(), 0.0)
    assert rel(dh0, m) < 1e-5
    assert rel(dZ0, grad(dh0, Z0).to(torch.bfloat16)) < 1e-4
    # column sums: one running fp32 sum over the rows
    run = lambda t: torch.from_numpy(np.cumsum(t.float().cpu().numpy(), axis=0, dtype=np.float32)[-1])
    for got, t in [(db[0], grad(dh0, Z0)), (db[1], grad(dh, Z1)), (dbo, dout)] + \
            [(dWo[o], dout[:, o:o + 1] * h) for o in range(O)]:
        assert float(((got.cpu() - run(t)).abs() / t.abs().sum(0).cpu()).max()) < 1e-5


@pytest.mark.parametrize("N,C,G,cases", [(1, 4, 0, 1), (129, 4, 11, 2), (1000, 5, 18, 3)])
def test_inputs_in_the_input_layer_and_proposal(N, C, G, cases):
    """fvm_corrector_in_layer against fvm_corrector_inputs + fvm_in_layer, fvm_corrector_propose against
    fvm_corrector_combine with the shift formed in torch: bitwise."""
    from fvm_solver_b200 import _lib
    lib, s = _lib.load(), _lib.stream_ptr()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    U, r0, mean, inv = _rand(N, C, seed=1), _rand(N, C, seed=2), _rand(2 * C, seed=3), _rand(2 * C, seed=4).abs()
    geo, W, bias = _rand(N, max(G, 1), seed=5), _rand(64, 64, seed=6, scale=0.1, bf=True), _rand(64, seed=7)
    dt, k = _rand(cases, seed=8).abs(), 8
    cc = torch.sort(torch.randint(0, cases, (N,), device="cuda", dtype=torch.int32)).values
    kdt = dt * float(k)
    P = lambda t: t.data_ptr()
    X, base = torch.zeros(N, 64, dtype=torch.bfloat16, device="cuda"), torch.empty(N, C, device="cuda")
    _lib.check(lib.fvm_corrector_inputs(P(U), P(r0), P(kdt), P(cc), N, C, P(mean), P(inv), P(geo), G, P(base), P(X), 64, s), "inputs")
    want, got, base2 = torch.empty(N, 64, device="cuda"), torch.empty(N, 64, device="cuda"), torch.empty(N, C, device="cuda")
    _lib.check(lib.fvm_in_layer(P(X), N, P(W), P(bias), P(want), None, P(err), s), "in_layer")
    _lib.check(lib.fvm_corrector_in_layer(P(U), P(r0), P(dt), k, P(cc), N, C, P(mean), P(inv), P(geo), G, P(base2), P(W),
                                          P(bias), P(got), P(err), s), "corrector_in_layer")
    assert torch.equal(got, want) and torch.equal(base2, base) and int(err.item()) == 0
    out, scale = _rand(N, C, seed=9), _rand(C, seed=10).abs()
    sums, vol = _rand(cases, C, seed=11).double(), _rand(cases, seed=12).double().abs() + 0.1
    shift = torch.zeros(cases, C, device="cuda")
    shift[:, C - 2:] = (sums[:, C - 2:] / vol[:, None] * scale[C - 2:].double()).float()
    a, b = torch.empty(N, C, device="cuda"), torch.empty(N, C, device="cuda")
    _lib.check(lib.fvm_corrector_combine(P(U), P(base), P(out), P(scale), P(shift), P(cc), N, C, P(a), s), "combine")
    _lib.check(lib.fvm_corrector_propose(P(U), P(base), P(out), P(scale), P(sums), P(vol), C - 2, P(cc), N, C, P(b), s), "propose")
    assert torch.equal(a, b)


def test_adam_many():
    """fvm_adam_many on tensors of different sizes against fvm_adam one by one: bitwise."""
    from fvm_solver_b200 import _lib
    lib, s = _lib.load(), _lib.stream_ptr()
    shapes = [(4, 64), (1, 64), (64, 128), (1, 4), (64, 64), (3, 1)]
    def tensors():
        out = []
        for q, (r, c) in enumerate(shapes):
            p, g, m = (_rand(r, c, seed=3 * q + e) for e in range(3))
            pb = torch.zeros(r, c, dtype=torch.bfloat16, device="cuda") if q % 2 == 0 else None
            pbT = torch.zeros(c, r, dtype=torch.bfloat16, device="cuda") if q % 3 == 2 else None
            out.append([p, g, m, m.square(), pb, pbT])
        return out
    P = lambda t: None if t is None else t.data_ptr()
    want, got = tensors(), tensors()
    for (r, c), (p, g, m, v, pb, pbT) in zip(shapes, want):
        _lib.check(lib.fvm_adam(P(p), P(g), P(m), P(v), r * c, 1e-3, 0.9, 0.999, 1e-8, 3, P(pb), P(pbT), r, c, s), "adam")
    n = len(shapes)
    A = lambda e: (ct.c_void_p * n)(*[P(t[e]) for t in got])
    sizes = (ct.c_int64 * n)(*[r * c for r, c in shapes])
    rows, cols = (ct.c_int32 * n)(*[r for r, _ in shapes]), (ct.c_int32 * n)(*[c for _, c in shapes])
    _lib.check(lib.fvm_adam_many(n, A(0), A(1), A(2), A(3), sizes, 1e-3, 0.9, 0.999, 1e-8, 3, A(4), A(5), rows, cols, s),
               "adam_many")
    for a, b in zip(want, got):
        for x, y in zip(a, b):
            assert x is None or torch.equal(x, y)
    assert lib.fvm_adam_many(0, A(0), A(1), A(2), A(3), sizes, 1e-3, 0.9, 0.999, 1e-8, 3, A(4), A(5), rows, cols, s) != 0
