"""Corrector kernels and entry points at the edges of what they take.  Needs a B200."""
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


def _rand(*shape, seed, scale=1.0):
    return scale * torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 5, 6])
def test_input_layer_gradient_waits_for_its_products(tiles):
    """The input layer's dW = dZ^T X with 1 to 6 tiles of 128 rows per CTA (no reader follows the tiles'
    barriers there), many launches in a row.  Products of bf16 values are exact in fp32 and summed in
    fp32: rel-L2 <= 1e-5 against FP64, as for the other sizes of this kernel."""
    from fvm_solver_b200 import _lib
    lib, s = _lib.load(), _lib.stream_ptr()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    N = 128 * (sms * tiles) - 5
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    dZ, X = _rand(N, 64, seed=tiles).bfloat16(), _rand(N, 64, seed=10 + tiles).bfloat16()
    dW = torch.zeros(24, 64, 64, device="cuda")
    for q in range(24):
        _lib.check(lib.fvm_back_layer(dZ.data_ptr(), X.data_ptr(), None, None, 0, N, None, dW[q].data_ptr(),
                                      err.data_ptr(), s), "fvm_back_layer")
    want = (dZ.double().t() @ X.double()).cpu().numpy()
    assert int(err.item()) == 0
    for q in range(24):
        assert rel_l2(dW[q].double().cpu().numpy(), want) < 1e-5


@pytest.fixture(scope="module")
def batch():
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    from fvm_solver_b200 import batched as B, workloads as W
    cases, params = [], []
    for i, n in enumerate([1500, 2011]):
        p = W.ensemble_params(i)
        p["n_cells"] = n
        c = W.channel_cylinder(device="cuda", solver_name="Butcher", solver_extra="SSP_RK3", **p)
        c.cfg.cfl = None
        cases.append(c)
        params.append([p["mach"], np.log10(p["reynolds"])])
    b = B.BatchedFVM([B.build_case_tables(c) for c in cases], cases[0].cfg, device="cuda")
    b.t_solver.update_cfl_dt(0.5)
    return b, torch.tensor(params, dtype=torch.float32)


def _model(batch):
    """(model, state, residual) on the batch, normalised."""
    from fvm_solver_b200.corrector import CorrectorModel
    b, params = batch
    m = CorrectorModel(b, params, seed=3)
    U = b.cells.state.clone()
    r0 = m.res(U, torch.empty_like(U))
    m.set_normalisation(torch.cat([U, U * 1e-3], 1).unsqueeze(0), (U * 1e-3 + 1e-3).unsqueeze(0))
    return m, U, r0


def test_proposal_leaves_its_features_to_the_network(batch):
    """After ``predict`` the network's input rows are those of its state, as after ``inputs`` (bitwise)."""
    m, U, r0 = _model(batch)
    m.inputs(U * 1.01, r0)
    m.predict(U, torch.empty_like(U), r0)
    out, X = m.net._bufs["out"].clone(), m.net._bufs["X"].clone()
    assert torch.equal(m.net.forward(m.nbr), out)
    assert torch.equal(m.inputs(U, r0), X)


def test_network_without_layers():
    """layers=0: the decoder reads the input layer's activations.  The bf16 products are exact in fp32 and
    summed in fp32, SiLU by the fast exponential: rel-L2 <= 1e-5 of FP64."""
    from fvm_solver_b200.corrector import CorrectorNet
    N = 300
    net = CorrectorNet(3, layers=0, seed=1, lr=1e-2)
    X = net._alloc(N)["X"]
    X[:N].copy_(_rand(N, 64, seed=2))
    nbr = torch.full((N, 3), -1, dtype=torch.int32, device="cuda")
    h = torch.nn.functional.silu(X[:N].double() @ net.bf["W_in"].double().t() + net.params["b_in"].double())
    want = h @ net.params["W_out"].double().t() + net.params["b_out"].double()
    for store_pre in (False, True):
        net._bufs["out"].zero_()
        out = net.forward(nbr, store_pre=store_pre)
        assert rel_l2(out.double().cpu().numpy(), want.cpu().numpy()) < 1e-5
    assert float(net.train_step(nbr, want.float() + 1.0)) == pytest.approx(1.0, rel=1e-4)
    assert float(net.params["b_out"].abs().min()) > 0


def test_column_sums_with_infinite_terms():
    """A sum with an infinite term is infinite, not NaN, and the others stay finite."""
    from fvm_solver_b200 import _lib
    lib, s = _lib.load(), _lib.stream_ptr()
    N, O = 5000, 4
    P = lambda t: t.data_ptr()
    h, Wo, dout, Z = _rand(N, 64, seed=1).abs(), _rand(O, 64, seed=2), _rand(N, O, seed=3).abs() + 0.1, _rand(N, 64, seed=4)
    h[2000, 5] = float("inf")
    dout[3000, 2] = float("inf")
    sums = torch.empty((O + 2, _lib.FVM_BACK_SET), device="cuda")
    dh, dZ = torch.empty(N, 64, device="cuda"), torch.empty(N, 64, device="cuda", dtype=torch.bfloat16)
    _lib.check(lib.fvm_back_top(P(h), P(Wo), P(dout), P(Z), N, O, P(dh), P(dZ), P(sums[1]), P(sums[0]), s), "top")
    _lib.check(lib.fvm_back_decoder(P(h), P(dout), N, O, P(sums[1]), s), "decoder")
    got = torch.zeros(O + 1, 64, device="cuda")
    n = O + 1
    _lib.check(lib.fvm_back_finish(n, (ct.c_void_p * n)(*[P(sums[1 + q]) for q in range(n)]),
                                   (ct.c_void_p * n)(*[P(got[q]) for q in range(n)]), (ct.c_int32 * n)(*([64] * O + [O])), s),
               "finish")
    want = torch.stack([(dout[:, o:o + 1].double() * h.double()).sum(0) for o in range(O)])
    assert not got.isnan().any()
    assert torch.equal(got[:O].isinf(), want.isinf())
    assert torch.equal(got[O, :O].isinf(), dout.sum(0).isinf())


def test_gradients_go_where_grads_points():
    """``train_step`` adds to the tensors that ``grads`` holds at the call, not to earlier ones.  The layers'
    gradients are added up by atomics in any order: 1e-4 of each."""
    from fvm_solver_b200.corrector import CorrectorNet
    N = 300
    net = CorrectorNet(3, layers=1, seed=1)
    net._alloc(N)["X"][:N].copy_(_rand(N, 64, seed=2))
    nbr, target = torch.full((N, 3), -1, dtype=torch.int32, device="cuda"), torch.zeros(N, 3, device="cuda")
    net.adam = lambda: None
    old = net.grads
    net.train_step(nbr, target)
    want = {k: v.clone() for k, v in old.items()}
    net.grads = {k: torch.zeros_like(v) for k, v in old.items()}
    net.train_step(nbr, target)
    for k, w in want.items():
        assert torch.equal(old[k], w), k
        assert torch.allclose(net.grads[k], w, rtol=1e-4, atol=1e-5 * float(w.abs().max())), k


def test_proposal_from_and_to_any_address(batch):
    """State, result and residual that start four bytes past a 16-byte boundary: bitwise as aligned ones."""
    def off(t):
        v = torch.empty(t.numel() + 4, device=t.device)[1:1 + t.numel()].view(t.shape)
        v.copy_(t)
        return v
    m, U, r0 = _model(batch)
    want = m.predict(U, torch.empty_like(U), r0).clone()
    for q in range(3):
        a = [U, torch.zeros_like(U), r0]
        a[q] = off(a[q])
        assert torch.equal(m.predict(*a), want)


@pytest.mark.parametrize("k", [np.int64(8), 8.0, np.float32(2.5)])
def test_window_length_of_any_number_type(batch, k):
    """``predict`` takes the window length as ``inputs`` does: base = float(k) dt r0."""
    m, U, r0 = _model(batch)
    m.k = k
    m.inputs(U, r0)
    base = m.base.clone()
    m.base.zero_()
    m.predict(U, torch.empty_like(U), r0)
    assert torch.equal(m.base, base)


@pytest.mark.parametrize("N", [128 * 148 * 4 - 1, 128 * 148 * 9 + 1, 1_000_003])
@pytest.mark.parametrize("layer", [True, False])
def test_weight_gradients_keep_their_accuracy(layer, N):
    """dW of one-signed terms against FP64, one to many chunks of rows per block.  A chunk is 512 rows: 32
    accumulations in the tensor core, each off by less than an ulp of the running sum in one direction, so
    at most 32 * 2^-23 = 3.8e-6 of a chunk and, with the rounded additions of the chunks, 4e-6 of the sum
    (a single accumulator for the block's rows is off by 2.5e-5 at 1 M rows)."""
    from fvm_solver_b200 import _lib
    lib, s = _lib.load(), _lib.stream_ptr()
    C = 128 if layer else 64
    err, P = torch.zeros(1, dtype=torch.int32, device="cuda"), lambda t: t.data_ptr()
    dZ, A = _rand(N, 64, seed=1).abs().bfloat16(), _rand(N, C, seed=2).abs().bfloat16()
    dW = torch.zeros(64, C, device="cuda")
    if layer:
        WT, nbr = torch.zeros(128, 64, device="cuda").bfloat16(), torch.full((N, 3), -1, dtype=torch.int32, device="cuda")
        dA = torch.empty(N, 128, device="cuda")
        rc = lib.fvm_back_layer(P(dZ), P(A), P(WT), P(nbr), 3, N, P(dA), P(dW), P(err), s)
    else:
        rc = lib.fvm_back_layer(P(dZ), P(A), None, None, 0, N, None, P(dW), P(err), s)
    want = sum(dZ[i:i + 400_000].double().t() @ A[i:i + 400_000].double() for i in range(0, N, 400_000))
    assert rc == 0 and int(err.item()) == 0
    assert float(((dW.double() - want).abs() / want).max()) < 4e-6
