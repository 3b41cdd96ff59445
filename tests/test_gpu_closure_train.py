"""The closure network's training step as one call, and the GEMM's vector and scalar epilogues.

Tolerances: the passes and the step differ from the separate calls only in the order of float32
sums over at most 4,096 rows (relative error at most sqrt(4096) * 6e-8 = 4e-6 in the typical
sense, 2e-5 with a margin of five); Adam divides by the gradient's own size, so parameters are
compared relative to their norm."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from fsi import _native as nat
from fsi import closure as cl
from helpers import rel_l2

pytestmark = pytest.mark.gpu


def _data(rows, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((rows, cl.FEATURES), generator=g, device="cuda")
    x[:, cl._ZERO_COLS] = 0.0
    t = torch.randn((rows, cl.OUT), generator=g, device="cuda")
    return x.to(torch.bfloat16), t


@pytest.mark.parametrize("rows,batch", [(100, 128), (500, 384), (5000, 4096)])
def test_fit_is_forward_backward_adam(rows, batch):
    x, t = _data(rows, batch)
    one, many = cl.ClosureMLP(seed=3), cl.ClosureMLP(seed=3)
    tr = cl.ClosureTrainer(one)
    tr.x, tr.t = x, t
    steps, lr = 3, 1e-3
    hist = tr.fit(steps=steps, batch=batch, lr=lr, seed=7)
    g = torch.Generator(device="cpu").manual_seed(7)
    m = max(128, min(batch, rows) // 128 * 128)
    want = []
    for it in range(steps):
        idx = torch.randint(0, rows, (m,), generator=g).cuda()
        xb = x[idx].contiguous()
        y, acts = many.forward(xb, keep=True)
        want.append(many.backward(xb, y, acts, t[idx].contiguous(), xt=xb.t().contiguous()))
        many.adam_step(lr=lr * 0.5 ** (it / steps * 3.0))
    np.testing.assert_allclose(hist, want, rtol=2e-5)
    for a, b in zip(one.gviews, many.gviews):
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 1e-3  # third step: weights differ a little
    assert rel_l2(one.params.cpu().numpy(), many.params.cpu().numpy()) < 1e-4
    assert one.step_count == many.step_count == steps
    bf = torch.bfloat16
    W1, b1, W2, b2, W3, b3, W4, b4 = one.views
    for got, ref in ((one.w1, W1), (one.w2, W2), (one.w3, W3), (one.w4, W4), (one.w2t, W2.t()),
                     (one.w3t, W3.t()), (one.w4t, W4.t())):
        assert torch.equal(got, ref.to(bf))
    assert torch.equal(one.bias, torch.cat([b1, b2, b3, b4]))


def test_first_step_gradients():
    x, t = _data(4096, 1)
    net = cl.ClosureMLP(seed=4)
    ref = cl.ClosureMLP(seed=4)
    tr = cl.ClosureTrainer(net)
    tr.x, tr.t = x, t
    tr.fit(steps=1, batch=4096, lr=1e-3, seed=1)
    idx = torch.randint(0, 4096, (4096,), generator=torch.Generator().manual_seed(1)).cuda()
    xb = x[idx].contiguous()
    y, acts = ref.forward(xb, keep=True)
    ref.backward(xb, y, acts, t[idx].contiguous(), xt=xb.t().contiguous())
    for a, b in zip(net.gviews, ref.gviews):
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 2e-5


def test_train_step_arguments():
    lib = nat.load()
    assert lib.fsi_closure_train_bytes(128) > 0
    for m in (0, -128, 100):
        assert lib.fsi_closure_train_bytes(m) == -1
    with pytest.raises(ValueError, match="NULL"):
        nat.call("fsi_closure_train_step", nat.ClosureTrainDesc(), nat.stream_ptr())


@pytest.mark.parametrize("n", [16, 19, 24, 64, 100, 128, 144])
@pytest.mark.parametrize("m,k", [(1, 8), (130, 200), (256, 656)])
def test_gemm_epilogues_for_whole_and_ragged_columns(m, n, k):
    rng = np.random.default_rng(m + n + k)
    a = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).cuda().to(torch.bfloat16)
    b = torch.from_numpy(rng.standard_normal((n, k)).astype(np.float32)).cuda().to(torch.bfloat16)
    bias = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    acc = a.double() @ b.double().T
    tol = 1e-4 * float(np.sqrt(k))
    for ld in (n, n + 3):  # rows of C at 16-byte boundaries or not
        c = torch.full((m, ld), 0.5, device="cuda")
        cl._gemm(a, b, k, k, m, n, k, nat.GEMM_STORE, err, c=c, ldc=ld)
        assert float((c[:, :n] - acc).abs().max()) < tol
        assert bool((c[:, n:] == 0.5).all())
        cl._gemm(a, b, k, k, m, n, k, nat.GEMM_ATOMIC, err, c=c, ldc=ld, k_chunk=64)
        assert float((c[:, :n] - 2 * acc).abs().max()) < 2 * tol
    z = torch.zeros((m, n), device="cuda")
    h = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
    ht = torch.zeros((n, m), dtype=torch.bfloat16, device="cuda")
    cl._gemm(a, b, k, k, m, n, k, nat.GEMM_GELU_FWD, err, bias=bias, h=h, ht=ht, ldht=m, zout=z)
    want = torch.nn.functional.gelu(acc + bias, approximate="tanh")
    assert float((z - acc - bias).abs().max()) < tol
    assert float((h.double() - want).abs().max()) < tol + 2e-2 * float(want.abs().max())
    assert torch.equal(ht, h.T)
    cl._gemm(a, b, k, k, m, n, k, nat.GEMM_GELU_BWD, err, h=h, ht=ht, ldht=m, zin=z)
    zz = z.double().requires_grad_(True)
    slope, = torch.autograd.grad(torch.nn.functional.gelu(zz, approximate="tanh").sum(), zz)
    want = acc * slope
    assert float((h.double() - want).abs().max()) < tol + 2e-2 * float(want.abs().max())
    assert torch.equal(ht, h.T)
    assert int(err.item()) == 0
