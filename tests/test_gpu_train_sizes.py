"""The trainer's gradients at the edges of its tiles (32 samples per CTA, 64
per cluster, clusters that take several tiles) against 64-bit autograd: after
one step from zero moments, m is a tenth of the mean gradient. Tolerance: the
sums are FP32 products accumulated in at most a few hundred terms in a row, so
the relative L2 error stays well below 1e-5."""
import ctypes as C

import numpy as np
import pytest

from dynamicradiancevolume_gb300 import abi, surrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 64, 65, 1000, 4864, 4865, 12345])
def test_gradients_match_fp64(n, lib, cuda):
    torch = pytest.importorskip("torch")
    g = torch.Generator().manual_seed(n)
    X = torch.rand((n, abi.SURROGATE_INPUTS), generator=g)
    X[:, 31] = 1.0
    Y = torch.rand((n,), generator=g)
    p0 = torch.from_numpy(surrogate.init_params(3))
    x, y, params = X.cuda(), Y.cuda(), p0.cuda()
    m, v, loss = torch.zeros_like(params), torch.zeros_like(params), torch.zeros(2, device="cuda")
    scratch = torch.empty(lib.drv_surrogate_train_scratch_floats(n), device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    tau = 0.03
    assert lib.drv_surrogate_train_step(ptr(x), ptr(y), n, ptr(params), ptr(m), ptr(v), ptr(scratch), 1, 1e-3, tau,
                                        0.0, ptr(loss), None) == abi.OK
    torch.cuda.synchronize()
    P = p0.double().requires_grad_(True)
    a, o = X.double(), 0
    for k, (rows, cols) in enumerate(((64, 32), (64, 64), (64, 64), (2, 64))):
        z = a @ P[o:o + rows * cols].view(rows, cols).T + P[o + rows * cols:o + rows * cols + rows]
        a = z * torch.sigmoid(1.702 * z) if k < 3 else z
        o += rows * cols + rows
    vis, conf = torch.sigmoid(a[:, 0]), torch.sigmoid(a[:, 1])
    near = (vis - Y.double()).abs().detach()
    assert float((near - tau).abs().min()) > 1e-6  # no confidence target within rounding of its threshold
    bce = lambda q, t: torch.nn.functional.binary_cross_entropy(q, t, reduction="sum")
    l0, l1 = bce(vis, Y.double()), bce(conf, (near < tau).double())
    ((l0 + l1) / n).backward()
    rel = lambda q, r: float((q.double().cpu() - r).norm() / r.norm())
    assert rel(m, 0.1 * P.grad) < 1e-5
    assert rel(loss, torch.stack([l0, l1]).detach()) < 1e-5
    assert np.isfinite(params.cpu().numpy()).all()
