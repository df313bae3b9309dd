"""The cost model's forward and gradient kernels at row counts where their split changes: below, at and one past a
CTA's tile of 40 rows, the last count that runs as one CTA and the first of two, an odd count whose last CTA holds
a few rows, and one with several tiles per CTA.  Against the float64 oracle, within the parity bar of the model's
gradients (1e-4 relative)."""
import ctypes

import numpy as np
import pytest

import __graft_entry__ as ge
from oracle import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 39, 40, 41, 75, 76, 301, 6400, 20001])
def test_forward_and_gradient(n):
    import torch
    ge.build()
    _, g = ge.package()
    g.init()
    rt = g.runtime()
    rt.dvmhgb_mlp_nparams.restype = ctypes.c_long
    rt.dvmhgb_mlp_work_floats.restype = ctypes.c_long
    P = rt.dvmhgb_mlp_nparams()
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    p = torch.empty(P, dtype=torch.float32, device="cuda")
    assert rt.dvmhgb_mlp_init(vp(p), ctypes.c_ulonglong(n), None) == 0
    rng = np.random.default_rng(n)
    X = torch.tensor(rng.standard_normal((n, 24)), dtype=torch.float32, device="cuda")
    y = torch.tensor(rng.standard_normal(n), dtype=torch.float32, device="cuda")
    grad = torch.full((P + 1,), 7.0, dtype=torch.float32, device="cuda")
    pred = torch.full((n + 1,), 7.0, dtype=torch.float32, device="cuda")
    loss = torch.empty(1, dtype=torch.float32, device="cuda")
    words = rt.dvmhgb_mlp_work_floats(ctypes.c_long(n))
    work = torch.full((words + 1,), 7.0, dtype=torch.float32, device="cuda")
    assert rt.dvmhgb_mlp_forward(vp(p), vp(X), ctypes.c_long(n), vp(pred), vp(work), None) == 0
    assert rt.dvmhgb_mlp_loss_grad(vp(p), vp(X), vp(y), ctypes.c_long(n), vp(grad), vp(loss), vp(work), None) == 0
    again = torch.empty_like(grad)
    assert rt.dvmhgb_mlp_loss_grad(vp(p), vp(X), vp(y), ctypes.c_long(n), vp(again), None, vp(work), None) == 0
    torch.cuda.synchronize()
    assert grad[P].item() == 7.0 and pred[n].item() == 7.0 and work[words].item() == 7.0  # nothing past the ends
    assert torch.equal(grad[:P], again[:P])  # the same every time, with or without the loss
    ph = p.cpu().numpy().astype(np.float64)
    ref_pred, _ = mlp_ref.forward(ph, X.cpu().numpy())
    ref_loss, ref_g = mlp_ref.loss_grad(ph, X.cpu().numpy(), y.cpu().numpy())
    got = grad[:P].cpu().numpy()
    assert np.linalg.norm(pred[:n].cpu().numpy() - ref_pred) <= 1e-4 * np.linalg.norm(ref_pred)
    assert abs(loss.item() - ref_loss) <= 1e-4 * abs(ref_loss)
    assert np.linalg.norm(got - ref_g) <= 1e-4 * np.linalg.norm(ref_g)
