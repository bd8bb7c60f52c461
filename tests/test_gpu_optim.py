"""Loss and Adam kernels vs torch (B200)."""
import ctypes

import numpy as np
import pytest
import torch

from difftetvr_b200 import _lib

pytestmark = pytest.mark.gpu


def test_l2_loss_kernel_matches_torch():
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.rand(64, 48, 4, device="cuda", generator=g)
    y = torch.rand(64, 48, 4, device="cuda", generator=g)
    adj = torch.empty_like(x)
    loss = torch.zeros(1, device="cuda")
    n = x.numel()
    _lib.call("dtv_loss_l2", x.data_ptr(), y.data_ptr(), n, 1.0 / n, adj.data_ptr(), loss.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
    xr = x.clone().requires_grad_(True)
    ref = torch.nn.functional.mse_loss(xr, y)
    ref.backward()
    assert torch.allclose(loss[0], ref, rtol=1e-5)
    assert torch.allclose(adj, xr.grad, rtol=1e-5, atol=1e-9)


@pytest.mark.parametrize("clamp", [0, 1])
def test_adam_kernel_matches_torch_adam(clamp):
    g = torch.Generator(device="cuda").manual_seed(1)
    p0 = torch.randn(3000, device="cuda", generator=g)
    p_ref = p0.clone().requires_grad_(True)
    opt = torch.optim.Adam([p_ref], lr=1e-2, betas=(0.9, 0.999), eps=1e-8)
    p = p0.clone()
    m = torch.zeros_like(p)
    v = torch.zeros_like(p)
    for step in range(1, 6):
        grad = torch.randn(3000, device="cuda", generator=g)
        p_ref.grad = grad.clone()
        opt.step()
        if clamp == 1:
            with torch.no_grad():
                p_ref -= torch.min(p_ref, torch.zeros_like(p_ref))
        _lib.call("dtv_adam_step", p.data_ptr(), grad.data_ptr(), m.data_ptr(), v.data_ptr(), p.numel(),
                  ctypes.c_float(1e-2), ctypes.c_float(0.9), ctypes.c_float(0.999), ctypes.c_float(1e-8), step,
                  clamp, None, 0, 1, torch.cuda.current_stream().cuda_stream)
    assert torch.allclose(p, p_ref.detach(), rtol=1e-5, atol=1e-6)


def test_adam_fixed_mask_modes():
    p = torch.ones(12, device="cuda")
    grad = torch.ones(12, device="cuda")
    mask = torch.tensor([1, 0, 0, 1], dtype=torch.int32, device="cuda")  # per vertex (stride 3)
    for mode in (1, 2):
        q = p.clone()
        m = torch.zeros_like(q)
        v = torch.zeros_like(q)
        _lib.call("dtv_adam_step", q.data_ptr(), grad.data_ptr(), m.data_ptr(), v.data_ptr(), 12,
                  ctypes.c_float(0.1), ctypes.c_float(0.9), ctypes.c_float(0.999), ctypes.c_float(1e-8), 1, 0,
                  mask.data_ptr(), mode, 3, torch.cuda.current_stream().cuda_stream)
        fixed = mask.repeat_interleave(3).bool()
        assert torch.all(q[fixed] == 1.0)
        assert torch.all(q[~fixed] < 1.0)
        if mode == 2:
            assert torch.all(m[fixed] == 0)


@pytest.mark.parametrize("n", [4096, 4099])   # four at a time, with a remainder
@pytest.mark.parametrize("value,want", [(3e19, float("inf")), (float("inf"), float("inf")), (float("nan"), float("nan"))])
def test_loss_of_values_beyond_fp32(n, value, want):
    """A square that overflows, an infinity and a NaN give what FP32 sums give."""
    from difftetvr_b200.optim import l2_loss
    x = torch.zeros(n, device="cuda")
    x[n // 3] = value
    loss = float(l2_loss(x, torch.zeros_like(x)))
    assert (np.isnan(want) and np.isnan(loss)) or loss == want


@pytest.mark.parametrize("value,want", [(3e19, float("inf")), (float("inf"), float("inf")), (float("nan"), float("nan"))])
def test_batch_loss_of_values_beyond_fp32(value, want):
    from difftetvr_b200.batch import BatchRenderer, View
    from helpers import Scene
    sc = Scene(3, 48)
    mesh, _ = sc.make_renderer()
    target = torch.zeros((48, 48, 4), device="cuda")
    target[7, 5, 1] = value
    br = BatchRenderer([mesh])
    loss = float(br.train_step([View(mesh=0, view_matrix=sc.view, width=48, height=48, fovy=sc.fovy, target=target)]))
    assert (np.isnan(want) and np.isnan(loss)) or loss == want


@pytest.mark.parametrize("n", [1, 151552, 3 * 151552, 4 * 151552, 4 * 151552 + 5])   # around whole passes of the grid
@pytest.mark.parametrize("shift", [0, 1])                                           # 16- and 4-byte aligned
def test_l2_loss_lengths_and_alignments(n, shift):
    """Loss within the rounding of 296 FP32 additions of carried sums (1e-5);
    at this scale the adjoint is the difference itself."""
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.rand(n + 1, device="cuda", generator=g)[shift:shift + n]
    y = torch.rand(n + 1, device="cuda", generator=g)[shift:shift + n]
    adj = torch.empty(n + 1, device="cuda")[shift:shift + n]
    loss = torch.zeros(1, device="cuda")
    _lib.call("dtv_loss_l2", x.data_ptr(), y.data_ptr(), n, 0.5, adj.data_ptr(), loss.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
    d = x.double() - y.double()
    assert abs(float(loss) - 0.5 * float((d * d).sum())) <= 1e-5 * 0.5 * float((d * d).sum())
    assert torch.equal(adj, x - y)
