"""Regularizer gradient over runs of consecutive tets (1, 2 and 6 per thread:
by the tet count) in meshes whose consecutive tets share vertices, share none,
or hold one vertex twice, with 4- and 8-byte aligned gradients, against FP64
torch.  Bound: a vertex gradient is a sum of at most a few dozen FP32 terms of
like magnitude, each from about a hundred roundings: 1e-5 of the norm."""
import numpy as np
import pytest
import torch

from helpers import rel_err

pytestmark = pytest.mark.gpu


def reference(cells, pos, lam, beta):
    p = torch.tensor(pos, dtype=torch.float64, requires_grad=True)
    v = p[torch.as_tensor(cells.astype(np.int64))]
    det = (torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]) * (v[:, 3] - v[:, 0])).sum(1)
    s = sum(((v[:, i] - v[:, j]) ** 2).sum(1) for i in range(4) for j in range(i))
    q = -12.0 * np.sqrt(3.0) * det / s ** 1.5
    loss = (lam / beta * torch.nn.functional.softplus(-beta * q, threshold=1e9)).sum()
    loss.backward()
    return p.grad.numpy(), float(loss)


@pytest.mark.parametrize("n,order", [(3, "grid"), (30, "grid"), (38, "grid"), (55, "grid"), (55, "shuffled"),
                                     (38, "repeated")])
def test_gradient_and_loss(n, order):
    import difftetvr_b200 as d
    from difftetvr_b200 import synthetic as S
    from difftetvr_b200.regularizer import TetRegularizer
    # Cells of side 1, so the denominator's clamp is never active.
    cells, pos = S.kuhn_mesh(n, seed=n, lo=0.0, hi=float(n))
    if order == "shuffled":
        cells = cells[np.random.default_rng(1).permutation(len(cells))]
    elif order == "repeated":
        cells[7::50, 3] = cells[7::50, 0]
    cells = cells[: len(cells) - 5]  # the last thread's run is short
    mesh = d.TetMesh()
    mesh.set_use_gradients(True)
    mesh.set_tet_mesh_data(cells, pos, S.gaussian_colors(pos, seed=1))
    reg = TetRegularizer(mesh, 0.1, 2.0)
    g_ref, l_ref = reference(cells, pos, np.float64(np.float32(0.1)), 2.0)
    V = pos.shape[0]
    for shift in (0, 1):  # base 16- and 4-byte aligned
        g = torch.zeros(3 * V + 1, device="cuda")[shift:shift + 3 * V].view(V, 3)
        loss = reg.compute_grad_into(g)
        assert rel_err(g.cpu().numpy(), g_ref) < 1e-5
        assert abs(float(loss) - l_ref) < 1e-5 * abs(l_ref)


@pytest.mark.parametrize("n", [38, 55])   # runs of 2 and of 6 tets
@pytest.mark.parametrize("pair", [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)])
def test_repeated_vertices_anywhere_in_a_run(n, pair):
    """Tets with the same vertex at two corners, at every position of a run and
    followed by the grid's tets, which share the vertex and bring new ones; the
    sums of test_gradient_and_loss, so its bound."""
    import difftetvr_b200 as d
    from difftetvr_b200 import synthetic as S
    from difftetvr_b200.regularizer import TetRegularizer
    cells, pos = S.kuhn_mesh(n, seed=n, lo=0.0, hi=float(n))
    for k in range(6):
        cells[6 * k + k::90, pair[1]] = cells[6 * k + k::90, pair[0]]
    mesh = d.TetMesh()
    mesh.set_use_gradients(True)
    mesh.set_tet_mesh_data(cells, pos, S.gaussian_colors(pos, seed=1))
    g_ref, l_ref = reference(cells, pos, np.float64(np.float32(0.1)), 2.0)
    g = torch.zeros(pos.shape, device="cuda")
    loss = TetRegularizer(mesh, 0.1, 2.0).compute_grad_into(g)
    assert rel_err(g.cpu().numpy(), g_ref) < 1e-5
    assert abs(float(loss) - l_ref) < 1e-5 * abs(l_ref)
