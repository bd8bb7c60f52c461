"""Adjoints of small meshes, whose gradient rows are held in several copies
(2, 32 and 64 here: by pixels and vertices), against the FP64 oracle (1e-4
relative, the bound of the paths' own parity tests)."""
import numpy as np
import pytest
import torch

from helpers import Scene, rel_err

pytestmark = pytest.mark.gpu

GRAD_TOL = 1e-4


@pytest.mark.parametrize("kind", ["list", "abs", "banded", "cells", "raytet", "batch"])
@pytest.mark.parametrize("res", [152, 520, 760])
def test_gradients_over_copies_match_fp64_oracle(oracle, kind, res):
    import difftetvr_b200 as d
    sc = Scene(3, res, seed=11)
    mesh, r = sc.make_renderer(d.RendererType.INTERSECTION if kind == "raytet" else None)
    col = sc.col
    if kind == "cells":
        col = sc.col[sc.cells.astype(np.int64)].mean(axis=1).astype(np.float32)
        mesh = d.TetMesh()
        mesh.set_use_gradients(True)
        mesh.set_tet_mesh_data_cell(sc.cells, sc.pos, col)
        r.set_tet_mesh(mesh)
    w = np.random.default_rng(5).normal(size=(res, res, 4)).astype(np.float32)
    wt = torch.from_numpy(w).cuda()
    pos = mesh.get_vertex_positions()
    c = mesh.get_cell_colors() if kind == "cells" else mesh.get_vertex_colors()
    gp, gc = torch.zeros_like(pos).detach(), torch.zeros_like(c).detach()
    if kind == "batch":
        from difftetvr_b200.batch import BatchRenderer, View
        br = BatchRenderer([mesh], attenuation=sc.attenuation, use_early_ray_termination=False)
        v = View(mesh=0, view_matrix=sc.view, width=res, height=res, fovy=sc.fovy, image_adjoint=wt, grad_slot=0)
        br.render([v])
        br.render_adjoint([(0, gp, gc)])
    else:
        r.render()
        if kind == "banded":
            r.set_fragment_budget_bytes(8 * (r.get_num_fragments() // 3))
            r.render()
            assert r.get_num_bands() > 1
        r.render_adjoint_into(wt, gp, gc, use_abs_grad=kind == "abs")
    fa = oracle.Faces(sc.cells, sc.pos.shape[0])
    cam, prm = sc.oracle_camera(oracle), sc.oracle_params(oracle, use_abs_grad=kind == "abs")
    w64 = w.astype(np.float64)
    if kind == "cells":
        gp_o, gc_o = oracle.render_cells(fa, sc.pos, col, cam, prm, w64)[-2:]
    elif kind == "raytet":
        gp_o, gc_o = oracle.raytet(fa, sc.pos, col, cam, prm, w64)[-2:]
    else:
        gp_o, gc_o = oracle.adjoint(fa, sc.pos, col, cam, prm, w64)
    assert rel_err(gp.cpu().numpy(), gp_o) < GRAD_TOL
    assert rel_err(gc.cpu().numpy(), gc_o) < GRAD_TOL
