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


# The scenes above have more pixels per vertex than copies are held for
# (kGradRowPixels), so their rows have one copy; the ones below are at its edge.
@pytest.mark.parametrize("kind", ["list", "abs", "banded", "cells", "raytet", "batch"])
@pytest.mark.parametrize("n,res", [(12, 187), (12, 189), (20, 384)])  # 15.9, 16.3 and 15.9 pixels per vertex
def test_gradients_at_the_edge_of_the_copies(oracle, kind, n, res):
    import difftetvr_b200 as d
    sc = Scene(n, res, seed=4)
    mesh, r = sc.make_renderer(d.RendererType.INTERSECTION if kind == "raytet" else None)
    if kind == "cells":
        mesh, col = cell_mesh(sc, sc.pos)
        r.set_tet_mesh(mesh)
    w = np.random.default_rng(5).normal(size=(res, res, 4)).astype(np.float32)
    gp, gc = gradients(kind, sc, mesh, r, torch.from_numpy(w).cuda())
    fa = oracle.Faces(sc.cells, sc.pos.shape[0])
    cam, prm = sc.oracle_camera(oracle), sc.oracle_params(oracle, use_abs_grad=kind == "abs")
    w64 = w.astype(np.float64)
    if kind == "cells":
        gp_o, gc_o = oracle.render_cells(fa, sc.pos, col, cam, prm, w64)[-2:]
    elif kind == "raytet":
        gp_o, gc_o = oracle.raytet(fa, sc.pos, sc.col, cam, prm, w64)[-2:]
    else:
        gp_o, gc_o = oracle.adjoint(fa, sc.pos, sc.col, cam, prm, w64)
    assert rel_err(gp.cpu().numpy(), gp_o) < GRAD_TOL
    assert rel_err(gc.cpu().numpy(), gc_o) < GRAD_TOL


def cell_mesh(sc, pos):
    import difftetvr_b200 as d
    col = sc.col[sc.cells.astype(np.int64)].mean(axis=1).astype(np.float32)
    mesh = d.TetMesh()
    mesh.set_use_gradients(True)
    mesh.set_tet_mesh_data_cell(sc.cells, pos, col)
    return mesh, col


def gradients(kind, sc, mesh, r, wt):
    pos = mesh.get_vertex_positions()
    c = mesh.get_cell_colors() if kind == "cells" else mesh.get_vertex_colors()
    gp, gc = torch.zeros_like(pos).detach(), torch.zeros_like(c).detach()
    if kind == "batch":
        from difftetvr_b200.batch import BatchRenderer, View
        br = BatchRenderer([mesh], attenuation=sc.attenuation, use_early_ray_termination=False)
        br.render([View(mesh=0, view_matrix=sc.view, width=sc.res, height=sc.res, fovy=sc.fovy, image_adjoint=wt,
                        grad_slot=0)])
        br.render_adjoint([(0, gp, gc)])
        return gp, gc
    r.render()
    if kind == "banded":
        r.set_fragment_budget_bytes(8 * (r.get_num_fragments() // 3))
        r.render()
        assert r.get_num_bands() > 1
    r.render_adjoint_into(wt, gp, gc, use_abs_grad=kind == "abs")
    return gp, gc


@pytest.mark.parametrize("kind", ["list", "abs", "banded", "cells", "raytet", "batch"])
def test_vertices_that_no_tet_has_leave_the_gradients_alone(kind):
    """A few hundred vertices under a megapixel: about 1e5 FP32 terms per row.
    However the rows are held, the number of vertices of the mesh must not move
    the gradients by more than another order of the additions does (a few 1e-6
    of the norm at 1e5 terms; bound 1e-5)."""
    import difftetvr_b200 as d
    sc = Scene(6, 1050, seed=11)
    # A smooth image adjoint, as a loss gives it: the terms add up instead of cancelling.
    yx = torch.stack(torch.meshgrid(torch.linspace(-1, 1, sc.res), torch.linspace(-1, 1, sc.res), indexing="ij"))
    wt = torch.exp(-2.0 * (yx ** 2).sum(0))[..., None].repeat(1, 1, 4).contiguous().cuda()
    extra = np.full((70000, 3), 0.25, np.float32)  # more rows than copies are held for
    got = []
    for pos in (sc.pos, np.concatenate([sc.pos, extra])):
        mesh, r = sc.make_renderer(d.RendererType.INTERSECTION if kind == "raytet" else None)
        if kind == "cells":
            mesh, _ = cell_mesh(sc, pos)
        else:
            mesh = d.TetMesh()
            mesh.set_use_gradients(True)
            mesh.set_tet_mesh_data(sc.cells, pos, np.concatenate([sc.col, np.ones((len(pos) - len(sc.pos), 4), np.float32)]))
        r.set_tet_mesh(mesh)
        gp, gc = gradients(kind, sc, mesh, r, wt)
        got.append((gp.cpu().numpy()[: len(sc.pos)], gc.cpu().numpy()[: len(sc.cells) if kind == "cells" else len(sc.pos)]))
    assert rel_err(got[0][0], got[1][0]) < 1e-5
    assert rel_err(got[0][1], got[1][1]) < 1e-5
