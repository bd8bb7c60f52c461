"""Meshes whose tets overlap, so that closed loops of faces cover many pixels:
the first render's walk leaves them to the rasteriser, later ones do not walk
(and a mesh with few such pixels keeps walking, with the faces that miss them
skipped).  Lists bit-exact against the CPU oracle in every render; images and
gradients the same from render to render (gradients: atomic sums in another
order, 1e-5)."""
import numpy as np
import pytest
import torch

from helpers import Scene, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jitter", [0.9, 3.0])
@pytest.mark.parametrize("bands", [False, True])
def test_lists_of_tangled_meshes_in_every_render(oracle, jitter, bands):
    sc = Scene(7, 101, seed=12, jitter=jitter)
    mesh, r = sc.make_renderer()
    fa = oracle.Faces(sc.cells, sc.pos.shape[0])
    off_o, rec_o = oracle.fragments(fa, sc.pos, sc.oracle_camera(oracle))
    w = torch.from_numpy(np.random.default_rng(2).normal(size=(101, 101, 4)).astype(np.float32)).cuda()
    if bands:
        r.set_fragment_budget_bytes(8 * (len(rec_o) // 3))
    first = None
    for _ in range(4):
        img = r.render().clone()
        if not bands:
            off, rec = r.get_fragment_lists()
            assert np.array_equal(off.astype(np.int64), off_o.astype(np.int64)) and np.array_equal(rec, rec_o)
        gp, gc = torch.zeros_like(mesh.get_vertex_positions()).detach(), torch.zeros_like(mesh.get_vertex_colors()).detach()
        r.render_adjoint_into(w, gp, gc)
        torch.cuda.synchronize()
        if first is None:
            first = (img, gp, gc)
        assert torch.equal(img, first[0])
        assert rel_err(gp.cpu().numpy(), first[1].cpu().numpy()) < 1e-5
        assert rel_err(gc.cpu().numpy(), first[2].cpu().numpy()) < 1e-5


@pytest.mark.parametrize("jitter", [0.9, 3.0])
def test_batches_of_tangled_meshes(jitter):
    from difftetvr_b200.batch import BatchRenderer, View
    sc = Scene(7, 101, seed=12, jitter=jitter)
    mesh, r = sc.make_renderer()
    img = r.render().clone()
    br = BatchRenderer([mesh], attenuation=sc.attenuation, use_early_ray_termination=False)
    views = [View(mesh=0, view_matrix=sc.view, width=101, height=101, fovy=sc.fovy) for _ in range(3)]
    for _ in range(4):
        for out in br.render(views):
            assert float((out - img).abs().max()) <= 1e-6
