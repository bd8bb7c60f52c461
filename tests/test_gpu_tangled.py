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


def test_lists_of_tangled_and_plain_meshes_in_turn_at_two_sizes(oracle):
    """What one render left decides on others: of another mesh, at another size."""
    made = []
    for jitter in (3.0, 0.2):
        sc = Scene(7, 101, seed=12, jitter=jitter)
        made.append((sc, sc.make_renderer()[0], oracle.Faces(sc.cells, sc.pos.shape[0])))
    r = made[0][0].make_renderer()[1]
    for k, res in [(0, 101), (0, 33), (1, 33), (1, 101), (0, 101), (0, 101), (0, 33), (0, 33), (1, 101)]:
        sc, mesh, fa = made[k]
        sc.res = res
        r.set_tet_mesh(mesh)
        r.set_viewport_size(res, res)
        r.render()
        off, rec = r.get_fragment_lists()
        off_o, rec_o = oracle.fragments(fa, sc.pos, sc.oracle_camera(oracle))
        assert np.array_equal(off.astype(np.int64), off_o.astype(np.int64)) and np.array_equal(rec, rec_o)


def test_batches_of_tangled_and_plain_meshes_in_turn():
    from difftetvr_b200.batch import BatchRenderer, View
    scs = [Scene(7, 101, seed=12, jitter=j) for j in (3.0, 0.2)]
    made = [sc.make_renderer() for sc in scs]
    imgs = [r.render().clone() for _, r in made]
    br = BatchRenderer([m for m, _ in made], attenuation=scs[0].attenuation, use_early_ray_termination=False)
    for idx in [(0, 0), (1, 1), (0, 1), (1, 1), (0,), (1,), (0, 0)]:
        views = [View(mesh=i, view_matrix=scs[i].view, width=101, height=101, fovy=scs[i].fovy) for i in idx]
        for i, out in zip(idx, br.render(views)):
            assert float((out - imgs[i]).abs().max()) <= 1e-6


def test_a_mesh_that_is_not_walked_holds_no_walk_tables():
    """Unconnected tets: device memory for faces, tets and boundary faces alone
    (225 bytes per tet; the walk's tables would be 128 more)."""
    from difftetvr_b200.tet_mesh import NativeMesh
    T = 300_000
    cells = np.arange(4 * T, dtype=np.uint32).reshape(-1, 4)
    NativeMesh(cells[:100], 400)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    mesh = NativeMesh(cells, 4 * T)
    used = free - torch.cuda.mem_get_info()[0]
    assert mesh.num_faces == 4 * T
    # face rows 64, face tets 32, boundary flags 16, tets 32 + 1, boundary faces 64 + 16, 225 in all; each
    # allocation in whole 2 MiB pages
    assert used <= 225 * T + 8 * (2 << 20)
