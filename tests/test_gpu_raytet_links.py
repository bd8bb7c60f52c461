"""The intersection renderer's walk on the mesh's links against its walk by
face search.  A mesh takes the search when most of its faces are boundary
faces, so 2,000 loose tets behind the camera send the same scene there: segment
counts are equal, images within 1e-5 (of max(1, |value|)) and gradients within
1e-4 relative, the path's own bounds."""
import numpy as np
import pytest
import torch

from helpers import Scene, rel_err, two_block_scene

pytestmark = pytest.mark.gpu

IMG_TOL = 1e-5
GRAD_TOL = 1e-4


def scene(kind: str) -> Scene:
    from difftetvr_b200 import synthetic as S
    if kind == "two_blocks":      # two intervals per ray
        return two_block_scene(4, 93, seed=3)
    sc = Scene(6, 93, seed=7, jitter=0.9 if kind == "inverted" else 0.2)
    if kind == "near":            # wide view from just outside: vertices behind the camera
        sc.view, sc.fovy = S.look_at_view([0.55, 0.02, 1.2]), 2.4
    elif kind == "far":           # vertices up to 180,000 px off screen
        sc.fovy = 5e-4
    elif kind == "orders":        # every tet's vertices in another order, a third of them mirrored
        rng = np.random.default_rng(4)
        even = [(0, 1, 2, 3), (1, 2, 0, 3), (3, 2, 1, 0), (2, 3, 0, 1)]
        perm = np.array([even[k] for k in rng.integers(0, 4, len(sc.cells))])
        sc.cells = np.take_along_axis(sc.cells, perm, axis=1)
        sc.cells[::3, [1, 2]] = sc.cells[::3, [2, 1]]
    elif kind == "ended":         # rays end inside the mesh
        sc.attenuation, sc.ert = 30.0, True
    return sc


def with_loose_tets(sc: Scene, count: int = 2000):
    eye = np.linalg.inv(np.asarray(sc.view, np.float64).reshape(4, 4))[3, :3]  # column-major view matrix
    rng = np.random.default_rng(8)
    p = eye + 8.0 * eye / np.linalg.norm(eye) + rng.uniform(-0.5, 0.5, (4 * count, 3))
    v = len(sc.pos)
    sc.cells = np.concatenate([sc.cells, v + np.arange(4 * count, dtype=np.uint32).reshape(-1, 4)]).astype(np.uint32)
    sc.pos = np.concatenate([sc.pos, p.astype(np.float32)])
    sc.col = np.concatenate([sc.col, np.zeros((4 * count, 4), np.float32)])


@pytest.mark.parametrize("kind", ["cube", "two_blocks", "inverted", "near", "far", "orders", "ended"])
def test_linked_walk_equals_the_search(kind):
    import difftetvr_b200 as d
    out = []
    verts = len(scene(kind).pos)
    for loose in (False, True):
        sc = scene(kind)
        if loose:
            with_loose_tets(sc)
        mesh, r = sc.make_renderer(d.RendererType.INTERSECTION)
        img = r.render().cpu().numpy().astype(np.float64)
        _, nseg = r.get_pixel_state()
        w = torch.from_numpy(np.random.default_rng(6).normal(size=(sc.res, sc.res, 4)).astype(np.float32)).cuda()
        gp = torch.zeros_like(mesh.get_vertex_positions()).detach()
        gc = torch.zeros_like(mesh.get_vertex_colors()).detach()
        r.render_adjoint_into(w, gp, gc)
        out.append((img, np.asarray(nseg), gp.cpu().numpy(), gc.cpu().numpy()))
    (img, nseg, gp, gc), (img_s, nseg_s, gp_s, gc_s) = out
    assert (nseg_s > 0).sum() > 0.1 * nseg_s.size
    assert np.array_equal(nseg, nseg_s)
    assert (np.abs(img - img_s) / np.maximum(1.0, np.abs(img_s))).max() < IMG_TOL
    assert rel_err(gp, gp_s[:verts]) < GRAD_TOL and rel_err(gc, gc_s[:verts]) < GRAD_TOL
    assert not gp_s[verts:].any() and not gc_s[verts:].any()
