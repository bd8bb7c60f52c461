"""Fragment lists built by walking the mesh, where the walk ends early or does
not apply: pixels whose faces are cut by the near plane, inverted tets, tets
that share no face structure a walk could follow, more chains than a pixel's
table holds, vertices far off screen.  Lists bit-exact against the CPU oracle;
images within the FP32-vs-FP64 bound of the list path (1e-5) where every
fragment is well conditioned."""
import numpy as np
import pytest
import torch

from helpers import Scene

pytestmark = pytest.mark.gpu

IMG_TOL = 1e-5


def slabs(count: int, res: int) -> Scene:
    """`count` separate one-cell-thick slabs along the view axis: as many
    chains per pixel."""
    from difftetvr_b200 import synthetic as S
    sc = Scene(1, res, seed=5)
    cells, pos = [], []
    for k in range(count):
        c, p = S.kuhn_mesh(1, seed=k, lo=-0.5, hi=0.5)
        p[:, 2] = p[:, 2] * 0.1 + (0.2 * k - 0.1 * count)
        cells.append(c + np.uint32(8 * k))
        pos.append(p)
    sc.cells, sc.pos = np.concatenate(cells).astype(np.uint32), np.concatenate(pos).astype(np.float32)
    sc.col = S.gaussian_colors(sc.pos, seed=2)
    sc.view = S.look_at_view([0.11, 0.07, 4.0])
    return sc


def scene(kind: str) -> Scene:
    from difftetvr_b200 import synthetic as S
    if kind.startswith("slabs"):
        return slabs(int(kind[5:]), 61)
    sc = Scene(6, 93, seed=7)
    if kind == "near":            # camera inside the mesh: rays start behind cut-away faces
        sc.view = S.look_at_view([0.31, 0.22, 0.43])
    elif kind == "inverted":
        sc = Scene(6, 93, seed=7, jitter=0.9)
    elif kind == "shared3":       # a third tet on an interior face
        apex = np.array([[0.05, 0.02, 0.9]], np.float32)
        sc.pos = np.concatenate([sc.pos, apex])
        sc.col = np.concatenate([sc.col, sc.col[:1]])
        inner = sc.cells[len(sc.cells) // 2]
        extra = np.array([[inner[0], inner[1], inner[2], len(sc.pos) - 1]], np.uint32)
        sc.cells = np.concatenate([sc.cells, extra])
    elif kind == "repeated":      # a tet with one vertex twice
        c = sc.cells[len(sc.cells) // 2].copy()
        c[3] = c[0]
        sc.cells = np.concatenate([sc.cells, c[None]])
    elif kind == "far":           # one corner 185,000 px off screen
        sc = Scene(2, 93, seed=3)
        sc.view = S.look_at_view([0.0, 0.001, 3.0])
        sc.pos[0] = (-160.0, -120.0, 2.9)
    return sc


KINDS = ["near", "inverted", "shared3", "repeated", "far", "slabs3", "slabs8", "slabs9"]


@pytest.mark.parametrize("kind", KINDS)
def test_lists_bit_exact(oracle, kind):
    sc = scene(kind)
    mesh, r = sc.make_renderer()
    fa = oracle.Faces(sc.cells, sc.pos.shape[0])
    off_o, rec_o = oracle.fragments(fa, sc.pos, sc.oracle_camera(oracle))
    assert rec_o.size > 0
    for _ in range(2):  # the first render sizes the record buffer, the second finds it
        img = r.render()
        off_g, rec_g = r.get_fragment_lists()
        assert np.array_equal(off_g.astype(np.int64), off_o) and np.array_equal(rec_g, rec_o)
    if kind.startswith("slabs"):
        ref = oracle.render(fa, sc.pos, sc.col, sc.oracle_camera(oracle), sc.oracle_params(oracle))[0]
        assert np.abs(img.cpu().numpy() - ref).max() <= IMG_TOL


@pytest.mark.parametrize("kind", ["near", "inverted", "slabs9"])
def test_per_cell_and_banded_lists(oracle, kind):
    """The same left-over pixels with per-cell colours (image against the
    oracle's bound of that path) and in row bands (bit-identical image)."""
    import difftetvr_b200 as d
    sc = scene(kind)
    mesh, r = sc.make_renderer()
    whole = r.render().clone()
    nf = r.get_num_fragments()
    r.set_fragment_budget_bytes(8 * (nf // 2))
    assert torch.equal(r.render(), whole) and r.get_num_bands() > 1
    cc = sc.col[sc.cells.astype(np.int64)].mean(axis=1).astype(np.float32)
    cm = d.TetMesh()
    cm.set_use_gradients(True)
    cm.set_tet_mesh_data_cell(sc.cells, sc.pos, cc)
    rc = sc.make_renderer()[1]
    rc.set_tet_mesh(cm)
    rc.render()
    fa = oracle.Faces(sc.cells, sc.pos.shape[0])
    off_o, rec_o = oracle.fragments(fa, sc.pos, sc.oracle_camera(oracle))
    off_g, rec_g = rc.get_fragment_lists()
    assert np.array_equal(off_g.astype(np.int64), off_o) and np.array_equal(rec_g, rec_o)


@pytest.mark.parametrize("kinds", [("near", "slabs9"), ("far", "shared3")])
def test_batch_matches_plain_views(kinds):
    """Views that leave pixels to the rasteriser, and a batch with a mesh that
    cannot be walked, against one view per launch."""
    from difftetvr_b200.batch import BatchRenderer, View
    scs = [scene(k) for k in kinds]
    made = [sc.make_renderer() for sc in scs]
    br = BatchRenderer([m for m, _ in made], attenuation=1.0, use_early_ray_termination=False)
    views = [View(mesh=i, view_matrix=sc.view, width=sc.res, height=sc.res, fovy=sc.fovy)
             for i, sc in enumerate(scs)]
    for img, (_, r) in zip(br.render(views), made):
        assert float((img - r.render()).abs().max()) <= 1e-6


NEAR, WHOLE, FAR_OFF = [0.31, 0.22, 0.43], [1.6, 1.1, 2.3], [0.1, 0.2, 1.02]


def test_lists_of_clipped_and_whole_views_in_turn(oracle):
    """Views with and without clipped vertices from one renderer, in every
    order of two; small and large ones (the record buffer grows in between)."""
    from difftetvr_b200 import synthetic as S
    sc = Scene(6, 93, seed=7)
    mesh, r = sc.make_renderer()
    fa = oracle.Faces(sc.cells, sc.pos.shape[0])
    for at, res in [(WHOLE, 40), (NEAR, 93), (NEAR, 40), (WHOLE, 93), (WHOLE, 93), (FAR_OFF, 93), (WHOLE, 150),
                    (NEAR, 150), (WHOLE, 40)]:
        sc.view, sc.res = S.look_at_view(at), res
        off_o, rec_o = oracle.fragments(fa, sc.pos, sc.oracle_camera(oracle))
        r.set_view_matrix(sc.view)
        r.set_viewport_size(res, res)
        r.render()
        off_g, rec_g = r.get_fragment_lists()
        assert np.array_equal(off_g.astype(np.int64), off_o) and np.array_equal(rec_g, rec_o)


@pytest.mark.parametrize("how", ["render", "async", "train"])
def test_batches_of_clipped_and_whole_views_in_turn(how):
    from difftetvr_b200 import synthetic as S
    from difftetvr_b200.batch import BatchRenderer, View
    sc = Scene(6, 93, seed=7)
    mesh, r = sc.make_renderer()
    br = BatchRenderer([mesh], attenuation=1.0, use_early_ray_termination=False)
    br.reserve(4, 4 * len(sc.pos), 4 * 93 * 93, 4 * 93 * 93 * 200, len(sc.pos))
    br.set_graph(how == "train")
    for cams in [[WHOLE, WHOLE], [WHOLE, NEAR], [NEAR, FAR_OFF], [WHOLE, WHOLE], [WHOLE, WHOLE], [FAR_OFF, WHOLE]]:
        views = [View(mesh=0, view_matrix=S.look_at_view(c), width=93, height=93, fovy=sc.fovy) for c in cams]
        if how == "render":
            br.render(views)
        elif how == "async":
            br.render_async(views)
            torch.cuda.synchronize()
            assert br.render_status()[0]
        else:
            for v in views:
                v.target = torch.zeros((93, 93, 4), device="cuda")
            br.train_step(views, lr_positions=0.0, lr_colors=0.0)  # the mesh stays
        for v in views:
            r.set_view_matrix(v.view_matrix)
            assert float((v.image - r.render()).abs().max()) <= 1e-6
