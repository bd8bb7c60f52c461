"""Composite with its loads ahead (few pixels, or many vertices per pixel) and
without (many pixels on a small mesh), per-vertex and per-cell, at list lengths
from nothing up and image sizes off the tiles: both sides of the rule against
the FP64 oracle (1e-5 absolute, the path's bound)."""
import numpy as np
import pytest

from helpers import Scene

pytestmark = pytest.mark.gpu

IMG_TOL = 1e-5


# 437^2 pixels are just over 148 x 1280: 1^3 and 3^3 (8 and 64 vertices) run
# plain there, 15^3 (4096 vertices) ahead; 435^2 is just under.
@pytest.mark.parametrize("n,res", [(1, 5), (2, 33), (1, 435), (1, 437), (3, 437), (15, 437)])
@pytest.mark.parametrize("cells", [False, True])
def test_images_match_fp64_oracle(oracle, n, res, cells):
    import difftetvr_b200 as d
    sc = Scene(n, res, seed=4)
    mesh, r = sc.make_renderer()
    fa = oracle.Faces(sc.cells, sc.pos.shape[0])
    cam, prm = sc.oracle_camera(oracle), sc.oracle_params(oracle)
    if cells:
        cc = sc.col[sc.cells.astype(np.int64)].mean(axis=1).astype(np.float32)
        mesh = d.TetMesh()
        mesh.set_use_gradients(True)
        mesh.set_tet_mesh_data_cell(sc.cells, sc.pos, cc)
        r.set_tet_mesh(mesh)
        ref = oracle.render_cells(fa, sc.pos, cc, cam, prm)[0]
    else:
        ref = oracle.render(fa, sc.pos, sc.col, cam, prm)[0]
    assert np.abs(r.render().cpu().numpy() - ref).max() <= IMG_TOL
