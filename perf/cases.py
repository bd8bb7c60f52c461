"""Performance cases of the framework: what a user's program has it do, through the public entry points, from a
single small view to a training step on a mesh of 5.3 M tets, with the exact (64-bit) outputs beside them.

The meshes are Kuhn-subdivided cube grids with jittered interior vertices, coloured by sums of Gaussians and seen by
cameras on a sphere, as in the tests and the benchmark (n: cubes per axis, 6 n^3 tets)."""
from __future__ import annotations

import math

import numpy as np
import torch

FOVY = math.radians(45.0)
CAMERAS = 4            # a program renders another view in each pass
ERT_THRESHOLD = 1e-4   # the renderer's default
LR_COLORS, LR_POSITIONS = 1e-2, 1e-4


def listed():
    return [
        # Interactive preview of a very small mesh: launches and latency are all there is.
        {"name": "view_8_64", "kind": "view", "n": 8, "w": 64, "h": 64, "atten": 1.0},
        # Preview of a mid-size mesh at the reference's default attenuation (opaque), odd window, no gradients.
        {"name": "view_33_721x479", "kind": "view", "n": 33, "w": 721, "h": 479, "atten": 100.0},
        # First training stage of a coarse-to-fine run: small mesh, small image.
        {"name": "step_16_256", "kind": "step", "n": 16, "w": 256, "h": 256, "atten": 1.0},
        # The gradient pass that picks the vertices to split: absolute gradients, odd image, ray termination in use.
        {"name": "step_37_613x401_abs", "kind": "step_abs", "n": 37, "w": 613, "h": 401, "atten": 20.0},
        # Ordinary training step.
        {"name": "step_64_512", "kind": "step", "n": 64, "w": 512, "h": 512, "atten": 1.0},
        # The benchmark's training step.
        {"name": "step_64_1024", "kind": "step", "n": 64, "w": 1024, "h": 1024, "atten": 1.0},
        # Training step at the end of a refinement: 5.3 M tets.
        {"name": "step_96_1536", "kind": "step", "n": 96, "w": 1536, "h": 1536, "atten": 1.0},
        # Training step with one colour per tet.
        {"name": "cells_48_768", "kind": "cells", "n": 48, "w": 768, "h": 768, "atten": 1.0},
        # Training step with the intersection renderer, which keeps no fragment lists.
        {"name": "raytet_64_1024", "kind": "raytet", "n": 64, "w": 1024, "h": 1024, "atten": 1.0},
        # Training step whose fragment lists exceed the memory allowed for them (row bands, lists built twice).
        {"name": "budget_64_1024", "kind": "budget", "n": 64, "w": 1024, "h": 1024, "atten": 1.0},
        # One captured step over many views of three meshes.
        {"name": "batch_train_24_384", "kind": "batch", "n": 24, "w": 384, "h": 384, "atten": 1.0, "views": 12},
        # The tet-quality regularizer of a training step.
        {"name": "regularizer_64", "kind": "regularizer", "n": 64, "w": 1, "h": 1, "atten": 1.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("view", "view", "step", "step", "step", "step_abs", "cells", "raytet", "budget", "batch",
                       "regularizer"))
    atten = rng.choice((1.0, 1.0, 5.0, 20.0, 100.0))
    if kind == "regularizer":
        return {"kind": kind, "n": _log_int(rng, 6, 90), "w": 1, "h": 1, "atten": 1.0}
    n, h = _log_int(rng, 6, 72), _log_int(rng, 48, 1100)
    w = max(40, int(h * rng.choice((1.0, 1.0, rng.uniform(0.7, 1.6)))))
    case = {"kind": kind, "n": n, "w": w, "h": h, "atten": atten}
    if kind == "batch":
        case.update(n=min(n, 32), w=min(w, 400), h=min(h, 400), views=rng.randint(2, 14))
    return case


# -- inputs -------------------------------------------------------------------
def _mesh_data(n, seed):
    from difftetvr_b200 import synthetic as S
    cells, pos = S.kuhn_mesh(n, seed=seed)
    return cells, pos, S.gaussian_colors(pos, seed=seed)


def _cell_colors(cells, colors):
    return colors[cells.astype(np.int64)].mean(axis=1).astype(np.float32)


def _cameras(seed, count):
    from difftetvr_b200 import synthetic as S
    return [S.sphere_camera(1000 * (seed + 1) + k) for k in range(count)]


def _target(w, h, seed, device="cuda"):
    """A smooth RGBA image: what the training fits to."""
    rng = np.random.default_rng(seed + 31)
    y, x = torch.meshgrid(torch.linspace(-1, 1, h, device=device), torch.linspace(-1, 1, w, device=device),
                          indexing="ij")
    image = torch.zeros((h, w, 4), device=device)
    for _ in range(6):
        cx, cy, s = rng.uniform(-0.5, 0.5), rng.uniform(-0.5, 0.5), rng.uniform(0.1, 0.4)
        color = torch.tensor(rng.uniform(0.0, 0.4, 4).astype(np.float32), device=device)
        image += torch.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2 * s * s))[..., None] * color
    return image.clamp_(0.0, 1.0)


def _batch_meshes(case):
    n = case["n"]
    return [n, max(4, n // 2), max(5, (3 * n) // 2)]


def _batch_sizes(case):
    """(mesh, width, height) of each view: the meshes in turn, a third of the views at half the size."""
    out = []
    for k in range(case["views"]):
        d = 2 if k % 3 == 2 else 1
        out.append((k % 3, max(16, case["w"] // d), max(16, case["h"] // d)))
    return out


def prepare(case, seed):
    import difftetvr_b200 as d
    from difftetvr_b200.batch import BatchRenderer, View
    kind, n, w, h = case["kind"], case["n"], case["w"], case["h"]
    state = {"kind": kind, "pass": 0}

    def tet_mesh(n, seed):
        cells, pos, col = _mesh_data(n, seed)
        mesh = d.TetMesh()
        mesh.set_use_gradients(kind != "view")
        if kind == "cells":
            mesh.set_tet_mesh_data_cell(cells, pos, _cell_colors(cells, col))
        else:
            mesh.set_tet_mesh_data(cells, pos, col)
        return mesh

    if kind == "batch":
        meshes = [tet_mesh(m, seed + 17 * i) for i, m in enumerate(_batch_meshes(case))]
        cams = _cameras(seed, case["views"])
        views = [View(mesh=m, view_matrix=cams[k], width=vw, height=vh, fovy=FOVY, target=_target(vw, vh, seed + k))
                 for k, (m, vw, vh) in enumerate(_batch_sizes(case))]
        batch = BatchRenderer(meshes, attenuation=case["atten"])
        batch.set_graph(True)
        return dict(state, meshes=meshes, views=views, batch=batch)
    mesh = tet_mesh(n, seed)
    if kind == "regularizer":
        from difftetvr_b200.regularizer import TetRegularizer
        return dict(state, mesh=mesh, regularizer=TetRegularizer(mesh, 0.1, 100.0),
                    grad=torch.zeros_like(mesh.get_vertex_positions()).detach())
    renderer = d.Renderer(d.RendererType.INTERSECTION if kind == "raytet" else d.RendererType.PPLL)
    renderer.set_tet_mesh(mesh)
    renderer.set_viewport_size(w, h)
    renderer.set_camera_fovy(FOVY)
    renderer.set_attenuation(case["atten"])
    if kind == "budget":
        # About a quarter of the records of the whole image.
        renderer.set_fragment_budget_bytes(max(1 << 16, int(8 * _fragments(case) / 4)))
    state.update(mesh=mesh, renderer=renderer, cameras=_cameras(seed, CAMERAS))
    if kind != "view":
        diff = d.DifferentiableRenderer(renderer)
        diff.set_use_abs_grad(kind == "step_abs")
        state.update(diff=diff, target=_target(w, h, seed))
    return state


# -- one pass -----------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "batch":
        loss = state["batch"].train_step(state["views"], lr_positions=LR_POSITIONS, lr_colors=LR_COLORS,
                                         clamp_colors=1)
        return {"loss": loss, "images": [v.image for v in state["views"]],
                "positions": [m.get_vertex_positions() for m in state["meshes"]],
                "colors": [m.get_vertex_colors() for m in state["meshes"]]}
    if kind == "regularizer":
        state["grad"].zero_()
        loss = state["regularizer"].compute_grad_into(state["grad"])
        return {"loss": loss, "grad": state["grad"]}
    renderer, mesh = state["renderer"], state["mesh"]
    renderer.set_view_matrix(state["cameras"][state["pass"] % CAMERAS])
    state["pass"] += 1
    if kind == "view":
        return renderer.render()
    from difftetvr_b200.optim import l2_loss
    positions = mesh.get_vertex_positions()
    colors = mesh.get_cell_colors() if kind == "cells" else mesh.get_vertex_colors()
    positions.grad.zero_()
    colors.grad.zero_()
    image = state["diff"]()
    loss = l2_loss(image, state["target"])
    loss.backward()
    return {"image": image, "loss": loss, "grad_positions": positions.grad, "grad_colors": colors.grad}


# -- what a pass cannot do without ----------------------------------------------
def _fragments(case):
    """Faces crossed by the pixels' rays: about 2.7 per pixel and cube of an axis where the mesh fills a square image."""
    return 2.7 * case["n"] * case["h"] * min(case["h"], case["w"])


def work(case):
    kind, n, pixels = case["kind"], case["n"], case["w"] * case["h"]
    if kind == "batch":
        nbytes = flops = 0.0
        for m, w, h in _batch_sizes(case):
            n = _batch_meshes(case)[m]
            nbytes += 4 * 16 * w * h
            flops += 530.0 * _fragments({"n": n, "w": w, "h": h})
        for n in _batch_meshes(case):
            nbytes += 16 * 6 * n ** 3 + 6 * 28 * (n + 1) ** 3
        return {"bytes": nbytes, "flops": flops}
    tets, verts = 6 * n ** 3, (n + 1) ** 3
    if kind == "regularizer":
        return {"bytes": 16.0 * tets + 36.0 * verts, "flops": 250.0 * tets}
    mesh_bytes = 16.0 * tets + 12.0 * verts + 16.0 * (tets if kind == "cells" else verts)
    if kind == "view":
        return {"bytes": mesh_bytes + 16.0 * pixels, "flops": 180.0 * _fragments(case)}
    grads = 12.0 * verts + 16.0 * (tets if kind == "cells" else verts)
    return {"bytes": 2 * mesh_bytes + grads + 3 * 16.0 * pixels,
            "flops": (300.0 if kind == "cells" else 530.0) * _fragments(case)}


# -- the same in 64 bits, in plain torch ------------------------------------------
class _Faces:
    """Unique faces of the tets: vertices (in the order of the first tet that has the face) and the tets beside it."""

    def __init__(self, cells):
        c = torch.as_tensor(cells.astype(np.int64)).cuda()
        order = torch.tensor([[0, 1, 2], [1, 0, 3], [0, 2, 3], [2, 1, 3]], device=c.device)
        every = c[:, order].reshape(-1, 3)
        s = every.sort(dim=1).values
        base = int(c.max()) + 1
        # Lexicographic order of the sorted triples, copies of a face in the order of their tets.
        perm = torch.argsort(s[:, 2], stable=True)
        perm = perm[torch.argsort((s[:, 0] * base + s[:, 1])[perm], stable=True)]
        t = s[perm]
        first = torch.ones(len(perm), dtype=torch.bool, device=c.device)
        first[1:] = (t[1:] != t[:-1]).any(dim=1)
        at = first.nonzero()[:, 0]
        self.tri = every[perm[at]]
        count = torch.diff(torch.cat([at, torch.tensor([len(perm)], device=c.device)]))
        tets = perm // 4
        second = torch.where(count == 2, tets[(at + 1).clamp(max=len(perm) - 1)], torch.full_like(at, -1))
        self.tets = torch.stack([tets[at], second], dim=1)


class _Camera:
    def __init__(self, view, w, h):
        self.view = torch.tensor(view, dtype=torch.float64).float().double().cuda()  # column-major, as given in 32 bits
        # fovy is given in 32 bits, the focal length follows in 64.
        self.f = 0.5 * h / math.tan(0.5 * float(np.float32(FOVY)))
        self.w, self.h = w, h

    def project(self, p):
        """Screen position, 1 / depth and depth of points [..., 3] in 64 bits."""
        v = self.view
        x, y, z = p.unbind(-1)
        xv, yv, zv = (v[k] * x + v[4 + k] * y + v[8 + k] * z + v[12 + k] for k in range(3))
        return 0.5 * self.w - self.f * xv / zv, 0.5 * self.h + self.f * yv / zv, -1.0 / zv, -zv

    def project32(self, p):
        """The same in 32 bits, rounded after each operation: what coverage and depth order are decided on."""
        v = self.view.float()
        x, y, z = p.unbind(-1)
        xv, yv, zv = (((v[k] * x + v[4 + k] * y) + v[8 + k] * z) + v[12 + k] for k in range(3))
        ze = -zv
        iz = 1.0 / ze
        f = torch.tensor(self.f, dtype=torch.float64, device=p.device).float()
        return torch.stack([0.5 * self.w + f * (xv * iz), 0.5 * self.h - f * (yv * iz), iz, ze], dim=-1)


def _fragment_lists(faces, pos, cam, row0, row1, most=24_000_000):
    """(pixel, face) of every pixel centre of rows [row0, row1) that a face covers, sorted by pixel, depth and face."""
    v32 = cam.project32(pos)
    fix = torch.round(v32[:, :2] * 256.0).to(torch.int64)
    q = fix[faces.tri]
    area = (q[:, 1, 0] - q[:, 0, 0]) * (q[:, 2, 1] - q[:, 0, 1]) - (q[:, 1, 1] - q[:, 0, 1]) * (q[:, 2, 0] - q[:, 0, 0])
    lo, hi = q.amin(dim=1), q.amax(dim=1)
    x0, x1 = (-((128 - lo[:, 0]) >> 8)).clamp(min=0), ((hi[:, 0] - 128) >> 8).clamp(max=cam.w - 1)
    y0, y1 = (-((128 - lo[:, 1]) >> 8)).clamp(min=row0), ((hi[:, 1] - 128) >> 8).clamp(max=row1 - 1)
    keep = ((area != 0) & (x0 <= x1) & (y0 <= y1)).nonzero()[:, 0]
    bw = (x1 - x0 + 1)[keep]
    size = bw * (y1 - y0 + 1)[keep]
    ends = torch.cumsum(size, 0)
    pixels, ids, depths = [], [], []
    begin = 0
    while begin < len(keep):
        base = int(ends[begin - 1]) if begin else 0
        end = max(begin + 1, int(torch.searchsorted(ends, base + most)))
        sel = torch.arange(begin, end, device=pos.device)
        owner = torch.repeat_interleave(sel, size[begin:end])
        k = torch.arange(len(owner), device=pos.device) - ((ends - size)[owner] - base)
        f = keep[owner]
        px, py = x0[f] + k % bw[owner], y0[f] + k // bw[owner]
        r = fix[faces.tri[f]] - torch.stack([256 * px + 128, 256 * py + 128], dim=-1)[:, None]
        swap = (area[f] < 0)[:, None]
        a, b, c = r[:, 0], torch.where(swap, r[:, 2], r[:, 1]), torch.where(swap, r[:, 1], r[:, 2])
        inside = torch.ones(len(f), dtype=torch.bool, device=pos.device)
        for s, e in ((b, c), (c, a), (a, b)):
            dx, dy = e[:, 0] - s[:, 0], e[:, 1] - s[:, 1]
            edge = dy * s[:, 0] - dx * s[:, 1]
            inside &= (edge > 0) | ((edge == 0) & ((dy < 0) | ((dy == 0) & (dx > 0))))
        f, px, py = f[inside], px[inside], py[inside]
        # The depth that orders the list, in 32 bits.
        va, vb, vc = v32[faces.tri[f]].unbind(1)
        qx, qy = px.float() + 0.5, py.float() + 0.5
        d = [(v[:, 0] - qx, v[:, 1] - qy) for v in (va, vb, vc)]
        e = [d[i][0] * d[j][1] - d[i][1] * d[j][0] for i, j in ((1, 2), (2, 0), (0, 1))]
        z = ((e[0] + e[1]) + e[2]) / ((e[0] * va[:, 2] + e[1] * vb[:, 2]) + e[2] * vc[:, 2])
        near = torch.minimum(torch.minimum(va[:, 3], vb[:, 3]), vc[:, 3])
        far = torch.maximum(torch.maximum(va[:, 3], vb[:, 3]), vc[:, 3])
        pixels.append(py * cam.w + px)
        ids.append(f)
        depths.append(torch.minimum(torch.maximum(z, near), far))
        begin = end
    if not pixels:
        empty = torch.zeros(0, dtype=torch.int64, device=pos.device)
        return empty, empty
    pixel, face, depth = torch.cat(pixels), torch.cat(ids), torch.cat(depths)
    perm = torch.argsort(face)
    perm = perm[torch.argsort(depth[perm], stable=True)]
    perm = perm[torch.argsort(pixel[perm], stable=True)]
    return pixel[perm], face[perm]


def _starts(pixel):
    """For each fragment, the index of its pixel's first one."""
    first = torch.ones(len(pixel), dtype=torch.bool, device=pixel.device)
    first[1:] = pixel[1:] != pixel[:-1]
    at = first.nonzero()[:, 0]
    return torch.repeat_interleave(at, torch.diff(torch.cat([at, torch.tensor([len(pixel)], device=pixel.device)])))


def _shade(kind, cam, atten, ert, pixel, vertex_pos, colors):
    """RGBA of the listed pixels' fragments: `vertex_pos` [N, 3, 3] of each fragment's face, `colors` [N, 3, 4] of its
    vertices, or [N - 1, 4] of the tet between each fragment and the next (alpha 0: none)."""
    sx, sy, iz, ze = cam.project(vertex_pos)
    qx, qy = (pixel % cam.w).double() + 0.5, (pixel // cam.w).double() + 0.5
    dx, dy = sx - qx[:, None], sy - qy[:, None]
    e = torch.stack([dx[:, i] * dy[:, j] - dy[:, i] * dx[:, j] for i, j in ((1, 2), (2, 0), (0, 1))], dim=1)
    u = e / e.sum(dim=1, keepdim=True) * iz
    zb = 1.0 / u.sum(dim=1)
    z = torch.minimum(torch.maximum(zb, ze.amin(dim=1)), ze.amax(dim=1))
    t = z[1:] - z[:-1]
    if kind == "raytet":
        t = t * torch.sqrt(1.0 + ((qx[1:] - 0.5 * cam.w) / cam.f) ** 2 + ((qy[1:] - 0.5 * cam.h) / cam.f) ** 2)
    pair = (pixel[1:] == pixel[:-1]).double()
    if kind == "cells":
        x = colors[:, 3] * atten * t * pair
    else:
        col = ((u * zb[:, None])[..., None] * colors).sum(dim=1)
        c0, c1 = col[:-1], col[1:]
        t = 0.25 * t
        s = (torch.arange(4, device=t.device, dtype=torch.float64) + 0.5) / 4
        a = (c0[:, 3:] + (c1 - c0)[:, 3:] * s) * atten
        xs = a * t[:, None]
        x = xs.sum(dim=1) * pair
    # Transmittance before each segment: exp of minus the optical depth since the pixel's first fragment.
    depth = torch.cat([x.new_zeros(1), torch.cumsum(x, 0)])
    start = _starts(pixel)
    before = depth[:-1] - depth[start[:-1]]
    go = pair
    if ert:
        go = pair * (torch.exp(-before) >= ERT_THRESHOLD)
    front = torch.exp(-before) * go
    if kind == "cells":
        rgb = (front * -torch.expm1(-x))[:, None] * colors[:, :3]
    else:
        # (1 - A) c0 + K (c0 - c1) of the four parts, A = exp(-x), K = (t + 1 / a) A - 1 / a = -t x psi(x).
        parts = xs * go[:, None]
        inner = torch.exp(-(torch.cumsum(parts, dim=1) - parts)) * front[:, None]
        big = xs.clamp(min=0.02)
        small = xs.clamp(max=0.05)
        series = sum((-1) ** m * (m + 1) / math.factorial(m + 2) * small ** m for m in range(9))
        direct = (-torch.expm1(-big) / big - torch.exp(-big)) / big
        k = t[:, None] * xs * torch.where(xs < 0.04, series, direct)
        # c1 - c0 of a part is a quarter of the segment's; K is per unit length of the part.
        lead = inner * -torch.expm1(-xs)
        along = inner * torch.where(t[:, None] != 0, k / torch.where(t == 0, torch.ones_like(t), t)[:, None],
                                    torch.zeros_like(k))
        k = along * t[:, None]
        s0 = torch.arange(4, device=t.device, dtype=torch.float64) / 4
        rgb = lead.sum(1)[:, None] * c0[:, :3] + ((lead * s0 + 0.25 * k).sum(1))[:, None] * (c1 - c0)[:, :3]
    total = x.new_zeros(cam.w * cam.h, 4)
    total = total.index_add(0, pixel[:-1], torch.cat([rgb, (x * go)[:, None]], dim=1))
    return torch.cat([total[:, :3], -torch.expm1(-total[:, 3:])], dim=1)


def _exact_view(kind, cells, faces, pos, col, view, w, h, atten, ert, adjoint=None, chunk=6_000_000):
    """Image [h, w, 4] in 64 bits, or with `adjoint` (image -> its adjoint [h, w, 4]) the image and the gradients of
    positions and colours."""
    cam = _Camera(view, w, h)
    p32 = torch.as_tensor(pos).cuda()
    p, c = p32.double(), torch.as_tensor(col).cuda().double()
    rows = max(1, int(chunk / max(1.0, 2.7 * round((len(cells) / 6) ** (1 / 3)) * w)))
    image = torch.zeros((h * w, 4), dtype=torch.float64, device="cuda")
    gp, gc = torch.zeros_like(p), torch.zeros_like(c)

    def chunks():
        for y in range(0, h, rows):
            pixel, face = _fragment_lists(faces, p32, cam, y, min(h, y + rows))
            if len(pixel) < 2:
                continue
            tri = faces.tri[face]
            if kind == "cells":
                a, b = faces.tets[face[:-1]], faces.tets[face[1:]]
                x0 = ((a[:, 0] == b[:, 0]) | (a[:, 0] == b[:, 1])) & (pixel[1:] == pixel[:-1])
                x1 = ((a[:, 1] == b[:, 0]) | (a[:, 1] == b[:, 1])) & (a[:, 1] >= 0) & (pixel[1:] == pixel[:-1])
                # The renderer tries the later face's tets first; the two faces share one tet at most.
                open_ = torch.where(x0, a[:, 0], torch.where(x1, a[:, 1], torch.full_like(a[:, 0], -1)))
                yield pixel, tri, open_
            else:
                yield pixel, tri, None

    def leaves(tri, open_, grad):
        vp = p[tri].requires_grad_(grad)
        if open_ is None:
            return vp, c[tri].requires_grad_(grad)
        cc = c[open_.clamp(min=0)] * (open_ >= 0)[:, None]
        return vp, cc.requires_grad_(grad)

    with torch.no_grad():
        for pixel, tri, open_ in chunks():
            vp, cc = leaves(tri, open_, False)
            image += _shade(kind, cam, atten, ert, pixel, vp, cc)
    out = image.reshape(h, w, 4)
    if adjoint is None:
        return out
    g = adjoint(out).reshape(h * w, 4)
    for pixel, tri, open_ in chunks():
        vp, cc = leaves(tri, open_, True)
        dp, dc = torch.autograd.grad((_shade(kind, cam, atten, ert, pixel, vp, cc) * g).sum(), (vp, cc))
        if kind == "step_abs":
            dp, dc = dp.abs(), dc.abs()
        gp.index_add_(0, tri.reshape(-1), dp.reshape(-1, 3))
        if open_ is None:
            gc.index_add_(0, tri.reshape(-1), dc.reshape(-1, 4))
        else:
            gc.index_add_(0, open_.clamp(min=0), dc * (open_ >= 0)[:, None])
    return out, gp, gc


def _exact_regularizer(cells, pos, reg_lambda, beta):
    p = torch.as_tensor(pos).cuda().double()
    v = p[torch.as_tensor(cells.astype(np.int64)).cuda()]
    e1, e2, e3 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0], v[:, 3] - v[:, 0]
    dd = torch.stack([torch.linalg.cross(e2, e3), torch.linalg.cross(e3, e1), torch.linalg.cross(e1, e2)], dim=1)
    dd = torch.cat([-dd.sum(dim=1, keepdim=True), dd], dim=1)
    det = (dd[:, 3] * e3).sum(1)
    s = sum(((v[:, i] - v[:, j]) ** 2).sum(1) for i in range(4) for j in range(i))
    c = 12.0 * math.sqrt(3.0)
    q = -c * det / s ** 1.5
    # The denominator's clamp belongs to the measure's definition.
    den = torch.clamp(s ** 2.5, min=1e-5)
    ds = 2.0 * (4.0 * v - v.sum(dim=1, keepdim=True))
    dq = (-c * s / den)[:, None, None] * dd + (1.5 * c * det / den)[:, None, None] * ds
    g = (-reg_lambda * torch.sigmoid(-beta * q))[:, None, None] * dq
    grad = torch.zeros_like(p).index_add_(0, torch.as_tensor(cells.astype(np.int64)).cuda().reshape(-1),
                                          g.reshape(-1, 3))
    return {"loss": (reg_lambda / beta * torch.nn.functional.softplus(-beta * q, threshold=1e9)).sum().reshape(1),
            "grad": grad}


def exact(case, seed):
    kind, w, h, atten = case["kind"], case["w"], case["h"], case["atten"]
    if kind != "batch" and _fragments(case) > 2.2e8:
        return None  # more than about 20 seconds
    if kind == "batch":
        sizes, cams = _batch_sizes(case), _cameras(seed, case["views"])
        data = [_mesh_data(m, seed + 17 * i) for i, m in enumerate(_batch_meshes(case))]
        faces = [_Faces(m[0]) for m in data]
        grads = [[torch.zeros(m[1].shape, dtype=torch.float64, device="cuda"),
                  torch.zeros(m[2].shape, dtype=torch.float64, device="cuda")] for m in data]
        loss, images = 0.0, []
        for k, (m, vw, vh) in enumerate(sizes):
            diff = {}

            def adjoint(image, k=k, vw=vw, vh=vh, diff=diff):
                diff["d"] = image - _target(vw, vh, seed + k).double()
                return 2.0 / image.numel() * diff["d"]

            img, gp, gc = _exact_view("step", data[m][0], faces[m], data[m][1], data[m][2], cams[k], vw, vh, atten,
                                      True, adjoint)
            loss = loss + (diff["d"] ** 2).mean()
            images.append(img)
            grads[m][0] += gp
            grads[m][1] += gc

        def adam(p, g, lr):
            return torch.as_tensor(p).cuda().double() - lr * g / (g.abs() + 1e-8)

        return {"loss": loss, "images": images,
                "positions": [adam(d[1], g[0], LR_POSITIONS) for d, g in zip(data, grads)],
                "colors": [adam(d[2], g[1], LR_COLORS).clamp(min=0.0) for d, g in zip(data, grads)]}
    cells, pos, col = _mesh_data(case["n"], seed)
    if kind == "regularizer":
        return _exact_regularizer(cells, pos, float(np.float32(0.1)), 100.0)
    if kind == "cells":
        col = _cell_colors(cells, col)
    view = _cameras(seed, CAMERAS)[0]
    faces = _Faces(cells)
    if kind == "view":
        # Early ray termination belongs to training.
        return _exact_view(kind, cells, faces, pos, col, view, w, h, atten, False)
    target = _target(w, h, seed).double()
    image, gp, gc = _exact_view(kind, cells, faces, pos, col, view, w, h, atten, True,
                                lambda image: 2.0 / image.numel() * (image - target))
    # The intersection renderer takes faces at (nearly) one depth in the order of the tets, not of their depths, and the
    # position gradients of thin faces show which.
    return {"image": image, "loss": ((image - target) ** 2).mean(),
            "grad_positions": None if kind == "raytet" else gp, "grad_colors": gc}
