// Fragment lists by walking the mesh, single view (the walk itself and why it
// finds the rasteriser's lists: dtv_walk.cuh), and the mesh's walk tables.
//
// One thread per pixel makes the pixel's list in order.  The vertices of the
// face it stands on stay in registers, so a record costs one new vertex row (32
// bytes), one link (16 bytes) and a quarter of a 32-byte store, instead of the
// fill's counter atomic and scattered 8-byte store and the record's share of a
// sort.  Fill (with its face order) + sort against the walk with the fill of
// the boundary faces it starts from (us): 1,348 + 307 -> 463 at 64^3 / 512^2
// (36.8 M records), 2,101 + 1,081 -> 1,270 at 64^3 / 1024^2 (147 M), 6,833 +
// 4,104 -> 4,118 at 96^3 / 1536^2 (495 M), 119 + 69 -> 81 at 16^3 / 256^2.
// Bound by instruction issue (143 warp instructions per 32 records, issue
// active 57 % at 25 warps per SM) and the L1 data pipe (64 %); with few pixels
// by the latency of a step, about 1.2 us.  Composited in the same pass (122
// registers) it was 15 % faster below 512^2 and 4 % slower above, and its
// depths were rounded in another vertex order than the composite's.
#include "dtv_internal.h"
#include "dtv_walk.cuh"

namespace dtv {

namespace {

// Local vertices of face j of a tet (TetMesh.cpp:1175-1181); face j lies
// opposite local vertex 3 - j.
__device__ __constant__ int kFaceVerts[4][3] = {{0, 1, 2}, {1, 0, 3}, {0, 2, 3}, {2, 1, 3}};

// Whether the stored order s of face j is an odd permutation of the tet's own
// (table) order; *same: it holds the same vertices at all.
__device__ bool face_odd(const uint32_t (&c)[4], int j, const uint32_t (&s)[3], bool* same) {
    const uint32_t a = c[kFaceVerts[j][0]], b = c[kFaceVerts[j][1]], d = c[kFaceVerts[j][2]];
    const bool even = (s[0] == a && s[1] == b && s[2] == d) || (s[0] == b && s[1] == d && s[2] == a) ||
                      (s[0] == d && s[1] == a && s[2] == b);
    const bool odd = (s[0] == b && s[1] == a && s[2] == d) || (s[0] == a && s[1] == d && s[2] == b) ||
                     (s[0] == d && s[1] == b && s[2] == a);
    *same = even || odd;
    return odd;
}

}  // namespace

__global__ void __launch_bounds__(256) k_build_walk(const uint4* __restrict__ cells, uint32_t T,
                                                    const uint4* __restrict__ tet_faces,
                                                    const uint4* __restrict__ faces, const uint2* __restrict__ f2t,
                                                    uint4* __restrict__ links, uint32_t* __restrict__ bad) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const uint4 cv = cells[t], tf = tet_faces[t];
    const uint32_t c[4] = {cv.x, cv.y, cv.z, cv.w}, fs[4] = {tf.x, tf.y, tf.z, tf.w};
    bool ok = c[0] != c[1] && c[0] != c[2] && c[0] != c[3] && c[1] != c[2] && c[1] != c[3] && c[2] != c[3];
    for (int k = 0; k < 4; ++k) {
        const int j = 3 - k;
        const uint32_t f = fs[j];
        const uint4 fv = faces[f];
        const uint32_t s[3] = {fv.x, fv.y, fv.z};
        const uint2 ft = f2t[f];
        bool same, alike = false;
        const bool odd = face_odd(c, j, s, &same);
        ok &= same && (ft.x == t || ft.y == t) && ft.x != ft.y;
        const uint32_t other = ft.x == t ? ft.y : ft.x;
        const bool bnd = (fv.w & 1u) != 0u;
        ok &= bnd == (other == 0xffffffffu);
        uint32_t third = 0;
        for (int q = 0; q < 4; ++q)
            if (c[q] == s[2]) third = uint32_t(q);
        uint32_t next = c[k], map = 0;
        if (other < T) {
            const uint4 ov = cells[other], of = tet_faces[other];
            const uint32_t oc[4] = {ov.x, ov.y, ov.z, ov.w}, ofs[4] = {of.x, of.y, of.z, of.w};
            int across = -1;
            for (int q = 0; q < 4; ++q)
                if (ofs[3 - q] == f) {
                    ok &= across < 0;
                    across = q;
                }
            ok &= across >= 0;
            if (across >= 0) {
                bool osame;
                alike = face_odd(oc, 3 - across, s, &osame) == odd;
                ok &= osame;
                next = oc[across];
                for (int l = 0; l < 4; ++l) {
                    uint32_t m = uint32_t(across);
                    for (int q = 0; q < 4; ++q)
                        if (l != k && oc[q] == c[l]) m = uint32_t(q);
                    map |= m << (8 * l);
                }
            }
        } else {
            ok &= bnd;
        }
        const bool flip = ft.x != t && !odd;
        links[4 * size_t(t) + k] = make_uint4((other < T ? other : kWalkNoTet) | (third << 28) | (flip ? 1u << 30 : 0u) |
                                                  (alike ? 1u << 31 : 0u),
                                              (f << 2) | (bnd ? 2u : 0u) | (odd ? 1u : 0u), next, map);
    }
    if (!ok) *bad = 1u;
}

__global__ void __launch_bounds__(256) k_build_walk_start(const uint4* __restrict__ cells,
                                                          const uint4* __restrict__ tet_faces,
                                                          const uint4* __restrict__ faces,
                                                          const uint2* __restrict__ f2t,
                                                          const uint32_t* __restrict__ bf_global, uint32_t Nb,
                                                          uint4* __restrict__ start) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Nb) return;
    const uint32_t f = bf_global[i], t = f2t[f].x;
    const uint4 cv = cells[t], tf = tet_faces[t], fv = faces[f];
    const uint32_t c[4] = {cv.x, cv.y, cv.z, cv.w}, s[3] = {fv.x, fv.y, fv.z};
    const uint32_t k = tf.x == f ? 3u : (tf.y == f ? 2u : (tf.z == f ? 1u : 0u));
    uint32_t loc = k << 24;
    for (int j = 0; j < 3; ++j)
        for (uint32_t q = 0; q < 4; ++q)
            if (c[q] == s[j]) loc = (loc & ~(255u << (8 * j))) | (q << (8 * j));
    start[i] = make_uint4(t, c[k], loc, f);
}

void launch_build_walk(const uint4* cells, uint32_t T, const uint4* tet_faces, const uint4* faces, const uint2* f2t,
                       const uint32_t* bf_global, uint32_t Nb, uint4* links, uint4* start, uint32_t* bad,
                       cudaStream_t s) {
    if (T == 0) return;
    k_build_walk<<<(T + 255) / 256, 256, 0, s>>>(cells, T, tet_faces, faces, f2t, links, bad);
    if (Nb) k_build_walk_start<<<(Nb + 255) / 256, 256, 0, s>>>(cells, tet_faces, faces, f2t, bf_global, Nb, start);
}

constexpr int kWalkListThreads = 128;

// Blocks of four warps of 8 x 4 pixels each, 16 x 8 pixels in all.
__global__ void __launch_bounds__(kWalkListThreads) k_walk_lists(
    const u64* __restrict__ offsets, u64* __restrict__ records, uint32_t* __restrict__ counts, WalkMesh wm,
    const WalkVertRow* __restrict__ verts, int W, int row0, int row1, ListInfo* __restrict__ info,
    uint32_t* __restrict__ redo, bool guarded) {
    constexpr int N = kWalkListThreads;
    __shared__ u64 starts[kWalkStarts * N];
    __shared__ u64 recs[4 * N];
    if (guarded && info->whole == 0u) return;
    const int lane = int(threadIdx.x & 31u), w = int(threadIdx.x >> 5);
    const int px = blockIdx.x * 16 + (w & 1) * 8 + lane % 8;
    const int py = row0 + int(blockIdx.y) * 8 + (w >> 1) * 4 + lane / 8;
    if (px >= W || py >= row1) return;
    const size_t p = size_t(py) * W + px;
    walk_pixel(px, py, p, offsets, records, counts, wm, verts, WalkSmem{starts + threadIdx.x, recs + threadIdx.x, N},
               WalkRedo{&info->n_redo, redo}, uint32_t(p));
}

void launch_walk_lists(const WalkMesh& wm, const u64* offsets, u64* records, uint32_t* counts,
                       const WalkVertRow* verts, int W, int row0, int row1, ListInfo* info, uint32_t* redo,
                       bool guarded, cudaStream_t s) {
    if (row1 <= row0) return;
    dim3 grid((W + 15) / 16, (row1 - row0 + 7) / 8);
    k_walk_lists<<<grid, kWalkListThreads, 0, s>>>(offsets, records, counts, wm, verts, W, row0, row1, info, redo,
                                                   guarded);
}

}  // namespace dtv
