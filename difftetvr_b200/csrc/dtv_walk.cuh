// Fragment lists by walking the mesh: each pixel's ray goes from tet to tet
// through face adjacency, and the faces it crosses come out in order, so no
// list is scattered by atomics and (nearly) none is sorted.  Shared by the
// single-view (dtv_walk.cu) and the batched kernels (dtv_batch.cu).
//
// Why the walk finds the rasteriser's lists.  The coverage rule decides on
// vertices snapped to 1/256 px and breaks ties as if the pixel centre were
// moved by (eps, eps^2), so it is the exact point-in-triangle test of one
// point against closed tets: of a tet's four projected faces either none or
// exactly two cover the pixel, one of each orientation.  The covering faces of
// a pixel therefore form chains from boundary face to boundary face (and, in
// meshes with inverted tets, possibly closed loops).  The walk follows every
// chain from its front-facing boundary face to its back-facing one and
// compares the number of faces it met with the rasteriser's count of the
// pixel: equal numbers mean equal sets.  Pixels where they differ (faces cut
// away by a clipping plane, loops, more chains than kWalkStarts, vertices
// beyond kWalkGuardPx) are listed and filled by the rasteriser and sorted.
// The depth keys, computed as the rasteriser computes them, are checked for
// strict order as they come; a face met out of order (faces at one depth up to
// rounding) is moved to its place.
#pragma once
#include "dtv_path.cuh"

namespace dtv {

constexpr int kWalkStarts = 8;          // chains of one pixel
constexpr float kWalkGuardPx = 32768.f; // snapped coordinates relative to a pixel centre are exact in FP32
constexpr uint32_t kWalkNoTet = 0x0fffffffu;

// Pixels whose list the rasteriser has to fill: how many, and which.
struct WalkRedo {
    uint32_t* n;
    uint32_t* list;
};

// The link entries of the next tet (64 bytes) into L1: which one is wanted is
// known only after the next face search.
__device__ __forceinline__ void prefetch_links(const uint4* p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p + 2));
}

// Four records (32-byte aligned).
__device__ __forceinline__ void store_sector(u64* p, u64 a, u64 b, u64 c, u64 d) {
    reinterpret_cast<ulonglong2*>(p)[0] = make_ulonglong2(a, b);
    reinterpret_cast<ulonglong2*>(p)[1] = make_ulonglong2(c, d);
}

// A vertex of the current face relative to the pixel centre (WalkVertRow):
// snapped position, and position, 1 / ze and ze of the depth key.
struct WalkVert {
    float sx, sy, px, py, iz, ze;
};

__device__ __forceinline__ WalkVert walk_vertex(uint32_t id, float qx, float qy,
                                                const WalkVertRow* __restrict__ verts) {
    const float4 q = verts[id].pos;
    const float2 z = verts[id].depth;
    return WalkVert{__fsub_rn(q.x, qx), __fsub_rn(q.y, qy), __fsub_rn(q.z, qx), __fsub_rn(q.w, qy), z.x, z.y};
}

// False for a vertex that is not projected (sx is NaN there) or so far off
// screen that its snapped position is not exact in FP32.
template <class V>
__device__ __forceinline__ bool walk_usable(const V& v) {
    return (fabsf(v.sx) < kWalkGuardPx) & (fabsf(v.sy) < kWalkGuardPx);
}

// Whether the pixel centre is on the inner side of the directed edge a -> b
// (edge_in on the exact value): the sign of the difference of products with
// the product's rounding error added back (Kahan) is the exact one.
template <class V>
__device__ __forceinline__ bool walk_side(const V& a, const V& b) {
    const float w = __fmul_rn(a.sy, b.sx);
    const float s = __fadd_rn(__fmaf_rn(a.sx, b.sy, -w), __fmaf_rn(-a.sy, b.sx, w));
    bool in = s > 0.f;
    if (s == 0.f) {
        const float dx = __fsub_rn(b.sx, a.sx), dy = __fsub_rn(b.sy, a.sy);
        in = dy < 0.f || (dy == 0.f && dx > 0.f);
    }
    return in;
}

// Edge function of the depth key (depth_key's operations; the reversed edge
// gives exactly the negative).
__device__ __forceinline__ float walk_key_cross(const WalkVert& a, const WalkVert& b) {
    return __fsub_rn(__fmul_rn(a.px, b.py), __fmul_rn(a.py, b.px));
}

// Depth key of the fragment on face (a, b, c) with edge functions K[0] = b x c,
// K[1] = c x a, K[2] = a x b: depth_key's value in any vertex order and
// orientation, since both sums change sign together and only the vertex that
// is summed last matters (t0, t1: a or b is the face's third stored vertex).
__device__ __forceinline__ uint32_t walk_key(const WalkVert& a, const WalkVert& b, const WalkVert& c,
                                             const float (&K)[3], bool t0, bool t1) {
    const float zmin = fminf(fminf(a.ze, b.ze), c.ze), zmax = fmaxf(fmaxf(a.ze, b.ze), c.ze);
    const float pa = __fmul_rn(K[0], a.iz), pb = __fmul_rn(K[1], b.iz), pc = __fmul_rn(K[2], c.iz);
    const float n0 = t0 ? pc : pa, n1 = t1 ? pc : pb, n2 = t0 ? pa : (t1 ? pb : pc);
    const float d0 = t0 ? K[2] : K[0], d1 = t1 ? K[2] : K[1], d2 = t0 ? K[0] : (t1 ? K[1] : K[2]);
    const float num = __fadd_rn(__fadd_rn(n0, n1), n2);
    const float den = __fadd_rn(__fadd_rn(d0, d1), d2);
    return __float_as_uint(fminf(fmaxf(__fdiv_rn(den, num), zmin), zmax));
}

// A thread's shared memory, entries `stride` apart: the pixel's chain starts
// and the records of the 32-byte sector being filled.
struct WalkSmem {
    u64* starts;   // [kWalkStarts]
    u64* recs;     // [4]
    int stride;
};

// The list of one pixel (n records at `out`, whose address is `phase` records
// past a 32-byte boundary).  The last nb records of the range are the pixel's
// boundary fragments (face field: boundary face index) when it starts.  False:
// the rasteriser has to fill the list.
__device__ __forceinline__ bool walk_list(float qx, float qy, u64* __restrict__ out, uint32_t phase, uint32_t n,
                                          uint32_t nb, const WalkMesh& wm, const WalkVertRow* __restrict__ verts,
                                          const WalkSmem& sm) {
    // Front-facing boundary fragments in order: the starts of the chains.
    int ns = 0;
    if (nb == 0) return false;
    for (uint32_t j = 0; j < nb; ++j) {
        const u64 r = out[n - nb + j];
        if (!(uint32_t(r) & 1u)) continue;
        if (ns == kWalkStarts) return false;
        int k = ns++;
        while (k > 0 && sm.starts[(k - 1) * sm.stride] > r) {
            sm.starts[k * sm.stride] = sm.starts[(k - 1) * sm.stride];
            --k;
        }
        sm.starts[k * sm.stride] = r;
    }
    uint32_t at = phase;  // phase + records so far
    const uint32_t end = phase + n;
    u64 newest = 0;
    for (int cs = 0; cs < ns; ++cs) {
        const uint32_t bk = uint32_t(sm.starts[cs * sm.stride]) >> 2;
        const uint4 bf = wm.bfaces[bk];
        const uint4 s0 = wm.start[bk];
        WalkVert a = walk_vertex(bf.x, qx, qy, verts), b = walk_vertex(bf.y, qx, qy, verts),
                 c = walk_vertex(bf.z, qx, qy, verts);
        if (!(walk_usable(a) & walk_usable(b) & walk_usable(c))) return false;
        uint32_t t = s0.x, dn = s0.y;
        // Local indices in t of the three slots' vertices and of the tet's
        // fourth one, one byte each.
        uint32_t loc = s0.z;
        // The vertices keep their slots until they are dropped, so the
        // directed edges of every face of the chain have the centre on the
        // side it has for the first one, a front face: the outer side.
        float K[3] = {walk_key_cross(b, c), walk_key_cross(c, a), walk_key_cross(a, b)};
        uint32_t key = walk_key(a, b, c, K, false, false);
        uint32_t bits = (s0.w << 2) | 3u;
        bool wound = true;   // the entry face is clockwise in the tet's own vertex order
        while (true) {
            // The tet's vertex off the entry face (after the chain's last face:
            // any one, unused).
            const WalkVert d = walk_vertex(dn, qx, qy, verts);
            const bool ended = t == kWalkNoTet;
            if (!ended) prefetch_links(wm.links + 4 * size_t(t));
            // The fragment into the list.
            if (at == end) return false;
            const u64 rec = (u64(key) << 32) | bits;
            const uint32_t q = at & 3u;
            u64* w = out + (int(at) - int(phase) - int(q));  // the sector's first record
            if (rec < newest) {
                // Met out of order (one depth up to rounding).
                uint32_t j = at;
                while (j > phase) {
                    const u64 r = ((j - 1) >> 2) == (at >> 2) ? sm.recs[int((j - 1) & 3u) * sm.stride]
                                                              : out[j - 1 - phase];
                    if (r < rec) break;
                    if ((j >> 2) == (at >> 2))
                        sm.recs[int(j & 3u) * sm.stride] = r;
                    else
                        out[j - phase] = r;
                    --j;
                }
                if ((j >> 2) == (at >> 2))
                    sm.recs[int(j & 3u) * sm.stride] = rec;
                else
                    out[j - phase] = rec;
            } else {
                sm.recs[int(q) * sm.stride] = rec;
                newest = rec;
            }
            if (q == 3u) {
                // A full sector of records (the first one of the list may be
                // shared with the pixel before).
                const u64 r0 = sm.recs[0], r1 = sm.recs[sm.stride], r2 = sm.recs[2 * sm.stride],
                          r3 = sm.recs[3 * sm.stride];
                if (at >= 3u + phase) {
                    store_sector(w, r0, r1, r2, r3);
                } else {
                    if (phase <= 1u) w[1] = r1;
                    if (phase <= 2u) w[2] = r2;
                    w[3] = r3;
                }
            }
            ++at;
            if (ended) break;
            if (!walk_usable(d)) return false;
            // The other face of the tet that covers the pixel: of (a, b, d),
            // (d, b, c) and (a, d, c) the one whose three directed edges all
            // have the centre on the outer side.
            const bool la = walk_side(a, d), lb = walk_side(b, d), lc = walk_side(c, d);
            const bool drop_c = la & !lb, drop_a = !drop_c & lb & !lc, drop_b = !drop_c & !drop_a;
            // Its link (the local index of the dropped vertex names it): the
            // tet across and flags, record bits, that tet's vertex off the
            // face, its local indices of this tet's vertices.
            const uint32_t k = (drop_a ? loc : (drop_b ? loc >> 8 : loc >> 16)) & 3u;
            const uint4 lk = wm.links[4 * size_t(t) + k];
            // Edge functions with the new vertex; the kept edge's stays.
            const float Ya = walk_key_cross(a, d), Yb = walk_key_cross(b, d), Yc = walk_key_cross(c, d);
            K[0] = drop_a ? K[0] : (drop_c ? Yb : -Yc);
            K[1] = drop_b ? K[1] : (drop_a ? Yc : -Ya);
            K[2] = drop_c ? K[2] : (drop_b ? Ya : -Yb);
            if (drop_a) a = d;
            if (drop_b) b = d;
            if (drop_c) c = d;
            dn = lk.z;
            loc = __byte_perm(loc, 0u, drop_a ? 0x4213u : (drop_b ? 0x4230u : 0x4310u));  // d takes the slot
            const uint32_t l3 = (lk.x >> 28) & 3u;
            key = walk_key(a, b, c, K, (loc & 255u) == l3, ((loc >> 8) & 255u) == l3);
            // The exit face has the other orientation in this tet's vertex order.
            const bool front = ((lk.y & 1u) != 0u) == wound;
            bits = (lk.y & ~1u) | (front ? 1u : 0u);
            // Local indices in the next tet (its own fourth vertex: byte k of w).
            const uint32_t sel = (loc & 0x3u) | ((loc >> 4) & 0x30u) | ((loc >> 8) & 0x300u) | (k << 12);
            loc = __byte_perm(lk.w, 0u, sel);
            t = lk.x & kWalkNoTet;
            wound = wound != ((lk.x >> 31) != 0u);
            // A chain between two front faces has another start as well.
            if (t == kWalkNoTet && front) return false;
        }
    }
    if (at != end) return false;
    // What is left of the last sector.
    for (uint32_t q = max(end & ~3u, phase); q < end; ++q) out[q - phase] = sm.recs[int(q & 3u) * sm.stride];
    return true;
}

// List of pixel p = (px, py) of an image whose arrays start at `offsets` and
// `counts` (redo_id: the pixel's index in the redo list).  `counts` holds what
// the boundary fill left of the pixel's count; it ends at zero, or at n for a
// pixel whose list the rasteriser has to fill.
__device__ __forceinline__ void walk_pixel(int px, int py, size_t p, const u64* __restrict__ offsets,
                                           u64* __restrict__ records, uint32_t* __restrict__ counts,
                                           const WalkMesh& wm, const WalkVertRow* __restrict__ verts,
                                           const WalkSmem& sm, const WalkRedo& redo, uint32_t redo_id) {
    const u64 beg = offsets[p];
    const uint32_t n = uint32_t(offsets[p + 1] - beg);
    if (n == 0) return;
    const bool ok = walk_list(float(px) + 0.5f, float(py) + 0.5f, records + beg, uint32_t(beg & 3u), n, n - counts[p],
                              wm, verts, sm);
    counts[p] = ok ? 0u : n;
    if (!ok) redo.list[atomicAdd(redo.n, 1u)] = redo_id;
}

}  // namespace dtv
