// Internal host-side declarations shared by the C-ABI layer and the kernel
// launch wrappers.  Not part of the public interface (include/difftetvr_b200.h).
#pragma once
#include <cstdint>
#include <string>
#include <vector>
#include <cuda_runtime.h>
#include "dtv_types.h"

namespace dtv {

// Face record on the device: three vertex indices (winding of the lowest
// faceId copy, TetMesh.cpp:1249-1252) and the boundary bit in .w.
struct MeshHost {
    uint64_t num_cells = 0, num_vertices = 0, num_faces = 0;
    std::vector<uint32_t> tri;            // 3F
    std::vector<uint32_t> face_boundary;  // F
    std::vector<uint32_t> face_to_tet;    // 2F
    std::vector<uint32_t> vertex_boundary;// V
    std::vector<uint32_t> cells;          // 4T
    std::vector<uint32_t> tet_faces;      // 4T: unique face index of face j of tet c (TetFaceTable order)
    // T: bit j set when face j's side seen from tet c is not given by the
    // winding of c's own vertex order (the shared face's stored winding, as
    // read with the owner rule, disagrees with c's order: inconsistently
    // oriented neighbours); 0 for a consistently oriented mesh.
    std::vector<uint8_t> tet_flip;
};

// Builds faces from cells (restates buildFacesSlim, TetMesh.cpp:1218-1268).
void build_faces(const uint32_t* cells, uint64_t T, uint64_t V, MeshHost& out);

// Split of the raster passes over few faces (a small mesh, or the boundary
// faces alone), which one thread (count) or 32 faces per warp (fill) would
// leave to a few warps, row after row.  Measured (us): count of 6^3 at 200^2
// (64-bit boxes) 49 -> 18, of 8^3 at 800^2 125 -> 36, of 16^3 at 1000^2 131 ->
// 55; fill of the boundary faces 12^3 at 600^2 904 -> 56, 8^3 at 64^2 53 -> 13,
// 64^3 at 1024^2 (10 -> 5 faces per warp) 96 -> 88.
// Count: threads per face (a power of two), each taking every so many rows.
inline uint32_t count_threads_per_face(uint64_t F) {
    uint32_t n = 1;
    while (n < 32 && F * n * 2 <= 148 * 2048) n *= 2;
    return n;
}
// Fill: faces that a warp takes one after another, and, with one face per warp
// and still few warps, the warps that share a face's groups of 32 rows (images
// of few rows have none to share).
struct FillSplit {
    uint32_t per_warp, parts;
};
inline FillSplit fill_split(uint64_t F, uint64_t image_rows) {
    if (F == 0) F = 1;
    uint64_t w = F / (148 * 64), p = 148 * 64 / F;
    if (p > 1 + image_rows / 128) p = 1 + image_rows / 128;
    return FillSplit{uint32_t(w < 1 ? 1 : (w > 32 ? 32 : w)), uint32_t(p < 1 ? 1 : (p > 16 ? 16 : p))};
}

// Whether boundary faces are so many (unconnected tets) that their fill in
// row-band order (launch_raster_fill) is worth ordering them: past 64 per warp
// slot of the GPU.  Boundary fill against fill in bands (us): 331 k faces at
// 512^2 495 and 527, at 1024^2 3,011 and 3,026; 786 k at 512^2 713 and 583, at
// 1024^2 3,798 and 3,388; 1.5 M at 1024^2 4,679 and 3,030.
inline bool many_boundary_faces(uint64_t F) { return F > 64 * 148 * 64; }

// Launch wrappers (dtv_kernels.cu).  All run on `s`.
// rows (optional): the vertices' walk rows as well; clipped (optional): set to
// 1 when a vertex is not projected; wide_list (optional): [0] cleared for the
// count.
void launch_project(const float* pos, uint32_t V, const CamDev& cam, float4* vproj, int2* vfix, VGeo* vgeo,
                    cudaStream_t s, WalkVertRow* rows = nullptr, uint32_t* clipped = nullptr,
                    uint32_t* wide_list = nullptr);
// Pixel rows [row0, row1) only (row1 < 0: all rows).  wide_list (u32[F + 1],
// optional, [0] zero: launch_project): the count lists the faces of the 64-bit path there, and the
// 64-bit count and the fill that follows (same rows) walk that list instead of
// setting up every face again; without it both 64-bit launches cover all F.
// rest (the fill): only pixels whose counter is not zero.
void launch_raster_count(const uint4* faces, uint32_t F, const float4* vproj, const int2* vfix, int W, int H,
                         uint32_t* counts, cudaStream_t s, int row0 = 0, int row1 = -1,
                         uint32_t* wide_list = nullptr);
void launch_raster_fill(const uint4* faces, uint32_t F, const float4* vproj, const int2* vfix, int W, int H,
                        uint32_t* counts, const unsigned long long* offsets, unsigned long long* records,
                        cudaStream_t s, int row0 = 0, int row1 = -1, const uint32_t* order = nullptr,
                        const uint32_t* wide_list = nullptr, bool rest = false);
// Fill of a few faces (the boundary's); nothing is done when *gate is zero.
void launch_boundary_fill(const uint4* faces, uint32_t F, const float4* vproj, const int2* vfix, int W, int row0,
                          int row1, uint32_t* counts, const unsigned long long* offsets, unsigned long long* records,
                          const uint32_t* gate, cudaStream_t s);
struct ListInfo;
// The few pixels the walk left to the rasteriser (nothing is done when there
// are none; many: launch_raster_fill with rest and launch_sort of the list):
// fill from all faces, sort of the listed pixels' lists.
void launch_rest_fill(const ListInfo* info, const uint4* faces, uint32_t F, const float4* vproj, const int2* vfix, int W,
                      int row0, int row1, uint32_t* counts, const unsigned long long* offsets,
                      unsigned long long* records, const uint32_t* redo, cudaStream_t s);
void launch_rest_sort(const ListInfo* info, const uint32_t* list, const unsigned long long* offsets,
                      unsigned long long* records, cudaStream_t s);
// Order of the faces for the fill, grouped by row bands of about
// kFillBandBytes of records each (nf records over H rows; order: F entries;
// band_scratch: 2 * kFillBands entries).
constexpr int kFillBands = 512;
constexpr uint64_t kFillBandBytes = 24ull << 20;
void launch_fill_order(const uint4* faces, uint32_t F, const int2* vfix, int H, uint64_t nf, uint32_t* order,
                       uint32_t* band_scratch, cudaStream_t s);
// Exclusive prefix of kFillBands band counts (one warp).
void launch_band_scan(const uint32_t* hist, uint32_t* cursor, cudaStream_t s);
// Exclusive scan of counts[n] into offsets[n+1]; scratch must hold scan_scratch_elems(n) u64.
constexpr uint64_t kScanTile = 4096;  // counts per scan block (1024 threads x 4)
constexpr size_t scan_scratch_elems(uint64_t n) { return size_t((n + kScanTile - 1) / kScanTile) + 1; }
// info (optional) gets the total, whether it is at most `capacity`, whether the
// projection clipped a vertex (*clipped, which is reset), and a zeroed redo
// counter.
struct ListInfo {
    unsigned long long nf;  // records of the lists
    uint32_t ok;            // they fit
    uint32_t clipped;
    uint32_t whole;         // ok and not clipped: the lists are walked
    uint32_t n_redo;        // pixels the walk left to the rasteriser
};
void launch_scan(const uint32_t* counts, uint64_t n, unsigned long long* offsets, unsigned long long* scratch,
                 cudaStream_t s, ListInfo* info = nullptr, unsigned long long capacity = ~0ull,
                 uint32_t* clipped = nullptr);
// Per-pixel sort of the lists of P pixels, any length.  scratch holds
// sort_scratch_elems(P) u32 (length-class counts and lists).  With a non-null
// `ok`, the sort does nothing when *ok == 0 (batched steps whose records
// overflowed the buffer).  list: only the *list_n listed pixels (at most P).
constexpr int kSortClasses = 9;  // list-length classes (dtv_kernels.cu)
constexpr size_t sort_scratch_elems(uint64_t P) { return 16 + size_t(kSortClasses) * size_t(P); }
// surrogate_classes: bit c set = list-length class c (1..4: up to 64, 128,
// 256, 512 records) is sorted through 32-bit surrogate keys, else through the
// 64-bit network (same result either way).
constexpr uint32_t kSortSurrogateDefault = 0x1eu;
constexpr uint32_t kSortBucketDefault = 0x3cu;  // classes sorted by distribution (bit c: class c, 2..5)
void launch_sort(const unsigned long long* offsets, unsigned long long* records, uint32_t P, uint32_t* scratch,
                 cudaStream_t s, const uint32_t* ok = nullptr,
                 uint32_t surrogate_classes = kSortSurrogateDefault, uint32_t bucket_classes = kSortBucketDefault,
                 const uint32_t* list = nullptr, const uint32_t* list_n = nullptr);
constexpr uint32_t kSortWarpCap = 1024;    // elements per warp list sorted in shared memory
constexpr uint32_t kSortBlockCap = 16384;  // elements per block-sorted list / chunk of a longer one (128 KiB shared memory)

// Whether the composite loads ahead (composite_pixel): a pixel's list is a chain
// of dependent loads, and running ahead of it is worth half the warps when the
// pixels do not fill the GPU with plain ones anyway, and later only while the
// vertices are too many to mostly hit L1.  pixels and V of one view, `all`
// pixels of the launch.  Measured (us, plain -> ahead): 64^3 at 128^2 583 ->
// 282, 16^3 at 256^2 75 -> 58, 33^3 at 721 x 479 330 -> 303, 64^3 at 512^2 586
// -> 517, at 1024^2 1,545 -> 1,526; 40^3 at 1000^2 850 -> 888, 16^3 at 1000^2
// 338 -> 362, 8^3 at 800^2 121 -> 129.
inline bool composite_ahead(uint64_t V, uint64_t pixels, uint64_t all) {
    if (all < 148 * 1280) return true;
    return pixels < (pixels < 148 * 2560 ? 64 : 6) * V;
}
// gate (optional): nothing is done when *gate is zero.
// tile: pixel tile of the 128-thread blocks (0: 16 x 8, 1: 32 x 4, 2: 8 x 16).
void launch_composite(const unsigned long long* offsets, const unsigned long long* records, const uint4* faces,
                      const VGeo* vgeo, const float4* colors, uint32_t V, int W, int H, const ShadeDev& sh,
                      float4* image, float* tfinal, uint32_t* term, cudaStream_t s, int row0 = 0, int row1 = -1, int tile = 0,
                      const uint32_t* gate = nullptr);
// Copies of the gradient rows of a mesh with few vertices (or cells): all
// pixels' atomics on a few thousand rows wait for one another in L2, so the
// blocks are spread over a power of two of copies with up to kGradRows rows in
// all, which the scatter sums.  One copy per 8192 pixels at most: a small image
// has no contention to spread, and clearing and summing 64 copies cost 12 us.
// Past kGradRowPixels pixels per row there is one copy: a row then gets so many
// terms that the rounding of its one long FP32 sum (relative to the gradient's
// norm 2e-6 at 200 pixels per vertex, 1.5e-5 to 2.9e-5 at 3,200) shows, and
// splitting it would move the values by that much; at 16 it moves them by less
// than another order of the atomics does (1e-6, 2e-6 at attenuation 100).
// Measured (us per step, one copy -> copies): 16^3 at 256^2 338 -> 321, a
// training step over 12 views of 12^3 to 36^3 at 384^2 4,308 -> 3,949.
constexpr uint64_t kGradRows = 1u << 17;
constexpr uint64_t kGradCopyPixels = 8192;
constexpr uint64_t kGradRowPixels = 16;
inline uint32_t grad_copies(uint64_t rows, uint64_t pixels) {
    uint32_t c = 1;
    if (pixels > kGradRowPixels * rows) return c;
    while (c < 64 && 2 * uint64_t(c) * rows <= kGradRows && 2 * uint64_t(c) * kGradCopyPixels <= pixels) c *= 2;
    return c;
}
// Adjoint of pixel rows [row0, row1) into the copies of grad_rows ([copies][V][2];
// no clearing, no scatter).
void launch_adjoint_rows(const unsigned long long* offsets, const unsigned long long* records, const uint4* faces,
                         const VGeo* vgeo, const float4* colors, const CamDev& cam, const ShadeDev& sh,
                         const float4* dimage, const float* tfinal, const uint32_t* term, int row0, int row1,
                         float4* grad_rows, uint32_t V, uint32_t copies, cudaStream_t s, int tile = 0);
// Adds the interleaved [V][2] gradient rows into grad_pos [V,3] / grad_col [V,4].
// screen_vgeo / cam: rows hold screen-space position adjoints of that camera
// (the list adjoint without absolute gradients); nullptr: world-space rows.
void launch_scatter_grads(const float4* grad_rows, uint32_t V, uint32_t copies, float* grad_pos, float4* grad_col, cudaStream_t s,
                          const VGeo* screen_vgeo = nullptr, const CamDev* cam = nullptr);

void launch_loss_l2(const float* image, const float* target, uint64_t n, float scale, float* adjoint,
                    float* loss_accum, cudaStream_t s);
void launch_adam(float* param, const float* grad, float* m, float* v, uint64_t n, float lr, float beta1,
                 float beta2, float eps, float bc1, float bc2, int clamp_mode, const uint32_t* fixed_mask,
                 int fixed_mode, int stride, cudaStream_t s);

// Per-cell colours (dtv_cells.cu): cell_colors f32[4T]; rows [row0, row1).
void launch_composite_cells(const unsigned long long* offsets, const unsigned long long* records, const uint4* faces,
                            const uint32_t* face_to_tet, const VGeo* vgeo, const float4* cell_colors, int W, int H,
                            const ShadeDev& sh, float4* image, float* tfinal, uint32_t* term, cudaStream_t s,
                            int row0, int row1, const uint32_t* gate = nullptr);
void launch_adjoint_cells_rows(const unsigned long long* offsets, const unsigned long long* records,
                               const uint4* faces, const uint32_t* face_to_tet, const VGeo* vgeo,
                               const float4* cell_colors, const CamDev& cam, const ShadeDev& sh, const float4* dimage,
                               const float* tfinal, const uint32_t* term, int row0, int row1, float4* grad_rows,
                               uint32_t V, uint32_t copies, float4* grad_cells, uint32_t T, uint32_t cell_copies,
                               cudaStream_t s);
// grad_cells[T] += the sum of the copies.
void launch_add_cell_copies(const float4* copies_base, uint32_t T, uint32_t copies, float4* grad_cells,
                            cudaStream_t s);
// Adds the position part of the [V][2] gradient rows into grad_pos [V,3]
// (vgeo non-null: the rows hold screen-space adjoints, converted per vertex
// with the render's camera, as the per-cell adjoint leaves them without
// absolute gradients).
void launch_scatter_positions(const float4* grad_rows, uint32_t V, uint32_t copies, float* grad_pos, cudaStream_t s,
                              const VGeo* vgeo = nullptr, const CamDev* cam = nullptr);

// Ray-tet path (dtv_raytet.cu).
void launch_walk_composite(const unsigned long long* b_offsets, const unsigned long long* b_records,
                           const uint32_t* bf_global, const uint4* faces, const uint32_t* face_to_tet,
                           const uint32_t* tet_faces, const uint32_t* cells, const uint8_t* tet_flip, const WalkMesh& wm,
                           uint32_t num_tets, const int2* vfix, const VGeo* vgeo,
                           const float4* colors, const CamDev& cam, const ShadeDev& sh, float4* image,
                           float* tfinal, uint4* wstate, cudaStream_t s);
void launch_walk_adjoint(const unsigned long long* b_offsets, const unsigned long long* b_records,
                         const uint32_t* bf_global, const uint4* faces, const uint32_t* face_to_tet,
                         const uint32_t* tet_faces, const uint32_t* cells, const uint8_t* tet_flip, const WalkMesh& wm,
                         uint32_t num_tets, const int2* vfix, const VGeo* vgeo,
                         const float4* colors, const CamDev& cam, const ShadeDev& sh, const float4* dimage,
                         const float* tfinal, const uint4* wstate, uint32_t V, float4* grad_rows, uint32_t copies, float* grad_pos,
                         float4* grad_col, cudaStream_t s);

// Fragment lists by walking the mesh (dtv_walk.cu).
// A mesh whose tets overlap (many inverted ones, as training without a
// regularizer leaves them) closes loops of faces over many pixels.  Past one
// pixel in kManyLeft the rasteriser's passes alone make the next kWalkRetry
// renders' lists (the same lists); the number is read back without a wait,
// after the lists.  Walk + rest against fill + sort (us), as training tangles the
// mesh: 64^3 / 1024^2 with 840 pixels left 1,906 against 3,300, 5,461 left 2,400
// against 3,340, 19,128 left 4,200 against 3,400; 32^3 / 512^2 with 800 left 540
// against 550, 1,600 left 670 against 555 (the whole step 1.57 ms either way).
constexpr uint64_t kManyLeft = 160;
constexpr int kWalkRetry = 64;
inline bool many_left(uint64_t left, uint64_t pixels) { return left > pixels / kManyLeft; }
// Whether the row bands of a render over its fragment budget are walked: a
// band of few pixels takes as long as its longest chain of steps (1.4 us each),
// while fill and sort of few records cost one pass over the faces.  Per list
// build, walk against fill + sort (us): lists of 97 records on average and bands
// of 580 pixels +33, of 9,200 -8; 151 records and 600 pixels +85, 9,200 +18,
// 37,000 -46; 193 records and 570 pixels +226, 3,100 +116, 9,200 -28, 12,300
// +32, 49,000 -46; 49 records and 640 pixels -11, 25 records -38.
inline bool walk_bands(uint64_t records, uint64_t pixels, uint64_t band_records) {
    return double(records) <= 64.0 * double(pixels) ||
           double(band_records) * double(pixels) >= 12288.0 * double(records);
}
// Fills the tables (links: 4 T, start: one per boundary face) from the device
// topology; *bad (device) is set to a non-zero value when the topology cannot
// be walked (a tet with a vertex twice, a face of more than two tets).
void launch_build_walk(const uint4* cells, uint32_t T, const uint4* tet_faces, const uint4* faces, const uint2* f2t,
                       const uint32_t* bf_global, uint32_t Nb, uint4* links, uint4* start, uint32_t* bad,
                       cudaStream_t s);
// Lists of pixel rows [row0, row1) from the boundary fragments at the end of
// each pixel's range.  Pixels it cannot finish are appended to `redo`
// (info->n_redo of them).  guarded: nothing is done when info->whole is zero.
void launch_walk_lists(const WalkMesh& wm, const unsigned long long* offsets, unsigned long long* records,
                       uint32_t* counts, const WalkVertRow* verts, int W, int row0, int row1, ListInfo* info,
                       uint32_t* redo, bool guarded, cudaStream_t s);

// Accessors used by the allocation-free entry point (dtv_noalloc.cu); they
// expose what dtv_renderer_render derives from its arguments.
struct MeshView {
    const uint4* faces;
    uint64_t num_faces;
    uint64_t num_vertices;
    WalkMesh walk;               // links null: the mesh cannot be walked
    uint32_t num_boundary_faces;
};

}  // namespace dtv

struct dtv_mesh;
struct dtv_camera;
struct dtv_render_params;

namespace dtv {
MeshView mesh_view(const dtv_mesh* m);
uint64_t mesh_num_cells(const dtv_mesh* m);
const uint32_t* mesh_cells_device(const dtv_mesh* m);  // u32[4T], 16-byte aligned
CamDev camera_constants(const dtv_camera& c);
ShadeDev shade_constants(const dtv_render_params& p);
}  // namespace dtv

// Sets the message returned by dtv_last_error_string() on this thread.
void dtv_set_last_error(const std::string& msg);
