// Plain structs and constants shared by host code and the sm_100a kernels.
#pragma once
#include <cstdint>
#include <climits>
#include <vector_types.h>

namespace dtv {

constexpr int kNumSubdivs = 4;             // Data/Shaders/Common/RayCommon.glsl:1-2
constexpr float kGuardPx = 1048576.0f;     // |screen coord| limit (2^20 px) for int64 edge functions
constexpr int32_t kInvalidFix = INT32_MIN; // marks a vertex outside [znear, zfar] or the guard band

// Camera constants, computed once on the host (see dtv_camera_constants).
struct CamDev {
    float V[16];    // view matrix, column-major
    float f;        // 0.5 * H / tan(fovy/2), rounded to FP32 (discrete path)
    float f_lo;     // its rounding error: f + f_lo carries the constant to ~2^-48 (continuous path)
    float cx, cy;   // 0.5 * W, 0.5 * H
    float znear, zfar;
    int W, H;
};

// Projection of a vertex for the continuous path (barycentrics, depth,
// adjoint), all FP32.  The screen position is split into the vertex's
// 1/256-pixel fixed-point position of the coverage rule (sx, sy: exact
// multiples of 1/256 px) and the residual of the exact projection against it
// (rx, ry, |r| <= ~1/512 px, from a compensated float-float projection).
// Pixel-centre differences of the snapped part are exact in FP32, so the
// edge functions of thin, nearly edge-on faces are formed from exact products
// plus small correction terms (face_interp).  1/ze, ze and the view-space
// x, y for the depth and the world-space adjoint.  32 bytes.
struct alignas(16) VGeo {
    float sx, sy;   // snapped position (px)
    float rx, ry;   // exact projected position - snapped position (px)
    float iz, ze, xv, yv;
};

// Per-view vertex row of the list walk, 32 bytes (one sector): what a step
// needs of a new vertex.
struct alignas(32) WalkVertRow {
    float4 pos;    // VGeo sx, sy (NaN when not projected); vproj x, y
    float2 depth;  // vproj 1 / ze, ze
    float2 pad;
};

// Walk tables of a mesh.  links[4 t + k] belongs to the face opposite tet t's
// local vertex k:
//   x  bits 0..27 the tet across the face (0x0fffffff: none), 28..29 the local
//      vertex that is the face's third stored vertex, 30 the face's bit of the
//      mesh's tet_flip, 31 whether the two tets' vertex orders wind the face
//      alike
//   y  face << 2 | boundary << 1 | whether the stored winding is odd against
//      the tet's own vertex order
//   z  the vertex of the tet across that is not on the face
//   w  byte l: the local index in the tet across of t's local vertex l, byte k
//      that of z
// and per boundary face k (vertices bfaces[k]) start[k] = its tet, that tet's
// vertex off the face, the local indices of the face's three vertices and of
// that one (a byte each), the face id.
struct WalkMesh {
    const uint4* links;
    const uint4* start;
    const uint4* bfaces;
};

// Per-render settings that the kernels read.
struct ShadeDev {
    float atten;
    float ert_thresh;   // terminate before a segment once T < ert_thresh
    int use_ert;
    int use_abs_grad;
    float clear[4];
};

}  // namespace dtv
