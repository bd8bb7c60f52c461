// Tet-quality regularizer gradient (the reference's TetRegularizerPass:
// Data/Shaders/Optimizer/TetRegularizer.glsl:108-166, dispatched by
// TetRegularizerPass.cpp:94 and bound as difftetvr.TetRegularizer,
// Module.cpp:663-695 / 983-995).
//
// Per tet with vertices p0..p3 (cell order):
//   D = det[p1 - p0, p2 - p0, p3 - p0]       (6 V = -D in the reference's sign)
//   S = sum of the six squared edge lengths   (l_rms^2 = S / 6)
//   q = 6 sqrt(2) V / l_rms^3 = -c D / S^(3/2),  c = 12 sqrt(3)   (Parthasarathy et al. 1991)
//   L = (lambda / beta) log(1 + exp(-beta q))    (mirrored softplus: low quality is penalised)
//   dL/dq = -lambda / (1 + exp(beta q))
//   dq/dp = (-c S dD/dp + 1.5 c D dS/dp) / max(S^(5/2), 1e-5)
// with dD/dp1 = (p2 - p0) x (p3 - p0), dD/dp2 = (p3 - p0) x (p1 - p0),
// dD/dp3 = (p1 - p0) x (p2 - p0), dD/dp0 = -(their sum), and
// dS/dpi = 2 (4 pi - sum_j pj).  The denominator clamp is the reference's
// (TetRegularizer.glsl:140-142); it is active for tets with S < 0.01.
// The gradient is added into the position gradient [3V]; the loss (a value
// the reference does not compute) is optionally accumulated.
#include "dtv_host.h"
#include "dtv_internal.h"
#include "difftetvr_b200.h"

namespace dtv {

constexpr float kRegC = 20.784609690826528f;  // 12 sqrt(3)

__device__ __forceinline__ float3 sub3(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 cross3(float3 a, float3 b) {
    return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float dot3(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

// grad[v] += g with two reductions: rows of three floats are 8-byte aligned at
// every second vertex, so (x, y), z or x, (y, z) (`pairs`: the base is 8-byte
// aligned).
__device__ __forceinline__ void add_row(float* grad, uint32_t v, float3 g, bool pairs) {
    float* r = grad + 3 * size_t(v);
    if (!pairs) {
        atomicAdd(r, g.x);
        atomicAdd(r + 1, g.y);
        atomicAdd(r + 2, g.z);
    } else {
        const bool odd = (v & 1u) != 0u;
        atomicAdd(reinterpret_cast<float2*>(r + (odd ? 1 : 0)), odd ? make_float2(g.y, g.z) : make_float2(g.x, g.y));
        atomicAdd(r + (odd ? 0 : 2), odd ? g.x : g.z);
    }
}

// Penalty gradient of one tet at its four vertices; returns q.
__device__ __forceinline__ float tet_penalty(const float3 (&p)[4], float lambda, float beta, float3 (&g)[4]) {
    const float3 e1 = sub3(p[1], p[0]), e2 = sub3(p[2], p[0]), e3 = sub3(p[3], p[0]);
    float3 dD[4];
    dD[1] = cross3(e2, e3);
    dD[2] = cross3(e3, e1);
    dD[3] = cross3(e1, e2);
    dD[0] = make_float3(-(dD[1].x + dD[2].x + dD[3].x), -(dD[1].y + dD[2].y + dD[3].y),
                        -(dD[1].z + dD[2].z + dD[3].z));
    const float D = dot3(dD[3], e3);
    const float3 e12 = sub3(p[2], p[1]), e13 = sub3(p[3], p[1]), e23 = sub3(p[3], p[2]);
    const float S = dot3(e1, e1) + dot3(e2, e2) + dot3(e3, e3) + dot3(e12, e12) + dot3(e13, e13) + dot3(e23, e23);
    const float s15 = S * sqrtf(S);
    const float q = -kRegC * D / s15;
    const float dLdq = -lambda / (1.f + expf(beta * q));
    const float den = fmaxf(S * s15, 1e-5f);
    const float a = -kRegC * S / den, b = 1.5f * kRegC * D / den;
    const float3 sum = make_float3(p[0].x + p[1].x + p[2].x + p[3].x, p[0].y + p[1].y + p[2].y + p[3].y,
                                   p[0].z + p[1].z + p[2].z + p[3].z);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float3 dS = make_float3(2.f * (4.f * p[j].x - sum.x), 2.f * (4.f * p[j].y - sum.y),
                                      2.f * (4.f * p[j].z - sum.z));
        g[j] = make_float3(dLdq * (a * dD[j].x + b * dS.x), dLdq * (a * dD[j].y + b * dS.y),
                           dLdq * (a * dD[j].z + b * dS.z));
    }
    return q;
}

// Each thread takes `run` consecutive tets.  Consecutive tets usually share
// vertices (the six tets of a split hexahedron use eight, and all hold its
// diagonal), so the gradients of the last tet's four vertices stay in
// registers and go out when a vertex is not in the next tet: 11 rows per
// hexahedron instead of 24.  The rows' reductions in L2 are what bounds the
// kernel; the losses are summed per block.
__global__ void __launch_bounds__(256) k_tet_regularizer(const uint4* __restrict__ cells, uint32_t T, uint32_t run,
                                                         const float* __restrict__ pos, float lambda, float beta,
                                                         float* __restrict__ grad, float* __restrict__ loss,
                                                         bool pairs) {
    constexpr uint32_t kNone = 0xffffffffu;
    __shared__ float sm[8];
    const uint64_t first = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) * run;
    uint32_t id[4] = {kNone, kNone, kNone, kNone};
    float3 acc[4] = {};
    float l = 0.f;
    const uint32_t n = first < T ? uint32_t(min(uint64_t(run), T - first)) : 0u;
    for (uint32_t k = 0; k < n; ++k) {
        const uint4 c = cells[first + k];
        const uint32_t vi[4] = {c.x, c.y, c.z, c.w};
        float3 p[4], g[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            p[j] = make_float3(pos[3 * size_t(vi[j])], pos[3 * size_t(vi[j]) + 1], pos[3 * size_t(vi[j]) + 2]);
        const float q = tet_penalty(p, lambda, beta, g);
        if (loss) {
            // (lambda / beta) softplus(-beta q), overflow-safe.
            const float z = -beta * q;
            l += (lambda / beta) * (fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))));
        }
        // Slots whose vertex this tet holds take its gradient; the others are
        // written out and given to the tet's vertices without one.
        uint32_t fresh = 15u;
        // A corner at an earlier corner's vertex (a tet may hold one twice) adds
        // to that corner: no two slots ever have one id, so every vertex of a
        // tet finds a slot.
        if ((vi[1] == vi[0]) | (vi[2] == vi[0]) | (vi[3] == vi[0]) | (vi[2] == vi[1]) | (vi[3] == vi[1]) |
            (vi[3] == vi[2])) {
#pragma unroll
            for (int j = 1; j < 4; ++j) {
#pragma unroll
                for (int i = 0; i < j; ++i) {
                    if (((fresh >> j) & 1u) && vi[i] == vi[j]) {
                        g[i] = make_float3(g[i].x + g[j].x, g[i].y + g[j].y, g[i].z + g[j].z);
                        g[j] = make_float3(0.f, 0.f, 0.f);
                        fresh &= ~(1u << j);
                    }
                }
            }
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            bool keep = false;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (id[s] == vi[j]) {
                    keep = true;
                    fresh &= ~(1u << j);
                    acc[s] = make_float3(acc[s].x + g[j].x, acc[s].y + g[j].y, acc[s].z + g[j].z);
                }
            }
            if (!keep) {
                if (id[s] != kNone) add_row(grad, id[s], acc[s], pairs);
                id[s] = kNone;
            }
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            if (id[s] == kNone && fresh) {
                const uint32_t j = uint32_t(__ffs(int(fresh))) - 1u;
                fresh &= fresh - 1u;
                id[s] = j == 0u ? vi[0] : (j == 1u ? vi[1] : (j == 2u ? vi[2] : vi[3]));
                acc[s] = j == 0u ? g[0] : (j == 1u ? g[1] : (j == 2u ? g[2] : g[3]));
            }
        }
    }
#pragma unroll
    for (int s = 0; s < 4; ++s)
        if (id[s] != kNone) add_row(grad, id[s], acc[s], pairs);
    if (loss) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = l;
        __syncthreads();
        if (threadIdx.x < 32) {
            l = threadIdx.x < 8 ? sm[threadIdx.x] : 0.f;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            if (threadIdx.x == 0 && l != 0.f) atomicAdd(loss, l);
        }
    }
}

}  // namespace dtv

extern "C" int32_t dtv_tet_regularizer_grad(const dtv_mesh* mesh, const float* d_positions, float lambda,
                                            float beta, float* d_grad_positions, float* d_loss, dtv_stream stream) {
    using namespace dtv_host;
    return guarded([&] {
        require(mesh != nullptr, "mesh is null");
        require(d_positions && d_grad_positions, "null device pointer");
        require(beta > 0.f, "softplus beta must be > 0");
        const uint64_t T = dtv::mesh_num_cells(mesh);
        if (T == 0) return;
        // Up to six tets per thread (a split hexahedron's) while that leaves
        // 1024 threads per SM (64^3, us without the loss: 52.6, 37.9, 33.2 and
        // 39.5 with 1, 2, 6 and 12; 40^3: 18.5, 14.2 and 16.8 with 1, 2 and 5).
        const uint32_t run = uint32_t(T / (148 * 1024) < 1 ? 1 : (T / (148 * 1024) > 6 ? 6 : T / (148 * 1024)));
        const uint64_t threads = (T + run - 1) / run;
        dtv::k_tet_regularizer<<<unsigned((threads + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
            reinterpret_cast<const uint4*>(dtv::mesh_cells_device(mesh)), uint32_t(T), run, d_positions, lambda, beta,
            d_grad_positions, d_loss, (reinterpret_cast<uintptr_t>(d_grad_positions) & 7u) == 0);
        check_launch("tet regularizer");
    });
}
