// wc_surface.cu — surface extraction from the particles: a colour field on a vertex grid and
// marching cubes over it (no counterpart in the reference, which draws the particles as
// points; surface reconstruction is its report's stated future work).
//
//   field      phi(v) = sum_j (m / rho0) W_poly6(|v - x_j|, h) over the particles of the 27 cells
//              around vertex v (the solver's sorted buffer and cell tables), about 1 inside the
//              fluid and 0 outside; every float operation is an explicit round-to-nearest one,
//              summed in the cell-row order of the tables, so the result is reproducible exactly
//   classify   per cube: corner bits (phi > iso), triangle count from the case table
//   scan       the decoupled look-back scan of the solver over the per-cube counts
//   emit       per cube: its triangles, each vertex interpolated on a cube edge whose
//              endpoints are taken in ascending order (neighbouring cubes produce the same
//              float coordinates, so the mesh is watertight)
//
// The case table is generated here, not typed in: for each of the 256 corner configurations
// the iso-segments of the six faces are walked (on a face with two diagonal inside corners the
// segments separate the inside corners; the decision depends only on the face, so both cubes
// sharing it agree), chained into closed loops, oriented so that the normal (Newell's method)
// points from the inside corners to the outside ones, and triangulated as fans.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <type_traits>
#include <vector>

#include "wc_internal.h"
#include "wc_util.h"

using namespace wc;

namespace {

constexpr int MAX_TRI = 12;  // per cube (a configuration yields at most 10)

// Corner c sits at offset (c & 1, (c >> 1) & 1, (c >> 2) & 1). Edge e joins corners
// EDGE_A[e] < EDGE_B[e], which differ in the bit of axis e / 4.
constexpr int EDGE_A[12] = {0, 2, 4, 6, 0, 1, 4, 5, 0, 1, 2, 3};
constexpr int EDGE_B[12] = {1, 3, 5, 7, 2, 3, 6, 7, 4, 5, 6, 7};

struct CaseTable {
    uint8_t count[256];
    int8_t tri[256][MAX_TRI * 3];
};

int edge_of(int a, int b) {
    if (a > b) std::swap(a, b);
    for (int e = 0; e < 12; ++e)
        if (EDGE_A[e] == a && EDGE_B[e] == b) return e;
    return -1;
}

void corner_pos(int c, double p[3]) {
    p[0] = c & 1;
    p[1] = (c >> 1) & 1;
    p[2] = (c >> 2) & 1;
}

// One configuration's triangles (edge triples).
void build_case(int cfg, std::vector<int>& tris) {
    tris.clear();
    auto inside = [&](int c) { return (cfg >> c) & 1; };
    std::vector<std::pair<int, int>> segs;  // undirected, between crossing edges
    for (int a = 0; a < 3; ++a) {
        const int u = (a + 1) % 3, v = (a + 2) % 3;
        for (int s = 0; s < 2; ++s) {
            // the face's corners in cyclic order (u, v) = (0,0), (1,0), (1,1), (0,1)
            int cyc[4];
            const int uv[4][2] = {{0, 0}, {1, 0}, {1, 1}, {0, 1}};
            for (int k = 0; k < 4; ++k) cyc[k] = (s << a) | (uv[k][0] << u) | (uv[k][1] << v);
            int fe[4];
            bool cross[4];
            int ncross = 0;
            for (int k = 0; k < 4; ++k) {
                fe[k] = edge_of(cyc[k], cyc[(k + 1) & 3]);
                cross[k] = inside(cyc[k]) != inside(cyc[(k + 1) & 3]);
                ncross += cross[k];
            }
            if (ncross == 2) {
                int e0 = -1, e1 = -1;
                for (int k = 0; k < 4; ++k)
                    if (cross[k]) (e0 < 0 ? e0 : e1) = fe[k];
                segs.push_back({e0, e1});
            } else if (ncross == 4) {
                // two diagonal inside corners: cut each off on its own
                for (int k = 0; k < 4; ++k)
                    if (inside(cyc[k])) segs.push_back({fe[(k + 3) & 3], fe[k]});
            }
        }
    }
    // chain into loops (every crossing edge has exactly two segments)
    std::vector<bool> used(segs.size(), false);
    for (size_t first = 0; first < segs.size(); ++first) {
        if (used[first]) continue;
        std::vector<int> loop;
        used[first] = true;
        const int start = segs[first].first;
        int cur = segs[first].second;
        loop.push_back(start);
        while (cur != start) {
            loop.push_back(cur);
            bool found = false;
            for (size_t i = 0; i < segs.size(); ++i) {
                if (used[i]) continue;
                if (segs[i].first == cur || segs[i].second == cur) {
                    used[i] = true;
                    cur = segs[i].first == cur ? segs[i].second : segs[i].first;
                    found = true;
                    break;
                }
            }
            if (!found) break;  // cannot happen for a closed surface
        }
        // orientation: Newell normal of the loop (edge midpoints) against inside -> outside
        double nrm[3] = {0, 0, 0}, din[3] = {0, 0, 0}, dout[3] = {0, 0, 0};
        const size_t L = loop.size();
        std::vector<std::array<double, 3>> pts(L);
        for (size_t i = 0; i < L; ++i) {
            double pa[3], pb[3];
            corner_pos(EDGE_A[loop[i]], pa);
            corner_pos(EDGE_B[loop[i]], pb);
            for (int k = 0; k < 3; ++k) pts[i][k] = 0.5 * (pa[k] + pb[k]);
            const bool ain = inside(EDGE_A[loop[i]]);
            for (int k = 0; k < 3; ++k) {
                din[k] += ain ? pa[k] : pb[k];
                dout[k] += ain ? pb[k] : pa[k];
            }
        }
        for (size_t i = 0; i < L; ++i) {
            const auto& p = pts[i];
            const auto& q = pts[(i + 1) % L];
            nrm[0] += (p[1] - q[1]) * (p[2] + q[2]);
            nrm[1] += (p[2] - q[2]) * (p[0] + q[0]);
            nrm[2] += (p[0] - q[0]) * (p[1] + q[1]);
        }
        const double dot = nrm[0] * (dout[0] - din[0]) + nrm[1] * (dout[1] - din[1]) + nrm[2] * (dout[2] - din[2]);
        if (dot < 0) std::reverse(loop.begin() + 1, loop.end());
        for (size_t i = 1; i + 1 < L; ++i) {
            tris.push_back(loop[0]);
            tris.push_back(loop[i]);
            tris.push_back(loop[i + 1]);
        }
    }
}

const CaseTable& case_table() {
    static CaseTable t;
    static std::once_flag once;
    std::call_once(once, [] {
        std::memset(&t, 0, sizeof t);
        std::memset(t.tri, -1, sizeof t.tri);
        std::vector<int> tris;
        for (int cfg = 0; cfg < 256; ++cfg) {
            build_case(cfg, tris);
            const int nt = (int)tris.size() / 3;
            t.count[cfg] = (uint8_t)(nt > MAX_TRI ? MAX_TRI : nt);
            for (int i = 0; i < t.count[cfg] * 3; ++i) t.tri[cfg][i] = (int8_t)tris[i];
        }
    });
    return t;
}

__constant__ uint8_t c_count[256];
__constant__ int8_t c_tri[256][MAX_TRI * 3];
__constant__ int8_t c_edge_a[12];
__constant__ int8_t c_edge_b[12];

struct Grid {
    uint32_t G;     // vertices per axis
    float spacing;  // size / (G - 1)
};

__device__ __forceinline__ float vcoord(uint32_t i, float spacing) { return __fmul_rn((float)i, spacing); }

// ---- packed f32x2 arithmetic (two floats in one 64-bit register, each operation rounded on its own) ----
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1,%2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk(f2 v, float& a, float& b) { asm("mov.b64 {%0,%1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// a * b rounded on its own: the assembler contracts a packed multiply, or a fused one with a constant
// zero, with the addition that follows, so this is a fused operation with a -0 it does not know.
__device__ __forceinline__ f2 mul2_alone(f2 a, f2 b, f2 minus_zero) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(minus_zero));
    return d;
}

// phi at every vertex (x fastest). One thread per vertex; a warp takes 4 x 4 x 2 of them and a block
// 8 x 8 x 4, so that its lanes lie in a cell or two and walk nearly the same candidates, four at a time
// from the lane passes' slots (padding lies far away and adds zero, and so do the places of a load outside a packed
// row; the weights are added in candidate order). Bound by the L1's data path: the lanes of a load lie in up to eight cells. 128^3
// vertices over 262,144 particles: 154 us with 32 x 1 x 1 vertices per warp and one candidate per load,
// 79 us in blocks, 65 us with the air left out block by block.
__global__ void __launch_bounds__(256) field_kernel(Grid g, const float* __restrict__ xyz, uint32_t pcap, uint32_t n,
                                                    uint32_t num_cells, const uint32_t* __restrict__ start,
                                                    const uint32_t* __restrict__ pstart, float bin, int32_t R, float h2,
                                                    float scale, float minus_zero, float* __restrict__ phi,
                                                    uint32_t* __restrict__ err) {
    const bool packed_slots = __ldg(pstart + num_cells) > pcap;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t ix = blockIdx.x * 8u + (warp & 1u) * 4u + (lane & 3u);
    const uint32_t iy = blockIdx.y * 8u + ((warp >> 1) & 1u) * 4u + ((lane >> 2) & 3u);
    const uint32_t iz = blockIdx.z * 4u + (warp >> 2) * 2u + (lane >> 4);
    auto cell = [&](float q) {
        const float f = __fdiv_rn(q, bin);
        int c = f >= 1.0f ? (int)f : 0;
        return c > R - 1 ? R - 1 : c;
    };
    // the cells around the block's vertices, one row of them per thread: air is left at once
    const uint32_t b0[3] = {blockIdx.x * 8u, blockIdx.y * 8u, blockIdx.z * 4u};
    int c0[3], c1[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        c0[a] = max(cell(vcoord(b0[a], g.spacing)) - 1, 0);
        c1[a] = min(cell(vcoord(min(b0[a] + (a < 2 ? 7u : 3u), g.G - 1u), g.spacing)) + 1, R - 1);
    }
    const uint32_t ny = (uint32_t)(c1[1] - c0[1] + 1), rows = ny * (uint32_t)(c1[2] - c0[2] + 1);
    if (rows <= 256u) {
        bool any = false;
        if (threadIdx.x < rows) {
            const uint32_t row = (((uint32_t)c0[2] + threadIdx.x / ny) * R + (uint32_t)c0[1] + threadIdx.x % ny) * R;
            any = __ldg(pstart + row + c0[0]) != __ldg(pstart + row + c1[0] + 1);
        }
        if (!__syncthreads_or(any)) {
            if (ix < g.G && iy < g.G && iz < g.G) phi[(iz * g.G + iy) * g.G + ix] = __fmul_rn(0.f, scale);
            return;
        }
    }
    if (ix >= g.G || iy >= g.G || iz >= g.G) return;
    const float px = vcoord(ix, g.spacing), py = vcoord(iy, g.spacing), pz = vcoord(iz, g.spacing);
    const int cx = cell(px), cy = cell(py), cz = cell(pz);
    const int x0 = cx > 0 ? cx - 1 : 0, x1 = cx + 1 < R ? cx + 1 : R - 1;
    const float* const X = xyz;
    const float* const Y = xyz + pcap;
    const float* const Z = xyz + 2 * (size_t)pcap;
    const f2 vx = pk(px, px), vy = pk(py, py), vz = pk(pz, pz), hh = pk(h2, h2), nz = pk(minus_zero, minus_zero);
    float acc = 0.f;
    auto walk = [&](auto layout) {
        constexpr bool packed = decltype(layout)::value;
        const uint32_t* const tab = packed ? start : pstart;
#pragma unroll(packed ? 1 : 9)
        for (int r = 0; r < 9; ++r) {
            const int y = cy + r % 3 - 1, z = cz + r / 3 - 1;
            if (y < 0 || y >= R || z < 0 || z >= R) continue;
            const uint32_t row = (uint32_t)((z * R + y) * R);
            // a timed-out scan (reported) leaves inconsistent tables: keep the range in the buffers
            const uint32_t hi = packed ? min(__ldg(tab + row + x1 + 1), n) : min(__ldg(tab + row + x1 + 1), pcap) & ~3u;
            const uint32_t lo = min(packed ? __ldg(tab + row + x0) : __ldg(tab + row + x0) & ~3u, hi);
            if (hi - lo > 3u * MAX_CELL_PARTICLES) {
                const uint32_t e = min(__ldg(start + row + x1 + 1), n);
                if (e - min(__ldg(start + row + x0), e) > 3u * MAX_CELL_PARTICLES) {  // a collapsed state: not evaluated
                    acc = __int_as_float(0x7fc00000);
                    atomicOr(err, DEVERR_CELL_OVERFLOW);
                    continue;
                }
            }
            for (uint32_t k = packed ? lo & ~3u : lo; k < hi; k += 4u) {
                const ulonglong2 qx = *reinterpret_cast<const ulonglong2*>(X + k);
                const ulonglong2 qy = *reinterpret_cast<const ulonglong2*>(Y + k);
                const ulonglong2 qz = *reinterpret_cast<const ulonglong2*>(Z + k);
                const f2 dx01 = sub2(vx, qx.x), dx23 = sub2(vx, qx.y);
                const f2 dy01 = sub2(vy, qy.x), dy23 = sub2(vy, qy.y);
                const f2 dz01 = sub2(vz, qz.x), dz23 = sub2(vz, qz.y);
                // t = h2 - d2 > 0 exactly when d2 < h2; zero (or not a number, as the comparison has it)
                // otherwise adds zero
                float t0, t1, t2, t3, w0, w1, w2, w3;
                upk(sub2(hh, add2(add2(mul2_alone(dx01, dx01, nz), mul2_alone(dy01, dy01, nz)), mul2_alone(dz01, dz01, nz))), t0, t1);
                upk(sub2(hh, add2(add2(mul2_alone(dx23, dx23, nz), mul2_alone(dy23, dy23, nz)), mul2_alone(dz23, dz23, nz))), t2, t3);
                if (packed) {
                    const uint32_t at = k - lo, len = hi - lo;
                    t0 = at < len ? t0 : 0.f;
                    t1 = at + 1u < len ? t1 : 0.f;
                    t2 = at + 2u < len ? t2 : 0.f;
                    t3 = at + 3u < len ? t3 : 0.f;
                }
                const f2 t01 = pk(fmaxf(t0, 0.f), fmaxf(t1, 0.f)), t23 = pk(fmaxf(t2, 0.f), fmaxf(t3, 0.f));
                upk(mul2_alone(mul2(t01, t01), t01, nz), w0, w1);
                upk(mul2_alone(mul2(t23, t23), t23, nz), w2, w3);
                acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, w0), w1), w2), w3);
            }
        }
    };
    if (packed_slots) walk(std::true_type{});
    else walk(std::false_type{});
    phi[(iz * g.G + iy) * g.G + ix] = __fmul_rn(acc, scale);
}

__device__ __forceinline__ uint32_t cube_config(const float* __restrict__ phi, uint32_t G, uint32_t ix, uint32_t iy,
                                                uint32_t iz, float iso) {
    uint32_t cfg = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const uint64_t idx = ((uint64_t)(iz + ((c >> 2) & 1)) * G + (iy + ((c >> 1) & 1))) * G + (ix + (c & 1));
        cfg |= (phi[idx] > iso ? 1u : 0u) << c;
    }
    return cfg;
}

__global__ void classify_kernel(uint32_t G, const float* __restrict__ phi, float iso, uint32_t* __restrict__ counts) {
    const uint32_t C = G - 1;
    const uint64_t cubes = (uint64_t)C * C * C;
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < cubes; q += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t ix = (uint32_t)(q % C), iy = (uint32_t)((q / C) % C), iz = (uint32_t)(q / ((uint64_t)C * C));
        counts[q] = c_count[cube_config(phi, G, ix, iy, iz, iso)];
    }
}

// The triangles of the scan's list of non-empty cubes (most cubes have none: 2.0 million cubes took 26 us). It is
// launched before the host has read the error word, so it looks itself: after a failed field or scan (whose list may
// have holes) it writes nothing, and the mesh of the extraction before stays whole.
__global__ void emit_kernel(Grid g, const float* __restrict__ phi, float iso, const uint32_t* __restrict__ offsets,
                            const uint32_t* __restrict__ list, const uint32_t* __restrict__ list_len,
                            const uint32_t* __restrict__ err, uint64_t max_tris, float* __restrict__ out) {
    if (*err) return;
    const uint32_t G = g.G, C = G - 1, cubes = C * C * C, len = min(*list_len, cubes);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < len; i += gridDim.x * blockDim.x) {
        const uint32_t q = list[i];
        if (q >= cubes) continue;
        const uint32_t ix = q % C, iy = (q / C) % C, iz = q / (C * C);
        const uint32_t cfg = cube_config(phi, G, ix, iy, iz, iso);
        const uint32_t nt = c_count[cfg];
        if (!nt) continue;
        const uint64_t base = offsets[q];
        for (uint32_t t = 0; t < nt; ++t) {
            if (base + t >= max_tris) return;  // more than the buffer holds: the host grows it and calls again
            float* o = out + (base + t) * 9u;
            for (int k = 0; k < 3; ++k) {
                const int e = c_tri[cfg][3 * t + k];
                const int a = c_edge_a[e], b = c_edge_b[e];
                const uint32_t ax = ix + (a & 1), ay = iy + ((a >> 1) & 1), az = iz + ((a >> 2) & 1);
                const uint32_t bx = ix + (b & 1), by = iy + ((b >> 1) & 1), bz = iz + ((b >> 2) & 1);
                const float fa = phi[((uint64_t)az * G + ay) * G + ax];
                const float fb = phi[((uint64_t)bz * G + by) * G + bx];
                const float s = __fdiv_rn(__fsub_rn(iso, fa), __fsub_rn(fb, fa));
                const float pa[3] = {vcoord(ax, g.spacing), vcoord(ay, g.spacing), vcoord(az, g.spacing)};
                const float pb[3] = {vcoord(bx, g.spacing), vcoord(by, g.spacing), vcoord(bz, g.spacing)};
#pragma unroll
                for (int d = 0; d < 3; ++d) o[3 * k + d] = __fadd_rn(pa[d], __fmul_rn(s, __fsub_rn(pb[d], pa[d])));
            }
        }
    }
}

template <class T>
wc_status dalloc(T** p, size_t count) {
    *p = nullptr;
    if (!count) return WC_OK;
    WC_TRY(::wc::device_alloc(reinterpret_cast<void**>(p), count * sizeof(T)));
    return WC_OK;
}

}  // namespace

struct wc_surface {
    wc_surface_params p{};
    uint32_t G = 0;
    float* phi = nullptr;
    uint32_t *counts = nullptr, *offsets = nullptr, *cell_list = nullptr, *words = nullptr, *err = nullptr;
    unsigned long long* desc = nullptr;
    float* tris = nullptr;
    uint64_t tri_cap = 0, ntris = 0;
    float spacing = 0.f, iso = 0.f;
    bool have = false;
    uint32_t* h_words = nullptr;  // pinned: triangles, error word
    cudaStream_t stream = nullptr;
    float ms_field = 0.f, ms_mesh = 0.f;
};

namespace {

wc_status upload_tables() {
    static std::once_flag once;
    static cudaError_t rc = cudaSuccess;
    std::call_once(once, [] {
        const CaseTable& t = case_table();
        int8_t ea[12], eb[12];
        for (int e = 0; e < 12; ++e) {
            ea[e] = (int8_t)EDGE_A[e];
            eb[e] = (int8_t)EDGE_B[e];
        }
        rc = cudaMemcpyToSymbol(c_count, t.count, sizeof t.count);
        if (rc == cudaSuccess) rc = cudaMemcpyToSymbol(c_tri, t.tri, sizeof t.tri);
        if (rc == cudaSuccess) rc = cudaMemcpyToSymbol(c_edge_a, ea, sizeof ea);
        if (rc == cudaSuccess) rc = cudaMemcpyToSymbol(c_edge_b, eb, sizeof eb);
    });
    if (rc != cudaSuccess) return fail(WC_ERR_CUDA, "surface tables: %s", cudaGetErrorString(rc));
    return WC_OK;
}

unsigned grid_blocks(uint64_t work) {
    const uint64_t b = (work + 255) / 256;
    return (unsigned)(b > 152ull * 64 ? 152ull * 64 : (b ? b : 1));
}

}  // namespace

extern "C" {

WC_API wc_status wc_surface_case_table(uint8_t* counts, int8_t* tris) {
    clear_error();
    if (!counts || !tris) return fail(WC_ERR_INVALID_ARG, "null argument");
    const CaseTable& t = case_table();
    std::memcpy(counts, t.count, sizeof t.count);
    std::memcpy(tris, t.tri, sizeof t.tri);
    return WC_OK;
}

WC_API wc_status wc_surface_create(const wc_surface_params* p, wc_surface** out) {
    clear_error();
    if (!p || !out) return fail(WC_ERR_INVALID_ARG, "null argument");
    if (p->grid_res < 2 || p->grid_res > 1024) return fail(WC_ERR_INVALID_ARG, "grid_res must be in 2..1024");
    wc_surface* s = new (std::nothrow) wc_surface();
    if (!s) return fail(WC_ERR_OOM, "host allocation failed");
    s->p = *p;
    s->G = p->grid_res;
    const uint64_t V = (uint64_t)s->G * s->G * s->G;
    const uint64_t C = (uint64_t)(s->G - 1) * (s->G - 1) * (s->G - 1);
    wc_status st = upload_tables();
    if (st == WC_OK && C > 0xffffffffull) st = fail(WC_ERR_INVALID_ARG, "too many cubes");
    if (st == WC_OK && cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess)
        st = fail(WC_ERR_CUDA, "stream creation failed");
    const uint64_t tiles = (C + SCAN_TILE - 1) / SCAN_TILE;
    if (st == WC_OK) st = dalloc(&s->phi, V);
    if (st == WC_OK) st = dalloc(&s->counts, C);
    if (st == WC_OK) st = dalloc(&s->offsets, C + 1);
    if (st == WC_OK) st = dalloc(&s->cell_list, C);
    if (st == WC_OK) st = dalloc(&s->words, 2);
    if (st == WC_OK) st = dalloc(&s->err, 1);
    if (st == WC_OK) st = dalloc(&s->desc, tiles ? tiles : 1);
    // room for 8 G^2 triangles from the start (a splashing scene's surface has about half of that): a first extraction
    // that found none waited for its count, an allocation and a second pass, 270 us instead of 145 at 60^3 vertices
    const uint64_t tri_cap = 8ull * s->G * s->G;
    if (st == WC_OK) st = dalloc(&s->tris, tri_cap * 9u);
    if (st == WC_OK) s->tri_cap = tri_cap;
    if (st == WC_OK && cudaMallocHost(reinterpret_cast<void**>(&s->h_words), 2 * sizeof(uint32_t)) != cudaSuccess)
        st = fail(WC_ERR_OOM, "pinned host allocation failed");
    if (st == WC_OK && cudaMemset(s->err, 0, sizeof(uint32_t)) != cudaSuccess) st = fail(WC_ERR_CUDA, "memset");
    if (st != WC_OK) {
        wc_surface_destroy(s);
        return st;
    }
    *out = s;
    return WC_OK;
}

WC_API void wc_surface_destroy(wc_surface* s) {
    if (!s) return;
    if (s->stream) cudaStreamSynchronize(s->stream);
    void* ptrs[] = {s->phi, s->counts, s->offsets, s->cell_list, s->words, s->err, s->desc, s->tris};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (s->h_words) cudaFreeHost(s->h_words);
    if (s->stream) cudaStreamDestroy(s->stream);
    delete s;
}

WC_API wc_status wc_surface_extract(wc_surface* s, wc_fluid* f, uint64_t* num_triangles) {
    clear_error();
    WC_NVTX("wc_surface_extract");
    if (!s || !f) return fail(WC_ERR_INVALID_ARG, "null argument");
    FluidInternals fi = fluid_internals(f);
    const DevBuffers& d = *fi.d;
    const SceneConsts& sc = *fi.sc;
    const float radius = s->p.radius > 0.f ? s->p.radius : sc.h;
    if (radius > sc.bin) return fail(WC_ERR_INVALID_ARG, "field radius %g exceeds the cell edge %g", radius, sc.bin);
    const uint32_t G = s->G, C = G - 1;
    const uint64_t cubes = (uint64_t)C * C * C;
    Grid g{G, sc.size / (float)(G - 1)};
    s->spacing = g.spacing;
    s->iso = s->p.iso;
    const float h2 = radius * radius;
    // m / rho0 * 315 / (64 pi r^9), the Poly6 normalisation for the field radius (r^9 by
    // repeated double multiplication, reproducible everywhere)
    const double r1 = radius, r2 = r1 * r1, r4 = r2 * r2, r8 = r4 * r4;
    const double c6 = 315.0 / (64.0 * M_PI * (r8 * r1));
    const float scale = (float)((double)sc.m / (double)sc.rho0 * c6);
    // sort the fluid's state (its cell tables then describe the sorted buffer), with the lane passes'
    // padded slots whatever its own pass variant
    WC_CUDA_TRY(cudaStreamSynchronize(s->stream));
    fluid_enqueue_sort(f, PASSES_LANE);
    cudaEvent_t e0, e1, e2;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventCreate(&e2);
    cudaEventRecord(e0, fi.stream);
    field_kernel<<<dim3((G + 7) / 8, (G + 7) / 8, (G + 3) / 4), 256, 0, fi.stream>>>(
        g, d.xyz, d.pcap, d.n, d.num_cells, d.start, d.pstart, sc.bin, sc.R, h2, scale, -0.0f, s->phi, s->err);
    cudaEventRecord(e1, fi.stream);
    classify_kernel<<<grid_blocks(cubes), 256, 0, fi.stream>>>(G, s->phi, s->p.iso, s->counts);
    DevBuffers sd{};
    sd.n = 0;
    sd.num_cells = (uint32_t)cubes;
    sd.num_tiles = (uint32_t)((cubes + SCAN_TILE - 1) / SCAN_TILE);
    sd.counts = s->counts;
    sd.start = s->offsets;
    sd.cell_list = s->cell_list;
    sd.num_nonempty = s->words + 1;
    sd.scan_desc = s->desc;
    sd.scan_tile_counter = s->words;
    sd.err = s->err;
    wc_status st = WC_OK;
    cudaError_t ce = cudaMemsetAsync(s->desc, 0, sizeof(unsigned long long) * (sd.num_tiles ? sd.num_tiles : 1), fi.stream);
    if (ce == cudaSuccess) ce = cudaMemsetAsync(s->words, 0, 2 * sizeof(uint32_t), fi.stream);
    launch_scan_cells(sd, fi.stream);
    // the triangles go out with the scan, into what the buffer holds; only a larger surface than any
    // before waits for its count, a larger buffer and a second call
    auto emit = [&] {
        if (s->tri_cap)
            emit_kernel<<<grid_blocks(std::min<uint64_t>(cubes, 152ull * 8 * 256)), 256, 0, fi.stream>>>(
                g, s->phi, s->p.iso, s->offsets, s->cell_list, s->words + 1, s->err, s->tri_cap, s->tris);
    };
    emit();
    cudaEventRecord(e2, fi.stream);
    if (ce == cudaSuccess)
        ce = cudaMemcpyAsync(s->h_words, s->offsets + cubes, sizeof(uint32_t), cudaMemcpyDeviceToHost, fi.stream);
    if (ce == cudaSuccess)
        ce = cudaMemcpyAsync(s->h_words + 1, s->err, sizeof(uint32_t), cudaMemcpyDeviceToHost, fi.stream);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(fi.stream);
    const uint32_t total = ce == cudaSuccess ? s->h_words[0] : 0u, err = ce == cudaSuccess ? s->h_words[1] : 0u;
    if (err) {
        cudaMemset(s->err, 0, sizeof(uint32_t));
        if (err & DEVERR_CELL_OVERFLOW)
            st = fail(WC_ERR_NUMERIC, "a cell row held more than %u particles (a collapsed or non-finite state)",
                      3u * MAX_CELL_PARTICLES);
        else
            st = fail(WC_ERR_TIMEOUT, "surface scan look-back exceeded its wait limit");
    } else if (total > s->tri_cap) {
        if (s->tris) cudaFree(s->tris);
        s->tris = nullptr;
        s->tri_cap = 0;
        s->have = false;  // the mesh of the extraction before went with its buffer
        st = dalloc(&s->tris, (size_t)total * 9u);
        if (st == WC_OK) {
            s->tri_cap = total;
            emit();
            cudaEventRecord(e2, fi.stream);
            ce = cudaStreamSynchronize(fi.stream);
        }
    }
    if (ce == cudaSuccess && st == WC_OK) {
        cudaEventElapsedTime(&s->ms_field, e0, e1);
        cudaEventElapsedTime(&s->ms_mesh, e1, e2);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaEventDestroy(e2);
    if (st != WC_OK) return st;
    if (ce != cudaSuccess) return fail(WC_ERR_CUDA, "surface extraction: %s", cudaGetErrorString(ce));
    s->ntris = total;
    s->have = true;
    if (num_triangles) *num_triangles = total;
    return WC_OK;
}

WC_API wc_status wc_surface_get_triangles(wc_surface* s, float* out, uint64_t num_triangles) {
    clear_error();
    if (!s || (!out && num_triangles)) return fail(WC_ERR_INVALID_ARG, "null argument");
    if (!s->have) return fail(WC_ERR_STATE, "no surface extracted yet");
    if (num_triangles != s->ntris)
        return fail(WC_ERR_INVALID_ARG, "buffer holds %llu triangles, the surface has %llu",
                    (unsigned long long)num_triangles, (unsigned long long)s->ntris);
    if (num_triangles)
        WC_CUDA_TRY(cudaMemcpy(out, s->tris, sizeof(float) * 9u * (size_t)num_triangles, cudaMemcpyDeviceToHost));
    return WC_OK;
}

WC_API wc_status wc_surface_get_field(wc_surface* s, float* out, uint64_t count) {
    clear_error();
    if (!s || !out) return fail(WC_ERR_INVALID_ARG, "null argument");
    if (!s->have) return fail(WC_ERR_STATE, "no surface extracted yet");
    if (count != (uint64_t)s->G * s->G * s->G) return fail(WC_ERR_INVALID_ARG, "field has grid_res^3 values");
    WC_CUDA_TRY(cudaMemcpy(out, s->phi, sizeof(float) * (size_t)count, cudaMemcpyDeviceToHost));
    return WC_OK;
}

WC_API wc_status wc_surface_timings(const wc_surface* s, float* ms_field, float* ms_mesh) {
    clear_error();
    if (!s) return fail(WC_ERR_INVALID_ARG, "null surface");
    if (ms_field) *ms_field = s->ms_field;
    if (ms_mesh) *ms_mesh = s->ms_mesh;
    return WC_OK;
}

}  // extern "C"
