// wc_nn_gemm.cu — BF16 tensor-core GEMM for the learned surrogate (sm_103a tcgen05 + TMEM).
//
//   C[m, n] = sum_k A[m, k] * B[k, n]        (BF16 operands, FP32 accumulation in TMEM)
//
// Five kernels, all with 128 x 128 tiles, operands in shared memory, tcgen05.mma issued by one thread into accumulators in
// tensor memory and the results read back with tcgen05.ld:
//   gemm_tma_kernel    row-major A (or two sources split at a whole slice of 64) and B^T, n <= 128, k <= 384: persistent,
//                      operands by TMA; results through shared memory and TMA, or a row per thread (launch_tma)
//   gemm_mlp_kernel    two layers and their LayerNorm, for inference
//   gemm_wgrad_kernel  X^T dY with m, n <= 128, both operands by TMA along their rows
//   gemm_pipe_kernel   the other row-major forms (A rows by index, a source split inside a slice, n > 128, k > 384,
//                      operands that TMA cannot address): persistent, a cp.async operand ring
//   gemm_kernel        the other transposed operands and splits of K, one tile per CTA: per 64-deep slice of K all
//                      threads stage A and B in the no-swizzle K-major layout (8-row x 16-byte core matrices; the next
//                      along K 128 B away, the next 8-row group 1,024 B away); warp w stores rows 32w .., one per thread
//
// Operand sources (staging policies):
//   A row-major [m x k] (lda), optionally with a row index (gather) and a second source for
//     the columns at and after k_split (concatenation [X | Y]); or A transposed: A[i][kk] =
//     a[kk * lda + i] (the weight-gradient GEMM X^T dY).
//   B as B^T row-major [n x k] (ldb) (a weight matrix stored output-major), or B row-major
//     [k x n] (the upstream gradient dY in X^T dY, and W in dY W^T).
// Every wait on the mbarrier is bounded; a wait that runs out sets an error flag, and the
// kernel still releases its tensor memory before it returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "wc_internal.h"
#include "wc_nn.h"
#include "wc_util.h"

namespace wc {
namespace nn {
namespace {

constexpr int BM = 128, BN = 128, BK = 64;
constexpr int THREADS = 128;
constexpr uint32_t TMEM_COLS = 128;
constexpr uint32_t WAIT_LIMIT = 1u << 22;

// Instruction descriptor of tcgen05.mma kind::f16: FP32 accumulator (bits 4-5 = 1), BF16 A and
// B (bits 7-9 = 1, bits 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24.
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                           ((uint32_t)(BM >> 4) << 24);

// Two buffers of each operand tile: the threads stage slice k+1 into one while the tensor core
// still reads slice k from the other.
struct __align__(1024) Tiles {
    __nv_bfloat16 a[2][BM * BK];  // 2 x 16 KB
    __nv_bfloat16 b[2][BN * BK];  // 2 x 16 KB
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor: start >> 4, LBO = 128 B (next core matrix along K),
// SBO = 1024 B (next 8-row group), version 1, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)(128u >> 4) << 16;
    d |= (uint64_t)(1024u >> 4) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Byte offset of element (r, k) of a 128 x 64 tile in the core-matrix layout.
__device__ __forceinline__ uint32_t tile_off(uint32_t r, uint32_t k) {
    return (((r >> 3) * 8u + (k >> 3)) << 7) + ((r & 7u) << 4) + ((k & 7u) << 1);
}

__device__ __forceinline__ bool mbar_wait(uint32_t addr, uint32_t parity) {
    for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Stage a 128 x 64 slice of an operand: rows [row0, row0 + 128) of the logical matrix, columns
// [k0, k0 + 64). T = transposed source (logical (r, k) = src[k * ld + r]).
struct OperandSrc {
    const __nv_bfloat16* p;   // primary source
    const __nv_bfloat16* p2;  // second source for columns >= k_split (row-major only), or null
    const uint32_t* rows;     // row gather (row-major only), or null
    uint32_t ld, ld2, k_split;
    uint32_t nrows, ncols;    // logical extent
    int transposed;
};

__device__ __forceinline__ void stage(const OperandSrc& s, __nv_bfloat16* tile, uint32_t row0, uint32_t k0) {
    unsigned char* base = reinterpret_cast<unsigned char*>(tile);
    if (!s.transposed) {
        // 1,024 chunks of 8 elements (16 B); chunk id -> (row r, k-group g).
        for (uint32_t id = threadIdx.x; id < (uint32_t)(BM * BK / 8); id += THREADS) {
            const uint32_t r = id >> 3, g = id & 7u;
            const uint32_t row = row0 + r, col = k0 + 8u * g;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (row < s.nrows && col < s.ncols) {
                const uint32_t src_row = s.rows ? __ldg(s.rows + row) : row;
                const __nv_bfloat16* src;
                if (s.p2 && col >= s.k_split)
                    src = s.p2 + (size_t)src_row * s.ld2 + (col - s.k_split);
                else
                    src = s.p + (size_t)src_row * s.ld + col;
                v = __ldg(reinterpret_cast<const uint4*>(src));
            }
            *reinterpret_cast<uint4*>(base + tile_off(r, 8u * g)) = v;
        }
    } else {
        // 128 blocks of 8 logical rows x 8 k: eight 16-byte loads (8 rows at one k each),
        // transposed in registers with byte permutes into eight 16-byte core-matrix rows.
        for (uint32_t b = threadIdx.x; b < (uint32_t)((BM / 8) * (BK / 8)); b += THREADS) {
            const uint32_t kg = b >> 4, rg = b & 15u;
            const uint32_t r = row0 + 8u * rg;
            uint4 v[8];
#pragma unroll
            for (uint32_t e = 0; e < 8; ++e) {
                const uint32_t kk = k0 + 8u * kg + e;
                v[e] = make_uint4(0u, 0u, 0u, 0u);
                if (kk < s.ncols && r < s.nrows) v[e] = __ldg(reinterpret_cast<const uint4*>(s.p + (size_t)kk * s.ld + r));
            }
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) {
                // row 8 rg + j: element e of the output row is element j of v[e]
                const uint32_t sel = (j & 1u) ? 0x7632u : 0x5410u;
                const uint32_t q = j >> 1;
                auto word = [&](const uint4& x) { return q == 0 ? x.x : q == 1 ? x.y : q == 2 ? x.z : x.w; };
                uint4 w;
                w.x = __byte_perm(word(v[0]), word(v[1]), sel);
                w.y = __byte_perm(word(v[2]), word(v[3]), sel);
                w.z = __byte_perm(word(v[4]), word(v[5]), sel);
                w.w = __byte_perm(word(v[6]), word(v[7]), sel);
                *reinterpret_cast<uint4*>(base + tile_off(8u * rg + j, 8u * kg)) = w;
            }
        }
    }
}

// The row-major staging as asynchronous copies (cp.async, 16 bytes each, zero-filled outside the
// matrix): no registers, and the copies of the next slice run while the tensor core works.
__device__ __forceinline__ void stage_async(const OperandSrc& s, __nv_bfloat16* tile, uint32_t row0, uint32_t k0) {
    const uint32_t base = smem_addr(tile);
#pragma unroll 4
    for (uint32_t id = threadIdx.x; id < (uint32_t)(BM * BK / 8); id += THREADS) {
        const uint32_t r = id >> 3, g = id & 7u;
        const uint32_t row = row0 + r, col = k0 + 8u * g;
        const __nv_bfloat16* src = s.p;  // nothing is read when bytes = 0
        uint32_t bytes = 0;
        if (row < s.nrows && col < s.ncols) {
            const uint32_t src_row = s.rows ? __ldg(s.rows + row) : row;
            if (s.p2 && col >= s.k_split)
                src = s.p2 + (size_t)src_row * s.ld2 + (col - s.k_split);
            else
                src = s.p + (size_t)src_row * s.ld + col;
            bytes = 16;
        }
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + tile_off(r, 8u * g)), "l"(src),
                     "r"(bytes)
                     : "memory");
    }
}

// x[0..ncols) += r[0..ncols) (bf16): 16-byte loads when the row segment is whole and aligned.
__device__ __forceinline__ void add_row(float x[32], const __nv_bfloat16* r, uint32_t ncols) {
    if (ncols == 32u && (reinterpret_cast<uintptr_t>(r) & 15u) == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint4 v = reinterpret_cast<const uint4*>(r)[q];
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 f = __bfloat1622float2(h[k]);
                x[8 * q + 2 * k] += f.x;
                x[8 * q + 2 * k + 1] += f.y;
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if ((uint32_t)j < ncols) x[j] += __bfloat162float(r[j]);
    }
}

// Bias, gathered row adds, ReLU and the stores of 32 accumulator columns of one row:
// x[0..ncols) belong to output columns col0 ..; kz: the split of the K range (partial outputs
// split_stride apart); i1, i2: the row's indices into the gathered operands.
__device__ __forceinline__ void epilogue_store(const GemmArgs& g, float x[32], uint32_t row, uint32_t col0,
                                               uint32_t ncols, uint32_t kz, uint32_t i1, uint32_t i2) {
    if (g.bias) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if ((uint32_t)j < ncols) x[j] += g.bias[col0 + j];
    }
    if (g.add1) add_row(x, g.add1 + (size_t)i1 * g.ld_add + col0, ncols);
    if (g.add2) add_row(x, g.add2 + (size_t)i2 * g.ld_add + col0, ncols);
    if (g.relu) {
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = fmaxf(x[j], 0.f);
    }
    // Stores: 16-byte vectors for whole aligned segments, otherwise element by element with
    // constant indices (the accumulator stays in registers either way).
    if (g.c_f32) {
        float* out = g.c_f32 + (size_t)kz * g.split_stride + (size_t)row * g.ldc + col0;
        if (ncols == 32 && ((reinterpret_cast<uintptr_t>(out) & 15u) == 0)) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                float4* o = reinterpret_cast<float4*>(out + j);
                float4 v = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
                if (g.accumulate) {
                    const float4 c = *o;
                    v.x += c.x;
                    v.y += c.y;
                    v.z += c.z;
                    v.w += c.w;
                }
                *o = v;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if ((uint32_t)j < ncols) out[j] = g.accumulate ? out[j] + x[j] : x[j];
        }
    }
    if (g.c_bf16) {
        __nv_bfloat16* out = g.c_bf16 + (size_t)row * g.ldc + col0;
        if (ncols == 32 && ((reinterpret_cast<uintptr_t>(out) & 15u) == 0)) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
                __nv_bfloat162 q0 = __floats2bfloat162_rn(x[j], x[j + 1]);
                __nv_bfloat162 q1 = __floats2bfloat162_rn(x[j + 2], x[j + 3]);
                __nv_bfloat162 q2 = __floats2bfloat162_rn(x[j + 4], x[j + 5]);
                __nv_bfloat162 q3 = __floats2bfloat162_rn(x[j + 6], x[j + 7]);
                uint4 w;
                w.x = *reinterpret_cast<uint32_t*>(&q0);
                w.y = *reinterpret_cast<uint32_t*>(&q1);
                w.z = *reinterpret_cast<uint32_t*>(&q2);
                w.w = *reinterpret_cast<uint32_t*>(&q3);
                *reinterpret_cast<uint4*>(out + j) = w;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if ((uint32_t)j < ncols) out[j] = __float2bfloat16_rn(x[j]);
        }
    }

}

__global__ void __launch_bounds__(THREADS) gemm_kernel(const GemmArgs g, uint32_t* err) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    Tiles& t = *reinterpret_cast<Tiles*>(smem_raw);
    __shared__ uint64_t mbar[2];  // MMA completion per operand buffer
    __shared__ uint32_t tmem_slot;
    __shared__ int s_failed;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const uint32_t kz = blockIdx.z;  // split of the K range (weight gradients)
    const uint32_t k_begin = kz * g.k_chunk;
    const uint32_t k_end = min(g.k, k_begin + g.k_chunk);

    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&mbar[0])));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&mbar[1])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_failed = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    OperandSrc A{g.a, g.a2, g.a_rows, g.lda, g.lda2, g.k_split, g.m, g.k, g.a_transposed};
    // B is staged as B^T (rows = output columns n, columns = k).
    OperandSrc B{g.b, nullptr, nullptr, g.ldb, 0u, 0u, g.n, g.k, g.b_rowmajor};

    uint32_t phase[2] = {0u, 0u};
    bool pending[2] = {false, false};  // an MMA batch reading this buffer may still run
    bool ok = true;
    uint32_t issued = 0;
    int last = -1;
    // Both operands row-major: asynchronous copies, one slice ahead. Otherwise the threads stage
    // through registers (the transposed forms), still into the buffer the tensor core is not
    // reading.
    const bool async = !A.transposed && !B.transposed;
    if (async && k_begin < k_end) {
        stage_async(A, t.a[0], m0, k_begin);
        stage_async(B, t.b[0], n0, k_begin);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (uint32_t k0 = k_begin; k0 < k_end; k0 += BK) {
        const int buf = (int)(issued & 1u);
        if (async) {
            const uint32_t kn = k0 + BK;
            if (kn < k_end) {
                const int nb = buf ^ 1;
                if (pending[nb]) {
                    // the batch that read buffer nb (one slice back) must finish before the rewrite
                    if (!mbar_wait(smem_addr(&mbar[nb]), phase[nb])) ok = false;
                    phase[nb] ^= 1u;
                    pending[nb] = false;
                }
                stage_async(A, t.a[nb], m0, kn);
                stage_async(B, t.b[nb], n0, kn);
                asm volatile("cp.async.commit_group;" ::: "memory");
                asm volatile("cp.async.wait_group 1;" ::: "memory");  // this slice's copies are done
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
        } else {
            if (pending[buf]) {
                // The batch two slices back read this buffer: it must finish before the rewrite.
                if (!mbar_wait(smem_addr(&mbar[buf]), phase[buf])) ok = false;
                phase[buf] ^= 1u;
                pending[buf] = false;
            }
            stage(A, t.a[buf], m0, k0);
            stage(B, t.b[buf], n0, k0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a_base = smem_addr(t.a[buf]), b_base = smem_addr(t.b[buf]);
#pragma unroll
            for (uint32_t j = 0; j < BK / 16; ++j) {
                const uint64_t ad = smem_desc(a_base + 256u * j);
                const uint64_t bd = smem_desc(b_base + 256u * j);
                const uint32_t acc = (issued > 0 || j > 0) ? 1u : 0u;
                asm volatile(
                    "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                    " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(IDESC), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_addr(&mbar[buf]))
                         : "memory");
        }
        pending[buf] = true;
        last = buf;
        ++issued;
    }
    // The last commit covers every MMA issued before it; the other buffer's arrival needs no wait.
    if (last >= 0) {
        if (!mbar_wait(smem_addr(&mbar[last]), phase[last])) ok = false;
    }
    if (!ok) atomicOr(&s_failed, 1);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    const bool failed = s_failed != 0;
    if (failed && threadIdx.x == 0 && err) atomicOr(err, DEVERR_MMA_TIMEOUT);

    // Epilogue: thread owns row m0 + 32 warp + lane; columns in chunks of 32.
    const uint32_t row = m0 + 32u * warp + lane;
    const bool row_ok = row < g.m && !failed;
    for (uint32_t c0 = 0; c0 < BN; c0 += 32) {
        uint32_t v[32];
        const uint32_t taddr = tmem + ((32u * warp) << 16) + c0;
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
              "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
              "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
            : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (!row_ok || n0 + c0 >= g.n) continue;
        float x[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = issued ? __uint_as_float(v[j]) : 0.f;
        epilogue_store(g, x, row, n0 + c0, min(32u, g.n - (n0 + c0)), kz, g.add1 ? g.add1_idx[row] : 0u,
                       g.add2 ? g.add2_idx[row] : 0u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

// ---- persistent, warp-specialised kernel (row-major A with gather / concatenation, B^T) --------
//
// Grid: one CTA per SM, looping over output tiles. Warps 0..3 (the producers) copy operand
// slices with cp.async into a ring of shared-memory slots, one commit group per ring step, and
// keep LAG groups in flight: after committing a group a thread waits until only the LAG newest
// are pending, fences the older ones into the async proxy and arrives on their `full` barriers.
// With B resident (RB: n <= 128 and k <= 384) the producers first copy the whole B^T tile once
// (barrier `b_full`) and the ring carries A slices only (6 slots, 4 in flight); otherwise each
// slot holds an A and a B slice (4 slots, 2 in flight). Warp 4 (lane 0) waits for `full`, issues
// the slice's four MMAs into one of two 128-column accumulators in tensor memory and commits them
// to the slot's `empty` barrier (the slot may be refilled) and, after a tile's last slice, to the
// accumulator's `acc_full` barrier. Warps 5..12 wait for `acc_full`, read 32 accumulator rows x 64
// columns each (warp w reads lanes 32 (w % 4) ..), apply the epilogue and arrive on `acc_empty`. So
// the copies of the next slices, the MMAs of one tile and the epilogue of the previous tile
// overlap. Every wait is bounded; a wait that runs out stops the CTA's loops
// (DEVERR_MMA_TIMEOUT) and the CTA still frees its tensor memory.
constexpr int PIPE_PRODUCERS = 4;  // warps 0..3 copy, warp 4 issues the MMAs, warps 5..12 drain
constexpr int PIPE_EPILOGUE = 8;   // two warps per 32-lane quarter of the accumulator, 64 columns each
constexpr int PIPE_THREADS = 32 * (PIPE_PRODUCERS + 1 + PIPE_EPILOGUE);
constexpr uint32_t PIPE_TMEM_COLS = 256;
constexpr uint32_t TILE_BYTES = BM * BK * 2;  // one 128 x 64 BF16 operand slice, 16 KB
// Resident B (RB): the whole B^T tile [128 x k] stays in shared memory, loaded once per CTA,
// and the ring carries A slices only. For n <= 128 (one column of tiles) and k <= 64 RB_MAX_SLICES.
constexpr uint32_t RB_MAX_SLICES = 6;
template <bool RB>
struct PipeShape {
    static constexpr int STAGES = RB ? 6 : 4;  // ring slots
    static constexpr int LAG = STAGES - 2;     // copy groups a producer keeps in flight
};

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(smem_addr(bar)) : "memory");
}

// A producer thread's share of one slice: 16-byte copies (PIPE_PRODUCERS warps), zero-filled
// outside the matrix.
__device__ __forceinline__ void pipe_stage_copy(const OperandSrc& s, __nv_bfloat16* tile, uint32_t row0, uint32_t k0,
                                                uint32_t ptid) {
    const uint32_t base = smem_addr(tile);
#pragma unroll 4
    for (uint32_t id = ptid; id < (uint32_t)(BM * BK / 8); id += 32u * PIPE_PRODUCERS) {
        const uint32_t r = id >> 3, g = id & 7u;
        const uint32_t row = row0 + r, col = k0 + 8u * g;
        const __nv_bfloat16* src = s.p;
        uint32_t bytes = 0;
        if (row < s.nrows && col < s.ncols) {
            const uint32_t src_row = s.rows ? __ldg(s.rows + row) : row;
            if (s.p2 && col >= s.k_split)
                src = s.p2 + (size_t)src_row * s.ld2 + (col - s.k_split);
            else
                src = s.p + (size_t)src_row * s.ld + col;
            bytes = 16;
        }
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + tile_off(r, 8u * g)), "l"(src),
                     "r"(bytes)
                     : "memory");
    }
}

// The epilogue warps of the persistent kernels: for each of the CTA's tiles wait for its
// accumulator (acc_full[t & 1]), read 32 rows (lanes 32 quarter ..) x 64 columns (64 half ..)
// with tcgen05.ld, apply the epilogue, and hand the accumulator back (acc_empty). A wait that runs
// out sets `failed`.
__device__ __forceinline__ void drain_accumulators(const GemmArgs& g, uint32_t tmem, uint64_t* acc_full,
                                                   uint64_t* acc_empty, volatile int* failed, uint32_t ntiles,
                                                   uint32_t tiles_n, uint32_t nslices, uint32_t quarter,
                                                   uint32_t half, uint32_t lane) {
    uint32_t t = 0;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++t) {
        const uint32_t b = t & 1u;
        const uint32_t m0 = (tile / tiles_n) * BM, n0 = (tile % tiles_n) * BN;
        const uint32_t row = m0 + 32u * quarter + lane;
        const bool row_ok = row < g.m;
        const uint32_t i1 = g.add1 && row_ok ? g.add1_idx[row] : 0u, i2 = g.add2 && row_ok ? g.add2_idx[row] : 0u;
        bool ok = !*failed && mbar_wait(smem_addr(&acc_full[b]), (t >> 1) & 1u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
            if (lane == 0) *failed = 1;
            break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (uint32_t c0 = 64u * half; c0 < 64u * half + 64u; c0 += 32) {
            uint32_t v[32];
            const uint32_t taddr = tmem + ((32u * quarter) << 16) + b * (uint32_t)BN + c0;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                  "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                  "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (!row_ok || n0 + c0 >= g.n) continue;
            float x[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] = nslices ? __uint_as_float(v[j]) : 0.f;
            epilogue_store(g, x, row, n0 + c0, min(32u, g.n - (n0 + c0)), 0u, i1, i2);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[b]);
    }
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t v[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}

template <bool RB>
__global__ void __launch_bounds__(PIPE_THREADS, 1) gemm_pipe_kernel(const GemmArgs g, uint32_t* err) {
    constexpr int STAGES = PipeShape<RB>::STAGES, LAG = PipeShape<RB>::LAG;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2], b_full;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_failed;
    volatile int* failed = &s_failed;  // polled by all three roles
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t tiles_m = (g.m + BM - 1) / BM, tiles_n = (g.n + BN - 1) / BN;
    const uint32_t ntiles = tiles_m * tiles_n;
    const uint32_t nslices = (g.k + BK - 1) / BK;
    // RB: [B slices 0 .. nslices)[A ring]; otherwise the ring's slots hold an A and a B slice each
    unsigned char* const ring = smem_raw + (RB ? nslices * TILE_BYTES : 0u);
    auto a_slot = [&](uint32_t st) { return ring + st * (RB ? 1u : 2u) * TILE_BYTES; };
    auto b_slice = [&](uint32_t st, uint32_t sl) {
        return RB ? smem_raw + sl * TILE_BYTES : ring + (2u * st + 1u) * TILE_BYTES;
    };

    if (threadIdx.x == 0) {
        for (int q = 0; q < STAGES; ++q) {
            mbar_init(&full[q], 32 * PIPE_PRODUCERS);
            mbar_init(&empty[q], 1);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(&acc_full[q], 1);
            mbar_init(&acc_empty[q], PIPE_EPILOGUE);  // one arrival per epilogue warp
        }
        mbar_init(&b_full, 32 * PIPE_PRODUCERS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_failed = 0;
    }
    if (warp == PIPE_PRODUCERS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)),
                     "r"(PIPE_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const OperandSrc A{g.a, g.a2, g.a_rows, g.lda, g.lda2, g.k_split, g.m, g.k, 0};
    const OperandSrc B{g.b, nullptr, nullptr, g.ldb, 0u, 0u, g.n, g.k, 0};

    if (warp < PIPE_PRODUCERS) {
        // producers: copy groups in commit order (RB: group 0 is B, group 1 + i the A slice of
        // ring step i; otherwise group i is ring step i); a group is published (fenced, its
        // barrier arrived on) once LAG later groups have been committed, or at the end
        const uint32_t ptid = threadIdx.x;
        uint32_t it = 0, committed = 0, published = 0;
        auto publish_upto = [&](uint32_t upto) {
            for (; published < upto; ++published) {
                if (RB && published == 0)
                    mbar_arrive(&b_full);
                else
                    mbar_arrive(&full[(published - (RB ? 1u : 0u)) % STAGES]);
            }
        };
        if (RB) {
            for (uint32_t sl = 0; sl < nslices; ++sl)
                pipe_stage_copy(B, reinterpret_cast<__nv_bfloat16*>(b_slice(0, sl)), 0u, sl * BK, ptid);
            asm volatile("cp.async.commit_group;" ::: "memory");
            ++committed;
        }
        for (uint32_t tile = blockIdx.x; tile < ntiles && !*failed; tile += gridDim.x) {
            const uint32_t m0 = (tile / tiles_n) * BM, n0 = (tile % tiles_n) * BN;
            for (uint32_t sl = 0; sl < nslices; ++sl, ++it) {
                const uint32_t st = it % STAGES;
                if (it >= (uint32_t)STAGES && !mbar_wait(smem_addr(&empty[st]), ((it / STAGES) - 1u) & 1u)) {
                    *failed = 1;
                    break;
                }
                pipe_stage_copy(A, reinterpret_cast<__nv_bfloat16*>(a_slot(st)), m0, sl * BK, ptid);
                if (!RB) pipe_stage_copy(B, reinterpret_cast<__nv_bfloat16*>(b_slice(st, sl)), n0, sl * BK, ptid);
                asm volatile("cp.async.commit_group;" ::: "memory");
                ++committed;
                if (committed > (uint32_t)LAG) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(LAG) : "memory");
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    publish_upto(committed - LAG);
                }
            }
            if (*failed) break;
        }
        // the last groups
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        publish_upto(committed);
    } else if (warp == PIPE_PRODUCERS) {
        // MMA issue (one thread)
        if (lane == 0) {
            uint32_t it = 0, t = 0;
            if (RB && ntiles > blockIdx.x && !mbar_wait(smem_addr(&b_full), 0u)) *failed = 1;
            for (uint32_t tile = blockIdx.x; tile < ntiles && !*failed; tile += gridDim.x, ++t) {
                const uint32_t b = t & 1u;
                if (t >= 2 && !mbar_wait(smem_addr(&acc_empty[b]), ((t >> 1) - 1u) & 1u)) {
                    *failed = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc_addr = tmem + b * (uint32_t)BN;
                for (uint32_t sl = 0; sl < nslices; ++sl, ++it) {
                    const uint32_t st = it % STAGES;
                    if (!mbar_wait(smem_addr(&full[st]), (it / STAGES) & 1u)) {
                        *failed = 1;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_base = smem_addr(a_slot(st)), b_base = smem_addr(b_slice(st, sl));
#pragma unroll
                    for (uint32_t j = 0; j < BK / 16; ++j) {
                        const uint64_t ad = smem_desc(a_base + 256u * j);
                        const uint64_t bd = smem_desc(b_base + 256u * j);
                        const uint32_t acc = (sl > 0 || j > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(acc_addr),
                            "l"(ad), "l"(bd), "r"(IDESC), "r"(acc));
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                     smem_addr(&empty[st]))
                                 : "memory");
                }
                if (*failed) break;
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_addr(&acc_full[b]))
                             : "memory");
            }
        }
        __syncwarp();
    } else {
        // epilogue: warp w reads accumulator lanes 32 (w % 4) .. + 31 (the lanes its position in
        // the warpgroup may address), columns 64 half .. + 63
        const uint32_t quarter = warp & 3u;
        const uint32_t half = (warp - (uint32_t)(PIPE_PRODUCERS + 1)) / 4u;
        drain_accumulators(g, tmem, acc_full, acc_empty, failed, ntiles, tiles_n, nslices, quarter, half, lane);
    }
    __syncthreads();
    if (*failed && threadIdx.x == 0 && err) atomicOr(err, DEVERR_MMA_TIMEOUT);
    if (warp == PIPE_PRODUCERS) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(PIPE_TMEM_COLS));
    }
}

// ---- TMA variant: plain row-major A and B^T, B resident ----------------------------------------
//
// For A without a row gather (a second source takes over at a whole slice), and B^T of one column of tiles (n <= 128,
// k <= 64 RB_MAX_SLICES): one thread of warp 0 copies the operands with cp.async.bulk.tensor
// (TMA) in the 128-byte-swizzled K-major layout — B^T once per CTA (barrier `b_full`), then the
// A slices of the CTA's tiles into a ring, each copy completing its slot's `full` barrier
// by its byte count (mbarrier expect_tx); warp 1 issues the MMAs with 128-byte-swizzle
// descriptors (a K step of 16 is a 32-byte advance inside the swizzle atom); warps 2..9 drain
// the accumulators, two warps per 32 rows, 64 columns each. The tensor maps cover this GPU's
// own global memory; no multicast.
//
// The epilogue never touches global memory a row per thread (32 lines per instruction): results
// leave through shared memory and TMA stores, a 32-row box per warp (FP32 accumulation into C as
// a TMA add), and what it reads per element arrives there first, 128 columns by 128 rows in two
// stages — the residual rows of a LayerNorm by TMA (AUX_TMA), the gathered rows added to a layer by
// four more warps with cp.async, 16 lanes to a row (AUX_GATHER). Forms that it cannot take are written from the
// registers (AUX_DIRECT, see launch_tma). BF16 results are written over
// the place of the values read. Bound by the traffic it cannot avoid: 460,000 rows of 128 with two
// gathered rows each take 55 us against 134 us with row-per-thread accesses (66 % of the copy
// bandwidth for A and C alone, the gathered rows come from L2 on top).
constexpr int TMA_THREADS = 32 * (2 + PIPE_EPILOGUE);
constexpr int GATHER_WARPS = 4;
constexpr int TMA_MAX_STAGES = 6;
constexpr uint32_t TMA_SMEM_LIMIT = 224u * 1024u;  // dynamic; the barriers and row sums take up to 3 KB more
enum : int { AUX_NONE = 0, AUX_TMA = 1, AUX_GATHER = 2, AUX_DIRECT = 3 };
constexpr uint32_t AUX_BYTES = BM * 128u * 2u;      // 128 rows of 128 BF16: two halves of 64 columns
constexpr uint32_t HALF_BYTES = AUX_BYTES / 2u;     // a half's rows of 128 bytes, swizzled
constexpr uint32_t F32_OUT_BYTES = BM * 128u * 4u;  // per warp two boxes of 32 rows x 32 columns

// Shared-memory descriptor of a K-major operand tile in the 128-byte swizzle layout: rows of
// 128 bytes, 8-row groups 1,024 bytes apart (SBO), the leading-byte offset unused, version 1.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024u >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

// One 64 x 128 box (64 K elements, 128 rows) of a 2-D BF16 tensor map into shared memory; the
// copy completes `bar` by its bytes. x (the K coordinate) is a multiple of 64 elements (128 B).
__device__ __forceinline__ void tma_load_box(const CUtensorMap* map, void* dst, uint32_t x, uint32_t y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_addr(bar))
        : "memory");
}

// A 32-row box from shared memory to the tensor of `map` (rows and columns outside it are not
// written), as a store or as an addition to what is there.
__device__ __forceinline__ void tma_store_box(const CUtensorMap* map, uint32_t src, uint32_t x, uint32_t y, bool add) {
    if (add)
        asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                         reinterpret_cast<uint64_t>(map)),
                     "r"(x), "r"(y), "r"(src)
                     : "memory");
    else
        asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                         reinterpret_cast<uint64_t>(map)),
                     "r"(x), "r"(y), "r"(src)
                     : "memory");
}

// Byte offset of 16-byte chunk c (0..7) of row r in a 128-byte-swizzled block.
__device__ __forceinline__ uint32_t sw128(uint32_t r, uint32_t c) { return r * 128u + ((c ^ (r & 7u)) << 4); }

__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts128(uint32_t a, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 q = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&q);
}
// x[0..8) += the eight BF16 of v, one instruction each (BF16 widens exactly)
__device__ __forceinline__ void add8(float* x, const uint4& v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k)
        asm("{\n .reg .b16 lo, hi;\n mov.b32 {lo, hi}, %2;\n add.rn.f32.bf16 %0, lo, %0;\n add.rn.f32.bf16 %1, hi, %1;\n}\n"
            : "+f"(x[2 * k]), "+f"(x[2 * k + 1])
            : "r"(w[k]));
}

// Shared memory of the TMA kernel: [B^T slices][A ring][two aux / BF16 output stages][FP32 output].
struct TmaPlan {
    uint32_t stages;     // A ring slots
    uint32_t aux_bytes;  // per stage: operands of 32 KB (AUX_GATHER with two: 64 KB), 0 without BF16 output or aux
    uint32_t f32_bytes;
    uint32_t one_stage;  // BF16 output, no aux rows: one stage instead of two
    uint32_t smem;
};

struct TmaMaps {
    CUtensorMap a, a2, b, aux, cb, cf;
};

__device__ __forceinline__ void pair_sync(uint32_t quarter) {
    asm volatile("bar.sync %0, 64;" ::"r"(1u + quarter) : "memory");
}

// The packed FP32 instructions on (a[0], a[1]), each half rounded as the scalar ones.
__device__ __forceinline__ void add_pair(float* a, float b0, float b1) {
    asm("{\n .reg .b64 a, b;\n mov.b64 a, {%0, %1};\n mov.b64 b, {%2, %3};\n add.rn.f32x2 a, a, b;\n mov.b64 {%0, %1}, a;\n}\n"
        : "+f"(a[0]), "+f"(a[1])
        : "f"(b0), "f"(b1));
}
// a = a m g + b
__device__ __forceinline__ void scale_pair(float* a, float m, float g0, float g1, float b0, float b1) {
    asm("{\n .reg .b64 a, m, g, b;\n mov.b64 a, {%0, %1};\n mov.b64 m, {%2, %2};\n mov.b64 g, {%3, %4};\n mov.b64 b, {%5, %6};\n"
        " mul.rn.f32x2 a, a, m;\n fma.rn.f32x2 a, a, g, b;\n mov.b64 {%0, %1}, a;\n}\n"
        : "+f"(a[0]), "+f"(a[1])
        : "f"(m), "f"(g0), "f"(g1), "f"(b0), "f"(b1));
}

// Eight consecutive values.
__device__ __forceinline__ void load8(float* o, const float* p) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = reinterpret_cast<const float4*>(p)[1];
    o[0] = a.x, o[1] = a.y, o[2] = a.z, o[3] = a.w, o[4] = b.x, o[5] = b.y, o[6] = b.z, o[7] = b.w;
}

// The LayerNorm of n = 128 columns. ln_centre: by the two warps of a pair, x a thread's 64 columns of its row, which
// becomes x - mean (xs, xv, oks as in tma_epilogue); false when a wait of either warp failed (both leave). ln_scale:
// eight columns o = gamma x rstd + beta.
template <bool VEC>
__device__ __forceinline__ void ln_scale(const float* gamma, const float* beta, const float* x, float rstd, float* o) {
    float gm[8], bt[8];
    if (VEC) {
#pragma unroll
        for (int k = 0; k < 8; k += 4) {
            const float4 g4 = *reinterpret_cast<const float4*>(gamma + k);
            const float4 b4 = *reinterpret_cast<const float4*>(beta + k);
            gm[k] = g4.x, gm[k + 1] = g4.y, gm[k + 2] = g4.z, gm[k + 3] = g4.w;
            bt[k] = b4.x, bt[k + 1] = b4.y, bt[k + 2] = b4.z, bt[k + 3] = b4.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            gm[k] = gamma[k];
            bt[k] = beta[k];
        }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = x[k] * rstd * gm[k] + bt[k];
}
__device__ __forceinline__ bool ln_centre(float (&x)[64], bool ok, float (*xs)[2][32], float (*xv)[2][32], int (*oks)[2],
                                          volatile int* failed, uint32_t quarter, uint32_t half, uint32_t lane, float* rstd) {
    constexpr float LN_EPSILON = 1e-5f;
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < 64; ++j) sum += x[j];
    xs[quarter][half][lane] = sum;
    if (lane == 0) oks[quarter][half] = ok ? 1 : 0;
    pair_sync(quarter);
    if (!(oks[quarter][0] && oks[quarter][1])) {
        if (lane == 0) *failed = 1;
        return false;
    }
    const float mean = (xs[quarter][0][lane] + xs[quarter][1][lane]) * (1.f / 128.f);
    float sq = 0.f;
#pragma unroll
    for (int j = 0; j < 64; j += 2) {
        add_pair(x + j, -mean, -mean);
        sq += x[j] * x[j];
        sq += x[j + 1] * x[j + 1];
    }
    xv[quarter][half][lane] = sq;
    pair_sync(quarter);
    const float var = (xv[quarter][0][lane] + xv[quarter][1][lane]) * (1.f / 128.f);
    *rstd = rsqrtf(var + LN_EPSILON);
    return true;
}

// The epilogue of one warp: rows 32 quarter .., columns 64 half .. of every tile of the CTA.
// LN (n = 128): the two warps that read the same 32 accumulator lanes hold a row's 128 columns
// between them (ln_centre). Each thread sums its 64 values, the pair exchanges the sums through shared memory at
// a named barrier of its 64 threads (ids 1 .. 4), then the squared deviations from the mean the
// same way, and each thread normalises, scales and shifts its own columns and adds the residual
// row. Both warps of a pair pass both barriers of every tile: whether each warp's waits succeeded is
// exchanged at the first barrier and the pair leaves together.
// LN with F32 (training, which keeps the rows before the LayerNorm and its statistics): a thread takes
// every second group of four columns, so that its sums and the pair's one exchange add in the order
// of layernorm_kernel's warp (four columns per lane, lanes in pairs 16, 8, 4, 2, 1 apart), whose
// results training had when it was a kernel of its own (the expressions are that kernel's too, so that
// they contract alike): the layer and its LayerNorm took ~145 us at 460,000 rows.
template <int AUX, bool LN, bool F32, bool BF>
__device__ __forceinline__ void tma_epilogue(const GemmArgs& g, const TmaMaps& maps, const TmaPlan& plan, uint32_t tmem,
                                             uint64_t* acc_full, uint64_t* acc_empty, uint64_t* aux_full,
                                             uint64_t* aux_empty, volatile int* failed, uint32_t ntiles, uint32_t quarter,
                                             uint32_t half, uint32_t lane, uint32_t aux_base, uint32_t f32_base,
                                             float* s_bias, float (*xs)[2][32], float (*xv)[2][32], int (*oks)[2]) {
    constexpr float LN_EPSILON = 1e-5f;
    const uint32_t col0 = 64u * half, r = 32u * quarter + lane;
    const uint32_t f32_buf = f32_base + (quarter * 2u + half) * (F32_OUT_BYTES / 8u);  // this warp's two boxes
    // LN: bias, gamma and beta four at a time when they allow 16-byte loads (uniform branch)
    const bool vec = LN && ((reinterpret_cast<uintptr_t>(g.bias) | reinterpret_cast<uintptr_t>(g.ln_gamma) |
                             reinterpret_cast<uintptr_t>(g.ln_beta)) & 15u) == 0;
    // The bias from shared memory (16,384 rows 4.5 us, one chunk ahead from L1 5.4; beside gathered rows, which leave
    // it no room in L1, 460,000 rows 54.9 against 57.9)
    if (!LN && g.bias) {
        const uint32_t c = threadIdx.x - 64u;
        if (c < 128u) s_bias[c] = c < g.n ? g.bias[c] : 0.f;
        asm volatile("bar.sync 5, 256;" ::: "memory");  // the epilogue's warps
    }
    uint32_t t = 0;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++t) {
        const uint32_t b = t & 1u;
        float bb[8];  // the bias, eight columns ahead of its use
        if (!LN && g.bias) load8(bb, s_bias + col0);
        bool ok = !*failed && mbar_wait(smem_addr(&acc_full[b]), (t >> 1) & 1u);
        if (AUX != AUX_NONE) ok = ok && mbar_wait(smem_addr(&aux_full[b]), (t >> 1) & 1u);
        ok = __all_sync(0xffffffffu, ok);
        if (!LN && !ok) {
            if (lane == 0) *failed = 1;
            break;
        }
        const uint32_t stage = aux_base + (AUX == AUX_NONE && plan.one_stage ? 0u : b) * plan.aux_bytes + half * HALF_BYTES;
        const uint32_t row0 = tile * BM + 32u * quarter;
        // The staging this warp is about to write has been read by its earlier stores: two tiles ago
        // (BF16, two stages), the previous tile's (FP32, one). With aux rows the previous tile's
        // stage, read by then, goes back to the producer, who fills it during this tile.
        if (lane == 0) {
            if (F32 || (AUX != AUX_NONE && BF) || plan.one_stage) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            else asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            if (AUX != AUX_NONE && BF && t > 0) mbar_arrive(&aux_empty[b ^ 1u]);
        }
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t taddr = tmem + ((32u * quarter) << 16) + b * (uint32_t)BN + col0;
        if constexpr (LN && F32) {
            float x[64];  // group j (0..15): columns 8 j + 4 half ..
            if (ok) {
                uint32_t v[64];
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j)
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(v[4 * j]), "=r"(v[4 * j + 1]), "=r"(v[4 * j + 2]), "=r"(v[4 * j + 3])
                                 : "r"(taddr - col0 + 8u * j + 4u * half));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 64; ++j) x[j] = __uint_as_float(v[j]);
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[b]);
            } else {
#pragma unroll
                for (int j = 0; j < 64; ++j) x[j] = 0.f;
            }
            auto four = [&](const float* base, uint32_t j) {  // columns of group j
                const float* q = base + 8u * j + 4u * half;
                return vec ? *reinterpret_cast<const float4*>(q) : make_float4(*q, q[1], q[2], q[3]);
            };
            float s[16];
            auto tree = [&]() {  // the sum of s[0..16) in pairs 8, 4, 2, 1 apart
#pragma unroll
                for (int h = 8; h > 0; h >>= 1)
#pragma unroll
                    for (int j = 0; j < h; ++j) s[j] += s[j + h];
                return s[0];
            };
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j) {
                float* y = x + 4 * j;
                if (g.bias) {
                    const float4 bb = four(g.bias, j);
                    y[0] += bb.x;
                    y[1] += bb.y;
                    y[2] += bb.z;
                    y[3] += bb.w;
                }
                s[j] = ((y[0] + y[1]) + y[2]) + y[3];
            }
            xs[quarter][half][lane] = tree();
            if (lane == 0) oks[quarter][half] = ok ? 1 : 0;
            pair_sync(quarter);
            if (!(oks[quarter][0] && oks[quarter][1])) {
                if (lane == 0) *failed = 1;
                break;
            }
            const float mean = (xs[quarter][0][lane] + xs[quarter][1][lane]) * (1.f / 128.f);
            const uint32_t f32_rows = f32_base + quarter * (F32_OUT_BYTES / 4u);
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j) {
                float* y = x + 4 * j;
                sts128(f32_rows + (j >> 2) * 4096u + sw128(lane, 2u * (j & 3u) + half),
                       make_uint4(__float_as_uint(y[0]), __float_as_uint(y[1]), __float_as_uint(y[2]), __float_as_uint(y[3])));
#pragma unroll
                for (int k = 0; k < 4; ++k) y[k] -= mean;
                s[j] = y[0] * y[0] + y[1] * y[1] + y[2] * y[2] + y[3] * y[3];
            }
            xv[quarter][half][lane] = tree();
            pair_sync(quarter);
            const float var = (xv[quarter][0][lane] + xv[quarter][1][lane]) * (1.f / 128.f);
            const float rstd = rsqrtf(var + LN_EPSILON);
            if (half == 0 && row0 + lane < g.m) {
                g.ln_mean[row0 + lane] = mean;
                g.ln_rstd[row0 + lane] = rstd;
            }
            const uint32_t rows = aux_base + (AUX == AUX_NONE && plan.one_stage ? 0u : b) * plan.aux_bytes;
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j) {
                const float* y = x + 4 * j;
                const float4 gm = four(g.ln_gamma, j), bt = four(g.ln_beta, j);
                float o[4] = {y[0] * rstd * gm.x + bt.x, y[1] * rstd * gm.y + bt.y, y[2] * rstd * gm.z + bt.z,
                              y[3] * rstd * gm.w + bt.w};
                const uint32_t at = rows + (j >> 3) * HALF_BYTES + sw128(r, j & 7u) + 8u * half;
                if (AUX == AUX_TMA) {
                    uint32_t w0, w1;
                    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(w0), "=r"(w1) : "r"(at) : "memory");
                    o[0] += __uint_as_float(w0 << 16);
                    o[1] += __uint_as_float(w0 & 0xffff0000u);
                    o[2] += __uint_as_float(w1 << 16);
                    o[3] += __uint_as_float(w1 & 0xffff0000u);
                }
                asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(at), "r"(pack2(o[0], o[1])), "r"(pack2(o[2], o[3])) : "memory");
            }
        } else if constexpr (LN) {
            float x[64];
            if (ok) {
                uint32_t v[32];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    tmem_ld32(taddr + 32u * q, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 32; ++j) x[32 * q + j] = g.k ? __uint_as_float(v[j]) : 0.f;
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[b]);
            } else {
#pragma unroll
                for (int j = 0; j < 64; ++j) x[j] = 0.f;
            }
            if (g.bias) {
#pragma unroll
                for (int j = 0; j < 64; j += 8) {
                    float bb[8];
                    if (vec) {
                        load8(bb, g.bias + col0 + j);
                    } else {
#pragma unroll
                        for (int k = 0; k < 8; ++k) bb[k] = g.bias[col0 + j + k];
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k) x[j + k] += bb[k];
                }
            }
            float rstd;
            if (!ln_centre(x, ok, xs, xv, oks, failed, quarter, half, lane, &rstd)) break;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                float o[8];
                if (vec) ln_scale<true>(g.ln_gamma + col0 + 8 * c, g.ln_beta + col0 + 8 * c, x + 8 * c, rstd, o);
                else ln_scale<false>(g.ln_gamma + col0 + 8 * c, g.ln_beta + col0 + 8 * c, x + 8 * c, rstd, o);
                const uint32_t at = stage + sw128(r, (uint32_t)c);
                if (AUX == AUX_TMA) add8(o, lds128(at));
                sts128(at, make_uint4(pack2(o[0], o[1]), pack2(o[2], o[3]), pack2(o[4], o[5]), pack2(o[6], o[7])));
            }
        } else {
#pragma unroll
            for (uint32_t q = 0; q < 2; ++q) {
                uint32_t v[32];
                float x[32];
                tmem_ld32(taddr + 32u * q, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 32; ++j) x[j] = g.k ? __uint_as_float(v[j]) : 0.f;
#pragma unroll
                for (uint32_t c = 0; c < 4; ++c) {
                    float* y = x + 8 * c;
                    const uint32_t at = stage + sw128(r, 4u * q + c);
                    if (g.bias) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) y[k] += bb[k];
                        if (4u * q + c < 7u) load8(bb, s_bias + col0 + 32u * q + 8u * (c + 1u));
                    }
                    if (AUX == AUX_GATHER) {
                        if (g.add1) add8(y, lds128(at));
                        if (g.add2) add8(y, lds128(at + (g.add1 ? AUX_BYTES : 0u)));
                    }
                    if (AUX == AUX_TMA) {  // relu_z
                        const uint4 z = lds128(at);
                        const uint32_t w[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            if (!(__uint_as_float(w[k] << 16) > 0.f)) y[2 * k] = 0.f;
                            if (!(__uint_as_float(w[k] & 0xffff0000u) > 0.f)) y[2 * k + 1] = 0.f;
                        }
                    }
                    if (g.relu) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) y[k] = fmaxf(y[k], 0.f);
                    }
                    if (F32) {
                        const uint32_t f = f32_buf + q * 4096u;  // columns 32 q .. of this warp's 64
                        sts128(f + sw128(lane, 2u * c), make_uint4(__float_as_uint(y[0]), __float_as_uint(y[1]),
                                                                  __float_as_uint(y[2]), __float_as_uint(y[3])));
                        sts128(f + sw128(lane, 2u * c + 1u), make_uint4(__float_as_uint(y[4]), __float_as_uint(y[5]),
                                                                       __float_as_uint(y[6]), __float_as_uint(y[7])));
                    }
                    if (BF) sts128(at, make_uint4(pack2(y[0], y[1]), pack2(y[2], y[3]), pack2(y[4], y[5]), pack2(y[6], y[7])));
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (LN && F32) pair_sync(quarter);  // a box holds both warps' columns
        else __syncwarp();
        if (lane == 0) {
            if (!LN) mbar_arrive(&acc_empty[b]);
            if (row0 < g.m) {
                if (BF && col0 < g.n) tma_store_box(&maps.cb, stage + 32u * quarter * 128u, col0, row0, false);
                if (F32 && col0 < g.n) tma_store_box(&maps.cf, f32_buf, col0, row0, g.accumulate != 0);
                if (F32 && col0 + 32u < g.n) tma_store_box(&maps.cf, f32_buf + 4096u, col0 + 32u, row0, g.accumulate != 0);
            }
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            if (AUX != AUX_NONE && !BF) mbar_arrive(&aux_empty[b]);  // read, and nothing is stored from it
        }
        __syncwarp();
    }
    // the stores have left shared memory before the CTA gives it up
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
}

template <int AUX, bool LN, bool F32, bool BF>
__global__ void __launch_bounds__(TMA_THREADS + (AUX == AUX_GATHER ? 32 * GATHER_WARPS : 0), 1)
    gemm_tma_kernel(const GemmArgs g, const __grid_constant__ TmaMaps maps, const TmaPlan plan, uint32_t* err) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ uint64_t full[TMA_MAX_STAGES], empty[TMA_MAX_STAGES], acc_full[2], acc_empty[2], aux_full[2], aux_empty[2], b_full;
    // LN: the warp pairs' exchanged row sums, squared deviations and wait outcomes
    __shared__ float s_lnx[LN ? 4 : 1][2][32], s_lnv[LN ? 4 : 1][2][32];
    __shared__ int s_lnok[LN ? 4 : 1][2];
    __shared__ __align__(16) float s_bias[LN ? 4 : 128];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_failed;
    volatile int* failed = &s_failed;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t ntiles = (g.m + BM - 1) / BM;
    const uint32_t nslices = (g.k + BK - 1) / BK;
    const uint32_t stages = plan.stages;
    unsigned char* const ring = smem_raw + nslices * TILE_BYTES;
    const uint32_t aux_base = smem_addr(ring) + stages * TILE_BYTES;
    const uint32_t f32_base = aux_base + (plan.one_stage ? 1u : 2u) * plan.aux_bytes;

    if (threadIdx.x == 0) {
        for (uint32_t q = 0; q < stages; ++q) {
            mbar_init(&full[q], 1);
            mbar_init(&empty[q], 1);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(&acc_full[q], 1);
            mbar_init(&acc_empty[q], PIPE_EPILOGUE);
            mbar_init(&aux_full[q], AUX == AUX_GATHER ? 32 * GATHER_WARPS : 1);
            mbar_init(&aux_empty[q], PIPE_EPILOGUE);
        }
        mbar_init(&b_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_failed = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)),
                     "r"(PIPE_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    after_previous();
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // B^T once, then the A slices (and the epilogue's rows) of every tile
            mbar_expect_tx(&b_full, nslices * TILE_BYTES);
            for (uint32_t sl = 0; sl < nslices; ++sl) tma_load_box(&maps.b, smem_raw + sl * TILE_BYTES, sl * BK, 0u, &b_full);
            uint32_t it = 0, t = 0;
            for (uint32_t tile = blockIdx.x; tile < ntiles && !*failed; tile += gridDim.x, ++t) {
                const uint32_t m0 = tile * BM;
                for (uint32_t sl = 0; sl < nslices; ++sl, ++it) {
                    const uint32_t st = it % stages;
                    if (it >= stages && !mbar_wait(smem_addr(&empty[st]), ((it / stages) - 1u) & 1u)) {
                        *failed = 1;
                        break;
                    }
                    mbar_expect_tx(&full[st], TILE_BYTES);
                    if (g.a2 && sl * BK >= g.k_split)
                        tma_load_box(&maps.a2, ring + st * TILE_BYTES, sl * BK - g.k_split, m0, &full[st]);
                    else
                        tma_load_box(&maps.a, ring + st * TILE_BYTES, sl * BK, m0, &full[st]);
                }
                if (AUX == AUX_TMA && !*failed) {
                    const uint32_t b = t & 1u;
                    if (t >= 2 && !mbar_wait(smem_addr(&aux_empty[b]), ((t >> 1) - 1u) & 1u)) {
                        *failed = 1;
                        break;
                    }
                    unsigned char* dst = ring + stages * TILE_BYTES + b * plan.aux_bytes;
                    mbar_expect_tx(&aux_full[b], AUX_BYTES);
                    tma_load_box(&maps.aux, dst, 0u, m0, &aux_full[b]);
                    tma_load_box(&maps.aux, dst + HALF_BYTES, 64u, m0, &aux_full[b]);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // MMA issue (one thread)
        if (lane == 0) {
            uint32_t it = 0, t = 0;
            if (!mbar_wait(smem_addr(&b_full), 0u)) *failed = 1;
            for (uint32_t tile = blockIdx.x; tile < ntiles && !*failed; tile += gridDim.x, ++t) {
                const uint32_t b = t & 1u;
                if (t >= 2 && !mbar_wait(smem_addr(&acc_empty[b]), ((t >> 1) - 1u) & 1u)) {
                    *failed = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc_addr = tmem + b * (uint32_t)BN;
                for (uint32_t sl = 0; sl < nslices; ++sl, ++it) {
                    const uint32_t st = it % stages;
                    if (!mbar_wait(smem_addr(&full[st]), (it / stages) & 1u)) {
                        *failed = 1;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_base = smem_addr(ring + st * TILE_BYTES);
                    const uint32_t b_base = smem_addr(smem_raw + sl * TILE_BYTES);
#pragma unroll
                    for (uint32_t j = 0; j < BK / 16; ++j) {
                        const uint64_t ad = sw128_desc(a_base + 32u * j);
                        const uint64_t bd = sw128_desc(b_base + 32u * j);
                        const uint32_t acc = (sl > 0 || j > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(acc_addr),
                            "l"(ad), "l"(bd), "r"(IDESC), "r"(acc));
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                     smem_addr(&empty[st]))
                                 : "memory");
                }
                if (*failed) break;
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_addr(&acc_full[b]))
                             : "memory");
            }
        }
        __syncwarp();
    } else if (warp < 2u + PIPE_EPILOGUE) {
        // warps 2..9: quarter w % 4 (the accumulator lanes its position in the warpgroup may
        // address), columns 64 ((w - 2) / 4) ..
        if constexpr (AUX == AUX_DIRECT)
            drain_accumulators(g, tmem, acc_full, acc_empty, failed, ntiles, 1u, nslices, warp & 3u, (warp - 2u) / 4u, lane);
        else tma_epilogue<AUX, LN, F32, BF>(g, maps, plan, tmem, acc_full, acc_empty, aux_full, aux_empty, failed, ntiles,
                                       warp & 3u, (warp - 2u) / 4u, lane, aux_base, f32_base, s_bias, s_lnx, s_lnv, s_lnok);
    } else {
        // AUX_GATHER: warp w copies the gathered rows of tile rows 32 w .. + 31, two rows per
        // instruction, 16 lanes of 16 bytes each; every thread's copies arrive on the stage's
        // barrier as they complete. Rows past the matrix are zero-filled.
        const uint32_t r0 = 32u * (warp - 2u - PIPE_EPILOGUE), chunk = lane & 15u;
        const __nv_bfloat16* const src[2] = {g.add1, g.add2};
        const uint32_t* const idx[2] = {g.add1_idx, g.add2_idx};
        uint32_t next[2];  // this lane's row indices, a tile ahead
        auto index = [&](uint32_t tile) {
            const uint32_t row = tile * BM + r0 + lane;
#pragma unroll
            for (int o = 0; o < 2; ++o) next[o] = src[o] && tile < ntiles && row < g.m ? idx[o][row] : 0u;
        };
        index(blockIdx.x);
        uint32_t t = 0;
        for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++t) {
            const uint32_t b = t & 1u, at[2] = {next[0], next[1]};
            index(tile + gridDim.x);
            bool ok = !*failed && (t < 2 || mbar_wait(smem_addr(&aux_empty[b]), ((t >> 1) - 1u) & 1u));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                if (lane == 0) *failed = 1;
                break;
            }
            uint32_t dst = aux_base + b * plan.aux_bytes + (chunk >> 3) * HALF_BYTES;
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                if (!src[o]) continue;
#pragma unroll 8
                for (uint32_t q = 0; q < 16u; ++q) {
                    const uint32_t rr = 2u * q + (lane >> 4);
                    const uint32_t k = __shfl_sync(0xffffffffu, at[o], (int)rr);
                    const uint32_t bytes = tile * BM + r0 + rr < g.m ? 16u : 0u;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + sw128(r0 + rr, chunk & 7u)),
                                 "l"(src[o] + (size_t)k * g.ld_add + 8u * chunk), "r"(bytes)
                                 : "memory");
                }
                dst += AUX_BYTES;
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(&aux_full[b])) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();
    if (*failed && threadIdx.x == 0 && err) atomicOr(err, DEVERR_MMA_TIMEOUT);
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(PIPE_TMEM_COLS));
    }
}

// ---- two layers and a LayerNorm in one kernel (inference) ----------------------------------------
//
// out = LN(relu(A W1 + b1 (+ P[i] + Q[j])) W2 + b2) gamma + beta (+ A), hidden and output width 128, k <= 128. As two
// launches the hidden rows cross memory twice and a message layer reads its edges' rows again as the residual: 1,280
// bytes per edge and layer where this kernel moves 512 (and the gathered rows, from L2).
// A tile of 128 rows passes through a pipeline of warps: warp 0's TMA brings A into one of three slots; warp 1 issues
// the first layer's MMAs; warps 8..15 add the bias and the gathered rows, apply the ReLU and write the hidden rows as
// BF16 into the 128-byte-swizzled K-major layout that warp 2's MMAs of the second layer read; warps 16..23 normalise,
// add the rows that the slot still holds, write the result over them and store it by TMA. Both layers' accumulators
// are double (all 512 TMEM columns). Q's rows are copied by warps 4..7 into the place of the hidden rows; P's are
// read straight into registers: edges are sorted by receiver, so the 32 rows of a warp share one or two of P's,
// which L1 serves (any index is correct). Registers are moved from the copying warps to the normalising ones.
// The arithmetic and its order are those of the two launches (the same results bit for bit).
// 1.85 M edges: 257 us against 203 + 231 in two launches. Bound by L1 (86 %), most of it the loads of bias, gamma and
// beta, which every warp needs for every tile. Slower: both epilogues in one group of eight warps with both gathered
// rows copied, 345 us; FP32 arithmetic in scalar instructions, 312; the constants as kernel parameters (constant
// cache misses), 352; the second layer's columns spread over the lanes so that a thread needs fewer of them, 286.
constexpr uint32_t MLP_SLOTS = 3;
constexpr int MLP_THREADS = 24 * 32;
constexpr uint32_t MLP_TMEM_COLS = 512;
// Registers per thread at launch, and by role (warpgroups 0, 1: 40, 2, 3: 80, 4, 5: 120) in the same total.
constexpr int MLP_REGS = 80;
static_assert(2 * 40 + 2 * 80 + 2 * 120 <= 6 * MLP_REGS, "the roles share what the block was launched with");
constexpr uint32_t mlp_smem(uint32_t nslices) { return (nslices + 2u) * TILE_BYTES + (MLP_SLOTS + 2u) * AUX_BYTES; }

struct MlpMaps {
    CUtensorMap a, w1, w2, c;
};

// max(x, 0) of two BF16 (a NaN gives 0, as fmaxf before the rounding does)
__device__ __forceinline__ uint32_t relu2(uint32_t w) {
    const __nv_bfloat162 h = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&w), __floats2bfloat162_rn(0.f, 0.f));
    return *reinterpret_cast<const uint32_t*>(&h);
}

// The MMAs of one 128 x 128 tile over nslices slices of 64 (operands TILE_BYTES apart), committed to `done`.
__device__ __forceinline__ void mma_tile(uint32_t acc_addr, uint32_t a, uint32_t b, uint32_t nslices, uint64_t* done) {
    for (uint32_t sl = 0; sl < nslices; ++sl) {
#pragma unroll
        for (uint32_t j = 0; j < BK / 16; ++j) {
            const uint64_t ad = sw128_desc(a + sl * TILE_BYTES + 32u * j);
            const uint64_t bd = sw128_desc(b + sl * TILE_BYTES + 32u * j);
            const uint32_t acc = (sl > 0 || j > 0) ? 1u : 0u;
            asm volatile(
                "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(acc_addr),
                "l"(ad), "l"(bd), "r"(IDESC), "r"(acc));
        }
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(done)) : "memory");
}

template <bool MP>
__global__ void __launch_bounds__(MLP_THREADS, 1)
    gemm_mlp_kernel(const MlpArgs g, const __grid_constant__ MlpMaps maps, uint32_t* err) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ uint64_t a_full[MLP_SLOTS], a_empty[MLP_SLOTS], acc1_full[2], acc1_empty[2], acc2_full[2], acc2_empty[2],
        z_full[2], q_full[2], w_full;
    __shared__ float s_lnx[4][2][32], s_lnv[4][2][32];
    __shared__ int s_lnok[4][2];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_failed;
    volatile int* failed = &s_failed;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t ntiles = (g.m + BM - 1) / BM, nslices = (g.k + BK - 1) / BK;
    const uint32_t mine = ntiles > blockIdx.x ? (ntiles - blockIdx.x + gridDim.x - 1u) / gridDim.x : 0u;  // this CTA's tiles
    const uint32_t w1 = smem_addr(smem_raw), w2 = w1 + nslices * TILE_BYTES;
    unsigned char* const slots = smem_raw + (nslices + 2u) * TILE_BYTES;
    const uint32_t z = smem_addr(slots) + MLP_SLOTS * AUX_BYTES;  // two stages of Q's, then the hidden rows

    if (threadIdx.x == 0) {
        for (uint32_t q = 0; q < MLP_SLOTS; ++q) {
            mbar_init(&a_full[q], 1);
            mbar_init(&a_empty[q], 8);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(&acc1_full[q], 1);
            mbar_init(&acc1_empty[q], 8);
            mbar_init(&acc2_full[q], 1);
            mbar_init(&acc2_empty[q], 8);
            mbar_init(&z_full[q], 8);
            mbar_init(&q_full[q], 4 * 32);
        }
        mbar_init(&w_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_failed = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)),
                     "r"(MLP_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    after_previous();
    const uint32_t tmem = tmem_slot;  // layer 1: columns 0 .., 128 ..; layer 2: 256 .., 384 ..

    if (warp < 4u) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (lane == 0 && warp == 0) {
            mbar_expect_tx(&w_full, (nslices + 2u) * TILE_BYTES);
            for (uint32_t sl = 0; sl < nslices; ++sl) tma_load_box(&maps.w1, smem_raw + sl * TILE_BYTES, sl * BK, 0u, &w_full);
            for (uint32_t sl = 0; sl < 2u; ++sl)
                tma_load_box(&maps.w2, smem_raw + (nslices + sl) * TILE_BYTES, sl * BK, 0u, &w_full);
            for (uint32_t t = 0; t < mine && !*failed; ++t) {
                const uint32_t st = t % MLP_SLOTS, u = t / MLP_SLOTS;
                if (u && !mbar_wait(smem_addr(&a_empty[st]), (u - 1u) & 1u)) {
                    *failed = 1;
                    break;
                }
                mbar_expect_tx(&a_full[st], nslices * TILE_BYTES);
                for (uint32_t sl = 0; sl < nslices; ++sl)
                    tma_load_box(&maps.a, slots + st * AUX_BYTES + sl * TILE_BYTES, sl * BK, (blockIdx.x + t * gridDim.x) * BM,
                                 &a_full[st]);
            }
        } else if (lane == 0 && warp == 1) {
            bool ok = mbar_wait(smem_addr(&w_full), 0u);
            for (uint32_t t = 0; t < mine && ok; ++t) {
                const uint32_t b = t & 1u, st = t % MLP_SLOTS;
                ok = !*failed && (t < 2 || mbar_wait(smem_addr(&acc1_empty[b]), ((t >> 1) - 1u) & 1u)) &&
                     mbar_wait(smem_addr(&a_full[st]), (t / MLP_SLOTS) & 1u);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                mma_tile(tmem + b * (uint32_t)BN, smem_addr(slots) + st * AUX_BYTES, w1, nslices, &acc1_full[b]);
            }
            if (!ok) *failed = 1;
        } else if (lane == 0 && warp == 2) {
            bool ok = mbar_wait(smem_addr(&w_full), 0u);
            for (uint32_t t = 0; t < mine && ok; ++t) {
                const uint32_t b = t & 1u;
                ok = !*failed && (t < 2 || mbar_wait(smem_addr(&acc2_empty[b]), ((t >> 1) - 1u) & 1u)) &&
                     mbar_wait(smem_addr(&z_full[b]), (t >> 1) & 1u);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                mma_tile(tmem + (2u + b) * (uint32_t)BN, z + b * AUX_BYTES, w2, 2u, &acc2_full[b]);
            }
            if (!ok) *failed = 1;
        }
        __syncwarp();
    } else if (warp < 8u) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (MP) {
            // Q's rows, two per instruction (16 lanes of 16 bytes each); rows past the matrix are zero-filled
            const uint32_t r0 = 32u * (warp - 4u), chunk = lane & 15u;
            auto index = [&](uint32_t t) {
                const uint32_t row = (blockIdx.x + t * gridDim.x) * BM + r0 + lane;
                return t < mine && row < g.m ? g.add2_idx[row] : 0u;
            };
            uint32_t next = index(0);
            for (uint32_t t = 0; t < mine; ++t) {
                const uint32_t b = t & 1u, row0 = (blockIdx.x + t * gridDim.x) * BM + r0, at = next;
                next = index(t + 1u);
                // the stage's hidden rows of two tiles ago have been read
                bool ok = !*failed && (t < 2 || mbar_wait(smem_addr(&acc2_full[b]), ((t >> 1) - 1u) & 1u));
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) {
                    if (lane == 0) *failed = 1;
                    break;
                }
                const uint32_t dst = z + b * AUX_BYTES + (chunk >> 3) * HALF_BYTES;
#pragma unroll 8
                for (uint32_t q = 0; q < 16u; ++q) {
                    const uint32_t rr = 2u * q + (lane >> 4);
                    const uint32_t k = __shfl_sync(0xffffffffu, at, (int)rr);
                    const uint32_t bytes = row0 + rr < g.m ? 16u : 0u;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + sw128(r0 + rr, chunk & 7u)),
                                 "l"(g.add2 + (size_t)k * 128u + 8u * chunk), "r"(bytes)
                                 : "memory");
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(&q_full[b])) : "memory");
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
    } else if (warp < 16u) {
        const uint32_t quarter = warp & 3u, half = (warp - 8u) / 4u, col0 = 64u * half, r = 32u * quarter + lane;
        auto index = [&](uint32_t t) {
            const uint32_t row = (blockIdx.x + t * gridDim.x) * BM + r;
            return MP && t < mine && row < g.m ? g.add1_idx[row] : 0u;
        };
        uint32_t next = index(0);
        for (uint32_t t = 0; t < mine; ++t) {
            const uint32_t b = t & 1u;
            const uint4* p_row = reinterpret_cast<const uint4*>(g.add1 + (size_t)next * 128u + col0);
            uint4 p[4];
            if (MP) {
#pragma unroll
                for (int c = 0; c < 4; ++c) p[c] = p_row[c];
            }
            next = index(t + 1u);
            bool ok = !*failed && mbar_wait(smem_addr(&acc1_full[b]), (t >> 1) & 1u);
            if (MP) ok = ok && mbar_wait(smem_addr(&q_full[b]), (t >> 1) & 1u);
            else if (t >= 2) ok = ok && mbar_wait(smem_addr(&acc2_full[b]), ((t >> 1) - 1u) & 1u);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                if (lane == 0) *failed = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (uint32_t q = 0; q < 2; ++q) {
                uint32_t v[32];
                float next_b[8];  // eight columns ahead of their use, as the rows of P
                if (g.b1) load8(next_b, g.b1 + col0 + 32u * q);
                tmem_ld32(tmem + ((32u * quarter) << 16) + b * (uint32_t)BN + col0 + 32u * q, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (uint32_t c = 0; c < 4; ++c) {
                    float y[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) y[k] = __uint_as_float(v[8 * c + k]);
                    if (g.b1) {
#pragma unroll
                        for (int k = 0; k < 8; k += 2) add_pair(y + k, next_b[k], next_b[k + 1]);
                        if (c < 3u) load8(next_b, g.b1 + col0 + 32u * q + 8u * (c + 1u));
                    }
                    const uint32_t at = z + b * AUX_BYTES + half * HALF_BYTES + sw128(r, 4u * q + c);
                    if (MP) {
                        add8(y, p[c]);
                        if (q == 0) p[c] = p_row[4 + c];
                        add8(y, lds128(at));
                    }
                    sts128(at, make_uint4(relu2(pack2(y[0], y[1])), relu2(pack2(y[2], y[3])), relu2(pack2(y[4], y[5])), relu2(pack2(y[6], y[7]))));
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&acc1_empty[b]);
                mbar_arrive(&z_full[b]);
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 120;");
        const uint32_t quarter = warp & 3u, half = (warp - 16u) / 4u, col0 = 64u * half, r = 32u * quarter + lane;
        for (uint32_t t = 0; t < mine; ++t) {
            const uint32_t b = t & 1u, st = t % MLP_SLOTS;
            bool ok = !*failed && mbar_wait(smem_addr(&acc2_full[b]), (t >> 1) & 1u) &&
                      mbar_wait(smem_addr(&a_full[st]), (t / MLP_SLOTS) & 1u);
            ok = __all_sync(0xffffffffu, ok);
            if (lane == 0 && t) {  // the previous tile has left its slot
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                mbar_arrive(&a_empty[(t - 1u) % MLP_SLOTS]);
            }
            __syncwarp();
            float x[64];
            if (ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t v[32];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    tmem_ld32(tmem + ((32u * quarter) << 16) + (2u + b) * (uint32_t)BN + col0 + 32u * q, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 32; ++j) x[32 * q + j] = __uint_as_float(v[j]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc2_empty[b]);
            } else {
#pragma unroll
                for (int j = 0; j < 64; ++j) x[j] = 0.f;
            }
            if (g.b2) {
#pragma unroll
                for (int j = 0; j < 64; j += 8) {
                    float bb[8];
                    load8(bb, g.b2 + col0 + j);
#pragma unroll
                    for (int k = 0; k < 8; k += 2) add_pair(x + j + k, bb[k], bb[k + 1]);
                }
            }
            float rstd;
            if (!ln_centre(x, ok, s_lnx, s_lnv, s_lnok, failed, quarter, half, lane, &rstd)) break;
            const uint32_t out = smem_addr(slots) + st * AUX_BYTES + half * HALF_BYTES;
            float gm[8], bt[8];  // eight columns ahead of their use
            load8(gm, g.gamma + col0);
            load8(bt, g.beta + col0);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                float o[8];
#pragma unroll
                for (int k = 0; k < 8; k += 2) {
                    o[k] = x[8 * c + k], o[k + 1] = x[8 * c + k + 1];
                    scale_pair(o + k, rstd, gm[k], gm[k + 1], bt[k], bt[k + 1]);
                }
                if (c < 7) {
                    load8(gm, g.gamma + col0 + 8 * (c + 1));
                    load8(bt, g.beta + col0 + 8 * (c + 1));
                }
                const uint32_t at = out + sw128(r, (uint32_t)c);
                if (MP) add8(o, lds128(at));
                sts128(at, make_uint4(pack2(o[0], o[1]), pack2(o[2], o[3]), pack2(o[4], o[5]), pack2(o[6], o[7])));
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                const uint32_t row0 = (blockIdx.x + t * gridDim.x) * BM + 32u * quarter;
                if (row0 < g.m) tma_store_box(&maps.c, out + 32u * quarter * 128u, col0, row0, false);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            __syncwarp();
        }
        // the stores have left shared memory before the CTA gives it up
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        __syncwarp();
    }
    __syncthreads();
    if (*failed && threadIdx.x == 0 && err) atomicOr(err, DEVERR_MMA_TIMEOUT);
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(MLP_TMEM_COLS));
    }
}

// ---- weight gradients: C = X^T dY, both operands read along their rows ---------------------------
//
// A transposed and B row-major (m, n <= 128; X [k x m], dY [k x n]): a slice of 64 rows of either is
// 64 x 64 boxes that TMA copies into shared memory as they lie, 128 bytes of columns per row,
// 128-byte swizzle, which is the tensor core's MN-major operand layout (8-row groups 1,024 bytes
// apart, the next 64 columns 8,192), so nothing is transposed on the way. One CTA per split of the
// rows, three 32 KB slots, two CTAs per SM: one thread feeds the ring, one issues the MMAs, then
// four warps drain the accumulator. Bound by the operands' bytes: 459,213 rows of 128 + 128 in 248
// splits take 49 us (5.1 TB/s, 75 % of the copy bandwidth) against 127 us with register transposes
// and two synchronous buffers (gemm_kernel, which keeps m or n > 128 and unaligned operands).
constexpr int WG_STAGES = 3;
constexpr uint32_t WG_SLOT = 2u * TILE_BYTES;
constexpr uint32_t WG_SMEM = WG_STAGES * WG_SLOT;

// Shared-memory descriptor of an MN-major operand in the 128-byte swizzle layout.
__device__ __forceinline__ uint64_t sw128_mn_desc(uint32_t saddr) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)(8192u >> 4) << 16;  // the next 64 columns
    d |= (uint64_t)(1024u >> 4) << 32;  // the next 8 rows of K
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

__global__ void __launch_bounds__(THREADS, 2) gemm_wgrad_kernel(const GemmArgs g, const __grid_constant__ CUtensorMap map_a,
                                                                const __grid_constant__ CUtensorMap map_b, uint32_t* err) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ uint64_t full[WG_STAGES], empty[WG_STAGES], done;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_failed;
    volatile int* failed = &s_failed;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t k_begin = blockIdx.x * g.k_chunk, k_end = min(g.k, k_begin + g.k_chunk);
    const uint32_t nslices = (k_end - k_begin + BK - 1) / BK;
    const uint32_t boxes_a = (g.m + 63u) / 64u, boxes_b = (g.n + 63u) / 64u;
    if (threadIdx.x == 0) {
        for (int q = 0; q < WG_STAGES; ++q) {
            mbar_init(&full[q], 1);
            mbar_init(&empty[q], 1);
        }
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_failed = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    after_previous();
    const uint32_t tmem = tmem_slot;
    if (warp == 0 && lane == 0) {
        for (uint32_t it = 0; it < nslices; ++it) {
            const uint32_t st = it % WG_STAGES;
            if (it >= (uint32_t)WG_STAGES && !mbar_wait(smem_addr(&empty[st]), ((it / WG_STAGES) - 1u) & 1u)) {
                *failed = 1;
                break;
            }
            unsigned char* const slot = smem_raw + st * WG_SLOT;
            mbar_expect_tx(&full[st], (boxes_a + boxes_b) * (TILE_BYTES / 2u));
            for (uint32_t q = 0; q < boxes_a; ++q)
                tma_load_box(&map_a, slot + q * (TILE_BYTES / 2u), 64u * q, k_begin + it * BK, &full[st]);
            for (uint32_t q = 0; q < boxes_b; ++q)
                tma_load_box(&map_b, slot + TILE_BYTES + q * (TILE_BYTES / 2u), 64u * q, k_begin + it * BK, &full[st]);
        }
    } else if (warp == 1 && lane == 0) {
        // both operands MN-major (bits 15 and 16), N the columns rounded up to 16; accumulator rows and
        // columns past the matrix hold whatever their operands' places did and are not read
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                               (((g.n + 15u) / 16u * 2u) << 17) | ((uint32_t)(BM >> 4) << 24);
        for (uint32_t it = 0; it < nslices; ++it) {
            const uint32_t st = it % WG_STAGES;
            if (!mbar_wait(smem_addr(&full[st]), (it / WG_STAGES) & 1u)) {
                *failed = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t base = smem_addr(smem_raw + st * WG_SLOT);
#pragma unroll
            for (uint32_t j = 0; j < BK / 16; ++j) {
                const uint64_t ad = sw128_mn_desc(base + 2048u * j);
                const uint64_t bd = sw128_mn_desc(base + TILE_BYTES + 2048u * j);
                const uint32_t acc = (it > 0 || j > 0) ? 1u : 0u;
                asm volatile(
                    "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                    " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_addr(&empty[st]))
                         : "memory");
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(&done))
                     : "memory");
    }
    __syncwarp();
    const bool ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&done), 0u));
    if (!ok) *failed = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    const bool bad = *failed != 0;
    if (bad && threadIdx.x == 0 && err) atomicOr(err, DEVERR_MMA_TIMEOUT);
    const uint32_t row = 32u * warp + lane;
    for (uint32_t c0 = 0; c0 < g.n; c0 += 32u) {
        uint32_t v[32];
        tmem_ld32(tmem + ((32u * warp) << 16) + c0, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (row >= g.m || bad) continue;
        float x[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(v[j]);
        epilogue_store(g, x, row, c0, min(32u, g.n - c0), blockIdx.x, g.add1 ? g.add1_idx[row] : 0u,
                       g.add2 ? g.add2_idx[row] : 0u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

}  // namespace

// 64 KB of operand buffers: at most three CTAs per SM, 3 x 128 of the SM's 512 columns of
// tensor memory, so tcgen05.alloc never has to wait for another CTA.
size_t gemm_smem_bytes() { return 65u * 1024u; }

wc_status check_gemm(const GemmArgs& g) {
    if (g.m == 0 || g.n == 0) return WC_OK;
    if (!g.a || !g.b || (!g.c_f32 && !g.c_bf16)) return fail(WC_ERR_INVALID_ARG, "gemm: null operand");
    if (!g.a_transposed && (g.lda % 8 || (g.a2 && (g.lda2 % 8 || g.k_split % 8))))
        return fail(WC_ERR_INVALID_ARG, "gemm: row-major A needs 16-byte aligned rows (lda %% 8 == 0)");
    if (g.a_transposed && (g.lda % 8 || g.m % 8)) return fail(WC_ERR_INVALID_ARG, "gemm: transposed A needs m, lda %% 8 == 0");
    if (!g.b_rowmajor && g.ldb % 8) return fail(WC_ERR_INVALID_ARG, "gemm: B^T rows need ldb %% 8 == 0");
    if (g.b_rowmajor && (g.ldb % 8 || g.n % 8)) return fail(WC_ERR_INVALID_ARG, "gemm: row-major B needs n, ldb %% 8 == 0");
    // Both operands staged along k (transposed A, row-major B) read single k rows: any k works.
    if (g.k % 8 && !(g.a_transposed && g.b_rowmajor))
        return fail(WC_ERR_INVALID_ARG, "gemm: k must be a multiple of 8 (pad with zeros)");
    if ((g.add1 && !g.add1_idx) || (g.add2 && !g.add2_idx)) return fail(WC_ERR_INVALID_ARG, "gemm: gather without index");
    if (g.k_chunk == 0 || g.k_chunk % BK) return fail(WC_ERR_INVALID_ARG, "gemm: k_chunk must be a multiple of 64");
    if (g.ln_gamma && (g.n != 128u || !g.ln_beta || !g.c_bf16 || (g.c_f32 && !(g.ln_mean && g.ln_rstd && g.k <= 128u)) || g.relu || g.add1 || g.add2 ||
                       g.accumulate || g.ldc != 128u || g.a_rows || g.a2 || g.a_transposed || g.b_rowmajor ||
                       g.k_chunk < g.k))
        return fail(WC_ERR_INVALID_ARG,
                    "gemm: the LayerNorm epilogue needs n = ldc = 128, beta, a BF16 output only and plain operands");
    if (g.relu_z && (g.n != 128u || !g.c_bf16 || !g.c_f32 || g.ln_gamma || g.relu || g.add1 || g.add2 || g.accumulate ||
                     g.a_rows || g.a2 || g.a_transposed || g.b_rowmajor || g.k > 128u || g.k_chunk < g.k))
        return fail(WC_ERR_INVALID_ARG, "gemm: the ReLU mask epilogue needs n = 128, k <= 128, both outputs and plain operands");
    return WC_OK;
}

// Dynamic shared memory of gemm_pipe_kernel<RB> for k (RB: the resident B slices and the ring).
size_t pipe_smem_bytes(bool rb, uint32_t k) {
    const uint32_t nslices = (k + BK - 1) / BK;
    return rb ? (size_t)(nslices + PipeShape<true>::STAGES) * TILE_BYTES
              : (size_t)PipeShape<false>::STAGES * 2u * TILE_BYTES;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (null when unavailable: the
// cp.async kernel then serves every shape).
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
    static const EncodeTiledFn fn = []() -> EncodeTiledFn {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// A 2-D row-major tensor [outer x inner] of BF16 (or FP32) with rows `stride_bytes` apart, accessed in
// boxes of 128 bytes x `rows` rows with the 128-byte swizzle, out-of-range elements read as zeros.
bool encode_operand(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint64_t stride_bytes,
                    uint32_t rows = BM, bool f32 = false) {
    const EncodeTiledFn fn = encode_tiled();
    if (!fn || reinterpret_cast<uintptr_t>(base) % 16u || stride_bytes % 16u || inner == 0 || outer == 0) return false;
    const cuuint64_t dims[2] = {inner, outer};
    const cuuint64_t strides[1] = {stride_bytes};
    const cuuint32_t box[2] = {f32 ? 32u : 64u, rows};
    const cuuint32_t elem[2] = {1, 1};
    return fn(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base),
              dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int sm_count() {
    static const int sms = [] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return n > 0 ? n : 1;
    }();
    return sms;
}

bool gemm_tma_available() { return encode_tiled() != nullptr; }

namespace {

template <int AUX, bool LN, bool F32, bool BF>
wc_status launch_tma_as(const GemmArgs& g, const TmaMaps& maps, const TmaPlan& plan, uint32_t grid, uint32_t* err,
                        cudaStream_t s) {
    static std::once_flag once;
    std::call_once(once, [] {
        cudaFuncSetAttribute(gemm_tma_kernel<AUX, LN, F32, BF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)TMA_SMEM_LIMIT);
    });
    const int threads = TMA_THREADS + (AUX == AUX_GATHER ? 32 * GATHER_WARPS : 0);
    launch_after(gemm_tma_kernel<AUX, LN, F32, BF>, grid, threads, plan.smem, s, g, maps, plan, err);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(WC_ERR_CUDA, "gemm launch: %s", cudaGetErrorString(e));
    return WC_OK;
}

// The TMA kernel for row-major A (or [A | A2] split at a whole slice: the node layers' 65,536 x 256 take
// 33 us with cp.async), n <= 128 and k <= 384, when every operand it moves by TMA has a
// tensor map (16-byte aligned base and rows). Its epilogue through shared memory needs tensor maps for the results
// too, whole and aligned gathered rows (n = 128) and room for at least two A slots (all but k > 256 with two gathered
// operands, or with FP32 and BF16 outputs together). The other forms write from the registers, a row per thread
// (AUX_DIRECT), and so do results of at most eight columns or of 32 in BF16 alone, whose rows a thread writes in a few
// whole accesses (460,000 rows, k = 16: 21.4 us against 25.6 at n = 8, 23.3 against 26.3 at n = 32; but 46 against 26
// at n = 16, and 47 against 27 where FP32 results are added to). With cp.async operands instead of TMA's, two gathered
// operands at k = 384 take 103 us per 200,000 rows (75 so), at n = 64 49 (37).
wc_status launch_tma(const GemmArgs& g, uint32_t grid, uint32_t* err, cudaStream_t s, bool* launched) {
    *launched = false;
    const bool gather = g.add1 || g.add2, aux = gather || g.ln_resid || g.relu_z, f32 = g.c_f32 != nullptr, bf = g.c_bf16 != nullptr;
    TmaMaps maps;
    if (g.a2 && (g.k_split % BK || g.k_split >= g.k || !encode_operand(&maps.a2, g.a2, g.k - g.k_split, g.m, 2ull * g.lda2)))
        return WC_OK;
    if (!encode_operand(&maps.a, g.a, g.a2 ? g.k_split : g.k, g.m, 2ull * g.lda) || !encode_operand(&maps.b, g.b, g.k, g.n, 2ull * g.ldb))
        return WC_OK;
    const uint32_t nslices = (g.k + BK - 1) / BK;
    TmaPlan plan{};
    plan.aux_bytes = (g.add1 && g.add2) ? 2u * AUX_BYTES : (aux || bf) ? AUX_BYTES : 0u;
    plan.f32_bytes = f32 ? F32_OUT_BYTES : 0u;
    // a second output stage only where it leaves the whole ring: at k = 384 it takes two of six slots (460,000 rows 81
    // us against 74, 82 before the output went through shared memory); up to k = 256 both fit
    plan.one_stage = !aux && bf &&
                     nslices * TILE_BYTES + 2u * plan.aux_bytes + plan.f32_bytes + TMA_MAX_STAGES * TILE_BYTES > TMA_SMEM_LIMIT;
    const uint32_t fixed = nslices * TILE_BYTES + (plan.one_stage ? 1u : 2u) * plan.aux_bytes + plan.f32_bytes;
    const bool narrow = !aux && !g.accumulate && (g.n <= 8u || (g.n == 32u && !f32)) && !g.ln_gamma;
    const bool shared = !narrow && fixed + 2u * TILE_BYTES <= TMA_SMEM_LIMIT &&
                        (!bf || encode_operand(&maps.cb, g.c_bf16, g.n, g.m, 2ull * g.ldc, 32)) &&
                        (!f32 || encode_operand(&maps.cf, g.c_f32, g.n, g.m, 4ull * g.ldc, 32, true)) &&
                        (!g.ln_resid || encode_operand(&maps.aux, g.ln_resid, 128, g.m, 256)) &&
                        (!g.relu_z || encode_operand(&maps.aux, g.relu_z, 128, g.m, 256)) &&
                        !(gather && (g.n != 128u || g.ld_add % 8u || reinterpret_cast<uintptr_t>(g.add1) % 16u ||
                                     reinterpret_cast<uintptr_t>(g.add2) % 16u));
    if (!shared) {
        if (g.ln_gamma || g.relu_z) return WC_OK;
        plan = TmaPlan{};
        plan.stages = TMA_MAX_STAGES;
        plan.smem = (nslices + TMA_MAX_STAGES) * TILE_BYTES;
        *launched = true;
        return launch_tma_as<AUX_DIRECT, false, false, false>(g, maps, plan, grid, err, s);
    }
    plan.stages = std::min<uint32_t>(TMA_MAX_STAGES, (TMA_SMEM_LIMIT - fixed) / TILE_BYTES);
    plan.smem = fixed + plan.stages * TILE_BYTES;
    *launched = true;
    if (g.ln_gamma && f32)
        return aux ? launch_tma_as<AUX_TMA, true, true, true>(g, maps, plan, grid, err, s)
                   : launch_tma_as<AUX_NONE, true, true, true>(g, maps, plan, grid, err, s);
    if (g.ln_gamma)
        return aux ? launch_tma_as<AUX_TMA, true, false, true>(g, maps, plan, grid, err, s)
                   : launch_tma_as<AUX_NONE, true, false, true>(g, maps, plan, grid, err, s);
    if (g.relu_z) return launch_tma_as<AUX_TMA, false, true, true>(g, maps, plan, grid, err, s);
    if (gather)
        return f32 ? (bf ? launch_tma_as<AUX_GATHER, false, true, true>(g, maps, plan, grid, err, s)
                         : launch_tma_as<AUX_GATHER, false, true, false>(g, maps, plan, grid, err, s))
                   : launch_tma_as<AUX_GATHER, false, false, true>(g, maps, plan, grid, err, s);
    return f32 ? (bf ? launch_tma_as<AUX_NONE, false, true, true>(g, maps, plan, grid, err, s)
                     : launch_tma_as<AUX_NONE, false, true, false>(g, maps, plan, grid, err, s))
               : launch_tma_as<AUX_NONE, false, false, true>(g, maps, plan, grid, err, s);
}

template <bool MP>
wc_status launch_mlp_as(const MlpArgs& g, const MlpMaps& maps, uint32_t* err, cudaStream_t s, bool* launched) {
    // the roles' register shares assume MLP_REGS per thread at launch
    static const bool usable = [] {
        cudaFuncAttributes a{};
        return cudaFuncGetAttributes(&a, gemm_mlp_kernel<MP>) == cudaSuccess && a.numRegs == MLP_REGS &&
               cudaFuncSetAttribute(gemm_mlp_kernel<MP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp_smem(2u)) ==
                   cudaSuccess;
    }();
    if (!usable) return WC_OK;
    const uint32_t tiles = (g.m + BM - 1) / BM, sms = (uint32_t)sm_count();
    launch_after(gemm_mlp_kernel<MP>, std::min(tiles, sms), MLP_THREADS, mlp_smem((g.k + BK - 1) / BK), s, g, maps, err);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(WC_ERR_CUDA, "mlp launch: %s", cudaGetErrorString(e));
    *launched = true;
    return WC_OK;
}

}  // namespace

wc_status launch_mlp(const MlpArgs& g, uint32_t* err, cudaStream_t s, bool* launched) {
    *launched = false;
    const auto at16 = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16u == 0; };
    MlpMaps maps;
    if (!g.m || g.k % 8u || g.k == 0 || g.k > 128u || (g.add1 && g.k != 128u) || !at16(g.b1) || !at16(g.b2) || !at16(g.gamma) ||
        !at16(g.beta) || !at16(g.add1) || !at16(g.add2) || !encode_operand(&maps.a, g.a, g.k, g.m, 2ull * g.k) ||
        !encode_operand(&maps.w1, g.w1, g.k, 128, 2ull * g.k) || !encode_operand(&maps.w2, g.w2, 128, 128, 256) ||
        !encode_operand(&maps.c, g.out, 128, g.m, 256, 32))
        return WC_OK;
    return g.add1 ? launch_mlp_as<true>(g, maps, err, s, launched) : launch_mlp_as<false>(g, maps, err, s, launched);
}

wc_status launch_gemm(const GemmArgs& g, uint32_t* err, cudaStream_t s) {
    const wc_status st = check_gemm(g);
    if (st != WC_OK || g.m == 0 || g.n == 0) return st;
    if (!g.a_transposed && !g.b_rowmajor && g.k_chunk >= g.k) {
        // row-major operands, no split of K: the persistent pipelined kernel, one CTA per SM;
        // B resident in shared memory when it is one column of tiles of at most RB_MAX_SLICES
        static std::once_flag pipe_once;
        const int sms = sm_count();
        std::call_once(pipe_once, [] {
            cudaFuncSetAttribute(gemm_pipe_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)pipe_smem_bytes(false, 0));
            cudaFuncSetAttribute(gemm_pipe_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)pipe_smem_bytes(true, RB_MAX_SLICES * BK));
        });
        const uint32_t tiles = ((g.m + BM - 1) / BM) * ((g.n + BN - 1) / BN);
        const uint32_t grid = tiles < (uint32_t)sms ? tiles : (uint32_t)sms;
        const bool rb = g.n <= (uint32_t)BN && (g.k + BK - 1) / BK <= RB_MAX_SLICES;
        if (rb && !g.a_rows) {
            bool launched = false;
            WC_TRY(launch_tma(g, grid, err, s, &launched));
            if (launched) return WC_OK;
        }
        if (g.relu_z) return fail(WC_ERR_STATE, "gemm: the ReLU mask epilogue needs the TMA kernel (plain A, k <= 128)");
        if (g.ln_gamma) return fail(WC_ERR_STATE, "gemm: the LayerNorm epilogue needs the TMA kernel (plain A, k <= 384)");
        if (rb)
            gemm_pipe_kernel<true><<<grid, PIPE_THREADS, pipe_smem_bytes(true, g.k), s>>>(g, err);
        else
            gemm_pipe_kernel<false><<<grid, PIPE_THREADS, pipe_smem_bytes(false, g.k), s>>>(g, err);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return fail(WC_ERR_CUDA, "gemm launch: %s", cudaGetErrorString(e));
        return WC_OK;
    }
    if (g.a_transposed && g.b_rowmajor && g.m <= (uint32_t)BM && g.n <= (uint32_t)BN && g.k && !g.a2 && !g.a_rows) {
        // the weight-gradient kernel where both operands have tensor maps
        CUtensorMap ma, mb;
        if (encode_operand(&ma, g.a, g.m, g.k, 2ull * g.lda, 64) && encode_operand(&mb, g.b, g.n, g.k, 2ull * g.ldb, 64)) {
            static std::once_flag once;
            std::call_once(once, [] {
                cudaFuncSetAttribute(gemm_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WG_SMEM);
            });
            launch_after(gemm_wgrad_kernel, (g.k + g.k_chunk - 1) / g.k_chunk, THREADS, WG_SMEM, s, g, ma, mb, err);
            const cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) return fail(WC_ERR_CUDA, "gemm launch: %s", cudaGetErrorString(e));
            return WC_OK;
        }
    }
    static bool attr_done = false;
    if (!attr_done) {
        cudaFuncSetAttribute(gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem_bytes());
        attr_done = true;
    }
    const dim3 grid((g.m + BM - 1) / BM, (g.n + BN - 1) / BN, (g.k + g.k_chunk - 1) / g.k_chunk);
    gemm_kernel<<<grid, THREADS, gemm_smem_bytes(), s>>>(g, err);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(WC_ERR_CUDA, "gemm launch: %s", cudaGetErrorString(e));
    return WC_OK;
}

}  // namespace nn
}  // namespace wc

extern "C" WC_API wc_status wc_nn_gemm(const wc_gemm_desc* d, uint32_t* d_err, void* stream) {
    wc::clear_error();
    if (!d) return wc::fail(WC_ERR_INVALID_ARG, "wc_nn_gemm: null descriptor");
    wc::nn::GemmArgs g{};
    g.m = d->m;
    g.n = d->n;
    g.k = d->k;
    g.k_chunk = d->k_chunk;
    g.a = static_cast<const __nv_bfloat16*>(d->a);
    g.a2 = static_cast<const __nv_bfloat16*>(d->a2);
    g.a_rows = d->a_rows;
    g.lda = d->lda;
    g.lda2 = d->lda2;
    g.k_split = d->k_split;
    g.a_transposed = d->a_transposed;
    g.b = static_cast<const __nv_bfloat16*>(d->b);
    g.ldb = d->ldb;
    g.b_rowmajor = d->b_rowmajor;
    g.bias = d->bias;
    g.add1 = static_cast<const __nv_bfloat16*>(d->add1);
    g.add1_idx = d->add1_idx;
    g.add2 = static_cast<const __nv_bfloat16*>(d->add2);
    g.add2_idx = d->add2_idx;
    g.ld_add = d->ld_add;
    g.relu = d->relu;
    g.c_f32 = d->c_f32;
    g.accumulate = d->accumulate;
    g.c_bf16 = static_cast<__nv_bfloat16*>(d->c_bf16);
    g.ldc = d->ldc;
    g.split_stride = d->split_stride;
    g.ln_gamma = d->ln_gamma;
    g.ln_beta = d->ln_beta;
    g.ln_resid = static_cast<const __nv_bfloat16*>(d->ln_resid);
    return wc::nn::launch_gemm(g, d_err, static_cast<cudaStream_t>(stream));
}

extern "C" WC_API wc_status wc_nn_mlp(const wc_mlp_desc* d, uint32_t* d_err, void* stream, int* launched) {
    wc::clear_error();
    if (!d || !launched) return wc::fail(WC_ERR_INVALID_ARG, "wc_nn_mlp: null argument");
    *launched = 0;
    if (!d->m) return WC_OK;
    if (!d->a || !d->w1 || !d->w2 || !d->gamma || !d->beta || !d->out) return wc::fail(WC_ERR_INVALID_ARG, "wc_nn_mlp: null operand");
    if (!d->add1 != !d->add2 || (d->add1 && (!d->add1_idx || !d->add2_idx)))
        return wc::fail(WC_ERR_INVALID_ARG, "wc_nn_mlp: both gathered operands with their indices, or neither");
    using Row = const __nv_bfloat16*;
    wc::nn::MlpArgs g{};
    g.m = d->m;
    g.k = d->k;
    g.a = static_cast<Row>(d->a);
    g.w1 = static_cast<Row>(d->w1);
    g.w2 = static_cast<Row>(d->w2);
    g.b1 = d->b1;
    g.b2 = d->b2;
    g.gamma = d->gamma;
    g.beta = d->beta;
    g.add1 = static_cast<Row>(d->add1);
    g.add1_idx = d->add1_idx;
    g.add2 = static_cast<Row>(d->add2);
    g.add2_idx = d->add2_idx;
    g.out = static_cast<__nv_bfloat16*>(d->out);
    bool ran = false;
    const wc_status st = wc::nn::launch_mlp(g, d_err, static_cast<cudaStream_t>(stream), &ran);
    *launched = ran ? 1 : 0;
    return st;
}
