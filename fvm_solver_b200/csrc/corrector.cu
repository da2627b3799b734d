// Learned k-step corrector: BF16 tcgen05 GEMMs (FP32 accumulation in TMEM), message passing over
// the mesh adjacency, SiLU, MSE loss and Adam -- forward, backward and optimiser all hand-written.
//
// GEMM form used throughout:  D[M][N] = epilogue(A[M][K] . B[N][K]^T)
//   A, B: bf16, row-major, K contiguous ("K-major" for both UMMA operands); M any (128-row tiles,
//   rows past M read as zero and are not stored); N in {32, 64, 128, 256}; K a multiple of 64.
// One CTA of 128 threads computes one 128 x N tile:
//   * the K loop stages 64-wide slices of A and B in shared memory in the canonical no-swizzle
//     K-major core-matrix layout (8 rows x 16 bytes per core matrix; the two 16-byte K halves of an
//     MMA step LBO = 128 B apart; 8-row groups SBO = 256 B apart);
//   * one elected thread issues tcgen05.mma.cta_group::1.kind::f16 (M = 128, N, K = 16) four times
//     per slice and tcgen05.commit's completion to an mbarrier, which all threads wait on with an
//     iteration limit (a timeout sets the error flag instead of hanging);
//   * the accumulator lives in tensor memory (N fp32 columns x 128 lanes, allocated per CTA); the
//     epilogue reads it back with tcgen05.ld (warp w owns lanes 32w..32w+31 = rows of the tile),
//     adds the bias, stores the pre-activation if asked, applies SiLU, adds a residual, and writes
//     fp32 and/or bf16.
// Split-K (for weight gradients, K = number of cells): `k_splits` > 1 makes each CTA handle one
// K range and atomically add its fp32 tile into D (no epilogue other than the add).
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include <algorithm>

#include "fvm_common.cuh"

namespace fvm {
namespace corr {

constexpr int TM = 128;          // tile rows (UMMA M)
constexpr int TK = 64;           // K slice staged per iteration
constexpr int kGemmThreads = 128;
constexpr long long kWaitLimit = 1LL << 22;   // mbarrier polls before a wait gives up

struct GemmArgs {
    const __nv_bfloat16* A;
    int64_t lda;
    const __nv_bfloat16* B;
    int64_t ldb;
    int M, N, K;
    int k_splits;                 // > 1: split-K with atomic accumulation into Df
    const float* bias;            // [N] or null
    const float* resid;           // [M][ldr] fp32 added after the activation, or null
    int64_t ldr;
    float* Df;                    // [M][ldd] fp32 output (or accumulation target), or null
    __nv_bfloat16* Db;            // [M][ldd] bf16 output, or null
    int64_t ldd;
    float* preact;                // [M][ldd] fp32 pre-activation, or null
    int act;                      // 0 none, 1 SiLU
    int* err;                     // device error flag (set to 1 on an mbarrier timeout)
    int vec;                      // every epilogue row chunk is 32-byte aligned: 256-bit accesses
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// UMMA shared-memory matrix descriptor: no swizzle, K-major, version 1 (sm100).
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;       // descriptor version for tcgen05
    return d;                      // base offset 0, lbo mode 0, layout type 0 (no swizzle)
}

// Instruction descriptor of kind::f16: D fp32, A and B bf16, both K-major, M = 128.
__host__ __device__ constexpr uint32_t make_idesc(int N) {
    return (1u << 4)                      // D format: F32
           | (1u << 7)                    // A format: BF16
           | (1u << 10)                   // B format: BF16
           | ((uint32_t)(N >> 3) << 17)   // N / 8
           | ((uint32_t)(TM >> 4) << 24); // M / 16
}

// Stage rows [r0, r0 + nrows) x K columns [k0, k0 + 64) of a row-major bf16 matrix into the
// core-matrix layout: 16-byte unit (row r, unit u of 8 K elements) -> slice u/2, half u%2.
__device__ __forceinline__ void stage_tile(uint8_t* smem, const __nv_bfloat16* src, int64_t ld, int r0, int rows_valid,
                                           int nrows, int k0, int kmax) {
    const int units = nrows * (TK / 8);
    const int slice_bytes = (nrows / 8) * 256;
    for (int t = threadIdx.x; t < units; t += blockDim.x) {
        const int r = t >> 3, u = t & 7;
        const int k = k0 + 8 * u;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (r < rows_valid && k < kmax) v = *reinterpret_cast<const uint4*>(src + (int64_t)(r0 + r) * ld + k);
        const int off = (u >> 1) * slice_bytes + (r >> 3) * 256 + (u & 1) * 128 + (r & 7) * 16;
        *reinterpret_cast<uint4*>(smem + off) = v;
    }
}

// Same layout as stage_tile, copied global -> shared by cp.async (no registers; rows past
// rows_valid and columns past kmax are zero-filled).  Thread -> (row, unit) mapping: the 32 lanes
// of a warp take 8 consecutive rows x 4 units, so their 16-byte stores cover all 32 banks once per
// 8 lanes (conflict-free) and each row's 4 units are 64 contiguous global bytes.
__device__ __forceinline__ void stage_tile_async(uint8_t* smem, const __nv_bfloat16* src, int64_t ld, int r0,
                                                 int rows_valid, int nrows, int k0, int kmax) {
    const int units = nrows * (TK / 8);
    const int slice_bytes = (nrows / 8) * 256;
    const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    for (int t = threadIdx.x; t < units; t += blockDim.x) {
        const int r = (t & 7) + 8 * (t >> 6), u = (t >> 3) & 7;
        const int k = k0 + 8 * u;
        const bool valid = r < rows_valid && k < kmax;
        const __nv_bfloat16* gp = valid ? src + (int64_t)(r0 + r) * ld + k : src;
        const uint32_t off = (uint32_t)((u >> 1) * slice_bytes + (r >> 3) * 256 + (u & 1) * 128 + (r & 7) * 16);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + off), "l"(gp),
                     "r"(valid ? 16 : 0)
                     : "memory");
    }
}

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done = 0;
    for (long long it = 0; it < kWaitLimit && !done; ++it) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(bar))), "r"(parity));
    }
    return done != 0;
}

// z sigmoid(z) with the fast-division intrinsic: the denominator is >= 1, so the intrinsic's range
// limit only matters where exp overflows and the quotient is 0 anyway (within 2 ulp elsewhere).
// Every residual added to it goes through __fadd_rn, so no kernel fuses the quotient's multiply
// with that add and all kernels round alike (the fused layer equals GEMM + epilogue bitwise).
__device__ __forceinline__ float silu(float z) { return __fdividef(z, 1.f + __expf(-z)); }

// 8 consecutive floats (32-byte aligned) with one 256-bit access.
__device__ __forceinline__ void ld8(const float* p, float* v) {
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}
__device__ __forceinline__ void st8(float* p, const float* v) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

// Epilogue of 32 consecutive accumulator columns [c0, c0 + 32) of one row with 256-bit accesses:
// each thread reads and writes whole 32-byte sectors of its own row (no partial-sector traffic).
__device__ __forceinline__ void epilogue_vec(const GemmArgs& g, int64_t row, int c0, const uint32_t (&r)[32]) {
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
    if (g.bias) {
        float b[32];
#pragma unroll
        for (int q = 0; q < 4; ++q) ld8(g.bias + c0 + 8 * q, b + 8 * q);
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] += b[j];
    }
    if (g.preact)
#pragma unroll
        for (int q = 0; q < 4; ++q) st8(g.preact + row * g.ldd + c0 + 8 * q, v + 8 * q);
    if (g.act == 1)
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = silu(v[j]);
    if (g.resid) {
        float x[32];
#pragma unroll
        for (int q = 0; q < 4; ++q) ld8(g.resid + row * g.ldr + c0 + 8 * q, x + 8 * q);
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __fadd_rn(v[j], x[j]);
    }
    if (g.Df)
#pragma unroll
        for (int q = 0; q < 4; ++q) st8(g.Df + row * g.ldd + c0 + 8 * q, v + 8 * q);
    if (g.Db) {
        float pk[16];   // bf16 pairs, bit patterns carried in float registers
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
            pk[j] = __uint_as_float(*reinterpret_cast<const uint32_t*>(&h));
        }
        float* dst = reinterpret_cast<float*>(g.Db + row * g.ldd + c0);
        st8(dst, pk);
        st8(dst + 8, pk + 8);
    }
}

template <int N>
__global__ void __launch_bounds__(kGemmThreads) k_gemm(GemmArgs g) {
    // Two staging buffers of one K slice each (A: TM x TK, B: N x TK, bf16): slice j + 1 is copied
    // (cp.async) while the tensor cores work on slice j; a buffer is refilled only after the MMAs
    // that read it have completed (their commit's mbarrier).
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int kStageBytes = TM * TK * 2 + N * TK * 2;
    __shared__ __align__(8) uint64_t mbar[2];
    __shared__ uint32_t s_taddr;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * TM;
    const int split = blockIdx.y;
    const int kchunks = g.K / TK;
    const int per = (kchunks + g.k_splits - 1) / g.k_splits;
    const int kc0 = split * per, kc1 = min(kchunks, kc0 + per);
    const int nk = max(0, kc1 - kc0);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_taddr)),
                     "r"((uint32_t)(N < 32 ? 32 : N)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[0])));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[1])));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t taddr = s_taddr;
    const uint32_t idesc = make_idesc(N);
    const int rows_a = min(TM, g.M - m0);
    // The epilogue's residual rows (one contiguous block of the tile's rows) go to L2 while the
    // tile is loaded and multiplied: the bulk-copy unit prefetches them, so the epilogue's loads
    // see L2 latency instead of DRAM latency.
    if (threadIdx.x == 0 && g.resid && g.k_splits == 1 && g.vec && rows_a > 0) {
        const uint32_t bytes = (uint32_t)((int64_t)rows_a * g.ldr * 4) & ~15u;
        if (bytes) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(g.resid + (int64_t)m0 * g.ldr),
                                "r"(bytes) : "memory");
    }
    auto stage = [&](int buf, int kc) {
        uint8_t* sA = smem + buf * kStageBytes;
        stage_tile_async(sA, g.A, g.lda, m0, rows_a, TM, kc * TK, g.K);
        stage_tile_async(sA + TM * TK * 2, g.B, g.ldb, 0, g.N, N, kc * TK, g.K);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    bool ok = true;
    for (int j = 0; j < min(2, nk); ++j) stage(j, kc0 + j);
    for (int j = 0; j < nk && ok; ++j) {
        const int buf = j & 1;
        if (j + 1 < nk) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t sa = smem_u32(smem + buf * kStageBytes), sb = sa + TM * TK * 2;
#pragma unroll
            for (int s = 0; s < TK / 16; ++s) {
                const uint64_t ad = make_desc(sa + s * (TM / 8) * 256, 128, 256);
                const uint64_t bd = make_desc(sb + s * (N / 8) * 256, 128, 256);
                const uint32_t acc = (j > 0 || s > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(taddr),
                    "l"(ad), "l"(bd), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&mbar[buf]))
                         : "memory");
        }
        // Refill this buffer with slice j + 2 once its MMAs are done; after the last slice, wait
        // for the last commit (the MMAs of one thread complete in order).
        const bool refill = j + 2 < nk, last = j + 1 == nk;
        if (refill || last) {                              // uniform across the block
            bool done = mbar_wait(&mbar[buf], (uint32_t)((j >> 1) & 1));
            if (!done) {
                // Give the MMAs in flight a second bounded chance to finish before the tensor memory
                // they write is released; the timeout is reported below.
                done = mbar_wait(&mbar[buf], (uint32_t)((j >> 1) & 1)) && false;
            }
            // one verdict for the whole block (also the barrier before the buffer is refilled)
            ok = __syncthreads_and(done) != 0;
            if (!ok) {
                if (threadIdx.x == 0 && g.err) atomicExch(g.err, 1);
            } else if (refill) {
                stage(buf, kc0 + j + 2);
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("tcgen05.fence::after_thread_sync;");
    const bool have = ok && kc1 > kc0;
    // Epilogue: warp w owns tile rows 32w .. 32w + 31 (TMEM lanes).
    const int row = m0 + warp * 32 + lane;
    if (have) {
#pragma unroll 1
        for (int c0 = 0; c0 < N; c0 += 32) {
            uint32_t r[32];
            const uint32_t a = taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                  "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
                  "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
                  "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                : "r"(a));
            asm volatile("tcgen05.wait::ld.sync.aligned;");
            if (row < g.M && g.vec && g.k_splits == 1) {
                epilogue_vec(g, row, c0, r);
            } else if (row < g.M) {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const int col = c0 + j;
                    if (col >= g.N) break;
                    float v = __uint_as_float(r[j]);
                    if (g.k_splits > 1) {
                        atomicAdd(g.Df + (int64_t)row * g.ldd + col, v);
                        continue;
                    }
                    if (g.bias) v += g.bias[col];
                    if (g.preact) g.preact[(int64_t)row * g.ldd + col] = v;
                    if (g.act == 1) v = silu(v);
                    if (g.resid) v = __fadd_rn(v, g.resid[(int64_t)row * g.ldr + col]);
                    if (g.Df) g.Df[(int64_t)row * g.ldd + col] = v;
                    if (g.Db) g.Db[(int64_t)row * g.ldd + col] = __float2bfloat16(v);
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr),
                     "r"((uint32_t)(N < 32 ? 32 : N)));
}

template <int N>
static int launch_gemm(const GemmArgs& g, cudaStream_t s) {
    // one staging buffer per K slice a CTA handles, at most two (fewer bytes: more CTAs per SM)
    const int kchunks = g.K / TK, per = (kchunks + g.k_splits - 1) / g.k_splits;
    const size_t smem = (size_t)(per >= 2 ? 2 : 1) * ((size_t)TM * TK * 2 + (size_t)N * TK * 2);
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(k_gemm<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(2 * ((size_t)TM * TK * 2 + (size_t)N * TK * 2)));
        attr = true;
    }
    dim3 grid((unsigned)((g.M + TM - 1) / TM), (unsigned)g.k_splits);
    FVM_LAUNCH(KID_CORRECTOR, s, k_gemm<N><<<grid, kGemmThreads, smem, s>>>(g));
    return launch_status();
}

}  // namespace corr
}  // namespace fvm

using namespace fvm;

extern "C" int fvm_gemm_bf16(const void* A, int64_t lda, const void* B, int64_t ldb, int32_t M, int32_t N, int32_t K,
                             int32_t k_splits, const float* bias, const float* resid, int64_t ldr, float* Df,
                             void* Db, int64_t ldd, float* preact, int32_t act, int32_t* err, void* stream) {
    if (!A || !B || M <= 0 || K <= 0 || K % corr::TK != 0 || k_splits < 1 || (!Df && !Db) || !err) return FVM_E_ARG;
    if (N != 32 && N != 64 && N != 128 && N != 256) return FVM_E_UNSUPPORTED;
    if ((uintptr_t)A % 16 || (uintptr_t)B % 16 || lda % 8 || ldb % 8) return FVM_E_ARG;
    if (k_splits > 1 && (!Df || bias || resid || preact || Db || act)) return FVM_E_ARG;
    // 256-bit epilogue when every row chunk of 32 columns starts on a 32-byte boundary.
    auto a32 = [](const void* p) { return ((uintptr_t)p & 31u) == 0; };
    const int vec = a32(bias) && a32(resid) && a32(Df) && a32(Db) && a32(preact) && (!resid || ldr % 8 == 0) &&
                    ((!Df && !preact) || ldd % 8 == 0) && (!Db || ldd % 16 == 0);
    corr::GemmArgs g{static_cast<const __nv_bfloat16*>(A), lda, static_cast<const __nv_bfloat16*>(B), ldb, M, N, K,
                     k_splits, bias, resid, ldr, Df, static_cast<__nv_bfloat16*>(Db), ldd, preact, act, err, vec};
    cudaStream_t s = (cudaStream_t)stream;
    switch (N) {
        case 32: return corr::launch_gemm<32>(g, s);
        case 64: return corr::launch_gemm<64>(g, s);
        case 128: return corr::launch_gemm<128>(g, s);
        default: return corr::launch_gemm<256>(g, s);
    }
}

// ------------------------------------------------------------------------------------------
// Message passing, activations, loss and optimiser kernels of the corrector.
// Activations h: bf16 [N][W] (W = 64); neighbour table nbr: int32 [N][KN] (-1 = none).
// ------------------------------------------------------------------------------------------
namespace fvm {
namespace corr {

__global__ void k_mse(const float* __restrict__ pred, const float* __restrict__ tgt, int64_t n_elem, float inv_n,
                      double* __restrict__ loss, float* __restrict__ dpred) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    __shared__ double red[32];
    double v[1] = {0.0};
    if (t < n_elem) {
        const float d = pred[t] - tgt[t];
        dpred[t] = 2.f * d * inv_n;
        v[0] = (double)d * d * inv_n;
    }
    block_sum<1>(v, red);
    if (threadIdx.x == 0) atomicAdd(loss, v[0]);
}

// Adam (decoupled bias correction) on fp32 master weights; refreshes the bf16 copy [rows][cols]
// and, if requested, its transpose [cols][rows] used by the backward GEMMs.  Zeroes the gradient.
// blockIdx.y is the tensor: the network's dozen tensors of 4 to 8192 entries are bound by their launches
// (12 x 2.4 us one by one), so all of them go in one.
constexpr int kAdamMany = 32;
struct AdamTensor {
    float *p, *g, *m, *v;
    __nv_bfloat16 *pb, *pbT;
    int64_t n;
    int rows, cols;
};
struct AdamArgs {
    AdamTensor t[kAdamMany];
};
__global__ void k_adam(const __grid_constant__ AdamArgs args, float lr, float b1, float b2, float eps, float c1, float c2) {
    const AdamTensor& a = args.t[blockIdx.y];
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= a.n) return;
    const float gr = a.g[t];
    const float mt = b1 * a.m[t] + (1.f - b1) * gr;
    const float vt = b2 * a.v[t] + (1.f - b2) * gr * gr;
    a.m[t] = mt;
    a.v[t] = vt;
    const float w = a.p[t] - lr * (mt / c1) / (sqrtf(vt / c2) + eps);
    a.p[t] = w;
    a.g[t] = 0.f;
    if (a.pb) a.pb[t] = __float2bfloat16(w);
    if (a.pbT) {
        const int r = (int)(t / a.cols), c = (int)(t % a.cols);
        a.pbT[(int64_t)c * a.rows + r] = __float2bfloat16(w);
    }
}

// Network input: X[i] = [(U_i - mean) * inv_std (C values), geometry (G values), zeros] bf16 [N][64].
__global__ void k_features(const float* __restrict__ state, int N, int C, const float* __restrict__ mean,
                           const float* __restrict__ inv_std, const float* __restrict__ geo, int G,
                           __nv_bfloat16* __restrict__ X, int XW) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= (int64_t)N * XW) return;
    const int i = (int)(t / XW), c = (int)(t % XW);
    float v = 0.f;
    if (c < C) v = (state[(int64_t)i * C + c] - mean[c]) * inv_std[c];
    else if (c < C + G) v = geo[(int64_t)i * G + (c - C)];
    X[t] = __float2bfloat16(v);
}

// U_new = U + scale * out (out: normalised increment, fp32 [N][C]).
__global__ void k_apply_increment(const float* __restrict__ state, const float* __restrict__ out,
                                  const float* __restrict__ scale, int N, int C, float* __restrict__ new_state) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= (int64_t)N * C) return;
    new_state[t] = state[t] + scale[t % C] * out[t];
}

// Corrector inputs, one thread per cell: base = k dt(case) * r0 and the bf16 feature row
// [(U - mean) * inv_std, (base - mean) * inv_std, geometry, zeros] (XW entries).
template <int C>
__global__ void k_corrector_inputs(const float* __restrict__ state, const float* __restrict__ r0,
                                   const float* __restrict__ kdt_case, const int32_t* __restrict__ cell_case, int N,
                                   const float* __restrict__ mean, const float* __restrict__ inv_std,
                                   const float* __restrict__ geo, int G, float* __restrict__ base,
                                   __nv_bfloat16* __restrict__ X, int XW) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const float h = kdt_case[cell_case ? __ldg(cell_case + i) : 0];
    float u[C], b[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        u[c] = __ldg(state + (int64_t)i * C + c);
        b[c] = h * __ldg(r0 + (int64_t)i * C + c);
        base[(int64_t)i * C + c] = b[c];
    }
    __nv_bfloat16* row = X + (int64_t)i * XW;
    // entries 0..15 hold the 2C <= 10 state / baseline features (indices known at compile time)
#pragma unroll
    for (int q = 0; q < 16; q += 8) {
        __align__(16) __nv_bfloat16 v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int c = q + e;
            float x = 0.f;
            if (c < C) x = (u[c < C ? c : 0] - __ldg(mean + c)) * __ldg(inv_std + c);
            else if (c < 2 * C) x = (b[(c >= C && c < 2 * C) ? c - C : 0] - __ldg(mean + c)) * __ldg(inv_std + c);
            else if (c < 2 * C + G) x = __ldg(geo + (int64_t)i * G + (c - 2 * C));
            v[e] = __float2bfloat16(x);
        }
        *reinterpret_cast<uint4*>(row + q) = *reinterpret_cast<const uint4*>(v);
    }
    for (int q = 16; q < XW; q += 8) {
        __align__(16) __nv_bfloat16 v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int c = q + e;
            v[e] = __float2bfloat16(c < 2 * C + G ? __ldg(geo + (int64_t)i * G + (c - 2 * C)) : 0.f);
        }
        *reinterpret_cast<uint4*>(row + q) = *reinterpret_cast<const uint4*>(v);
    }
}

// prop = state + base + scale * out - shift(case)  (shift: per-case [C] offsets, or null).
__global__ void k_corrector_combine(const float* __restrict__ state, const float* __restrict__ base,
                                    const float* __restrict__ out, const float* __restrict__ scale,
                                    const float* __restrict__ shift, const int32_t* __restrict__ cell_case, int N,
                                    int C, float* __restrict__ prop) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= (int64_t)N * C) return;
    const int i = (int)(t / C), c = (int)(t % C);
    float v = state[t] + base[t] + __ldg(scale + c) * out[t];
    if (shift) v -= __ldg(shift + (int64_t)(cell_case ? __ldg(cell_case + i) : 0) * C + c);
    prop[t] = v;
}

// Rows of C floats: whole where `whole` says that they start on 16-byte boundaries, else float by float
// (five floats always).
template <int C>
__device__ __forceinline__ void load_row_any(const float* p, bool whole, float (&v)[C]) {
    if (whole) load_row<C>(p, v);
    else
#pragma unroll
        for (int c = 0; c < C; ++c) v[c] = __ldg(p + c);
}
template <int C>
__device__ __forceinline__ void store_row_any(float* p, bool whole, const float (&v)[C]) {
    if (whole) store_row<C>(p, v);
    else
#pragma unroll
        for (int c = 0; c < C; ++c) p[c] = v[c];
}

// The same with the shift formed from the cases' sums of vol * out: the components from `first` on lose
// the volume-weighted mean of scale * out, (float)(sums / case_vol * scale).  One thread per cell.
template <int C>
__global__ void __launch_bounds__(256) k_corrector_propose(const float* __restrict__ state, const float* __restrict__ base,
                                                           const float* __restrict__ out, const float* __restrict__ scale,
                                                           const double* __restrict__ sums,
                                                           const double* __restrict__ case_vol, int first,
                                                           const int32_t* __restrict__ cell_case, int N, bool whole,
                                                           float* __restrict__ prop) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int cs = cell_case ? __ldg(cell_case + i) : 0;
    const double vol = __ldg(case_vol + cs);
    float u[C], b[C], o[C];
    load_row_any<C>(state + (int64_t)i * C, whole, u);
    load_row_any<C>(base + (int64_t)i * C, whole, b);
    load_row_any<C>(out + (int64_t)i * C, whole, o);
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const float sc = __ldg(scale + c);
        float v = u[c] + b[c] + sc * o[c];
        v -= c >= first ? (float)(__ldg(sums + (int64_t)cs * C + c) / vol * (double)sc) : 0.f;
        u[c] = v;
    }
    store_row_any<C>(prop + (int64_t)i * C, whole, u);
}

static inline unsigned nblk(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

}  // namespace corr
}  // namespace fvm

extern "C" int fvm_mse(const float* pred, const float* tgt, int64_t n_elem, double* loss, float* dpred,
                       void* stream) {
    if (!pred || !tgt || !loss || !dpred || n_elem <= 0) return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    FVM_LAUNCH(KID_CORRECTOR, s, corr::k_mse<<<corr::nblk(n_elem, 256), 256, 0, s>>>(
                                     pred, tgt, n_elem, 1.f / (float)n_elem, loss, dpred));
    return launch_status();
}

extern "C" int fvm_adam_many(int32_t count, float* const* p, float* const* g, float* const* m, float* const* v,
                             const int64_t* n, float lr, float beta1, float beta2, float eps, int32_t step,
                             void* const* pb, void* const* pbT, const int32_t* rows, const int32_t* cols, void* stream) {
    if (count < 1 || count > corr::kAdamMany || !p || !g || !m || !v || !n || !pb || !pbT || !rows || !cols || step < 1)
        return FVM_E_ARG;
    corr::AdamArgs a{};
    int64_t most = 0;
    for (int q = 0; q < count; ++q) {
        if (!p[q] || !g[q] || !m[q] || !v[q] || n[q] <= 0 || (pbT[q] && (int64_t)rows[q] * cols[q] != n[q]))
            return FVM_E_ARG;
        a.t[q] = corr::AdamTensor{p[q], g[q], m[q], v[q], static_cast<__nv_bfloat16*>(pb[q]),
                                  static_cast<__nv_bfloat16*>(pbT[q]), n[q], rows[q], cols[q]};
        most = std::max(most, n[q]);
    }
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    cudaStream_t s = (cudaStream_t)stream;
    FVM_LAUNCH(KID_CORRECTOR, s, corr::k_adam<<<dim3(corr::nblk(most, 256), (unsigned)count), 256, 0, s>>>(
                                     a, lr, beta1, beta2, eps, c1, c2));
    return launch_status();
}

extern "C" int fvm_adam(float* p, float* g, float* m, float* v, int64_t n, float lr, float beta1, float beta2, float eps,
                        int32_t step, void* pb, void* pbT, int32_t rows, int32_t cols, void* stream) {
    return fvm_adam_many(1, &p, &g, &m, &v, &n, lr, beta1, beta2, eps, step, &pb, &pbT, &rows, &cols, stream);
}

extern "C" int fvm_corrector_features(const float* state, int32_t N, int32_t C, const float* mean,
                                      const float* inv_std, const float* geo, int32_t G, void* X, int32_t XW,
                                      void* stream) {
    if (!state || !mean || !inv_std || !X || N <= 0 || C + G > XW || (G > 0 && !geo)) return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    FVM_LAUNCH(KID_CORRECTOR, s, corr::k_features<<<corr::nblk((int64_t)N * XW, 256), 256, 0, s>>>(
                                     state, N, C, mean, inv_std, geo, G, static_cast<__nv_bfloat16*>(X), XW));
    return launch_status();
}

extern "C" int fvm_apply_increment(const float* state, const float* out, const float* scale, int32_t N, int32_t C,
                                   float* new_state, void* stream) {
    if (!state || !out || !scale || !new_state || N <= 0 || C <= 0) return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    FVM_LAUNCH(KID_CORRECTOR, s, corr::k_apply_increment<<<corr::nblk((int64_t)N * C, 256), 256, 0, s>>>(
                                     state, out, scale, N, C, new_state));
    return launch_status();
}

extern "C" int fvm_corrector_inputs(const float* state, const float* r0, const float* kdt_case,
                                    const int32_t* cell_case, int32_t N, int32_t C, const float* mean,
                                    const float* inv_std, const float* geo, int32_t G, float* base, void* X,
                                    int32_t XW, void* stream) {
    if (!state || !r0 || !kdt_case || !mean || !inv_std || (G > 0 && !geo) || !base || !X || N <= 0 || G < 0 ||
        XW % 8 != 0 || XW < 16 || 2 * C + G > XW || ((uintptr_t)X & 15u) != 0)
        return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    if (C == 4)
        FVM_LAUNCH(KID_CORRECTOR, s, corr::k_corrector_inputs<4><<<corr::nblk(N, 128), 128, 0, s>>>(
                                         state, r0, kdt_case, cell_case, N, mean, inv_std, geo, G, base,
                                         static_cast<__nv_bfloat16*>(X), XW));
    else if (C == 5)
        FVM_LAUNCH(KID_CORRECTOR, s, corr::k_corrector_inputs<5><<<corr::nblk(N, 128), 128, 0, s>>>(
                                         state, r0, kdt_case, cell_case, N, mean, inv_std, geo, G, base,
                                         static_cast<__nv_bfloat16*>(X), XW));
    else
        return FVM_E_UNSUPPORTED;
    return launch_status();
}

extern "C" int fvm_corrector_combine(const float* state, const float* base, const float* out, const float* scale,
                                     const float* shift, const int32_t* cell_case, int32_t N, int32_t C, float* prop,
                                     void* stream) {
    if (!state || !base || !out || !scale || !prop || N <= 0 || C <= 0) return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    FVM_LAUNCH(KID_CORRECTOR, s, corr::k_corrector_combine<<<corr::nblk((int64_t)N * C, 256), 256, 0, s>>>(
                                     state, base, out, scale, shift, cell_case, N, C, prop));
    return launch_status();
}

extern "C" int fvm_corrector_propose(const float* state, const float* base, const float* out, const float* scale,
                                     const double* sums, const double* case_vol, int32_t first,
                                     const int32_t* cell_case, int32_t N, int32_t C, float* prop, void* stream) {
    if (!state || !base || !out || !scale || !sums || !case_vol || !prop || N <= 0 || first < 0) return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    const bool whole = (((uintptr_t)state | (uintptr_t)base | (uintptr_t)out | (uintptr_t)prop) & 15u) == 0;
    if (C == 4)
        FVM_LAUNCH(KID_CORRECTOR, s, corr::k_corrector_propose<4><<<corr::nblk(N, 256), 256, 0, s>>>(
                                         state, base, out, scale, sums, case_vol, first, cell_case, N, whole, prop));
    else if (C == 5)
        FVM_LAUNCH(KID_CORRECTOR, s, corr::k_corrector_propose<5><<<corr::nblk(N, 256), 256, 0, s>>>(
                                         state, base, out, scale, sums, case_vol, first, cell_case, N, whole, prop));
    else
        return FVM_E_UNSUPPORTED;
    return launch_status();
}

// ------------------------------------------------------------------------------------------
// Message-passing layer on an fp32 residual stream (fvm_mp_layer, fvm_mp_layer_train) and the
// network's input layer (fvm_in_layer).
//
//   h'_i = h_i + SiLU([bf16(h_i), bf16(mean_{j in nbr(i)} h_j)] . W^T + b)       (W: bf16 [64][128])
//   and, for the last layer, out_i = W_out h'_i + b_out (h' itself only if asked for);
//   input layer: h_i = SiLU(X_i . W^T + b)                                       (X, W: bf16, K = 64)
//
// Per row a layer reads h (256 B), gathers up to KN neighbour rows and writes h' (256 B); the
// neighbours of the Morton-ordered cells are mostly in the same tile, so the gathers hit L1 (72 %)
// and the floor is the 512 bytes of DRAM traffic.  What bounds it is latency: a tile is a chain of
// neighbour list -> gathers -> MMA -> epilogue.  One CTA of 128 rows therefore runs that chain without
// any role split, small enough (256 threads, 56 KB of shared memory, 64 TMEM columns) that three or four
// CTAs share an SM and fill each other's waits; one CTA per SM with gather and epilogue warps side by side
// left 12 warps per SM and took 111 us per layer at 278 k rows of 64 (now 50 us).  The
// epilogue goes through shared memory (the operand's own buffer, free once the MMAs are done), so
// the residual, the pre-activation and h' move as whole 128-byte lines instead of one line per lane.
// The mbarrier wait is bounded; a wait that gives up sets *err and ends the CTA.
// ------------------------------------------------------------------------------------------
namespace fvm {
namespace corr {

constexpr int kLayerThreads = 256;
// CTAs per SM: four of the input layer; three of the others, whose 80 registers hold a row's gathers
// without spills (50 us per layer at 278 k rows of 64; four with 64 registers spill, 55 us).
constexpr int layer_ctas(bool input) { return input ? 4 : 3; }
constexpr int kLayerW = 64;                              // channels
// One 8-channel unit of a tile's rows, 32 bytes apart from the next modulo 128: the 16-byte stores of
// four units x two rows (eight lanes) then hit every bank once.
constexpr int kUnitBytes = TM * 16 + 32;
constexpr int kLayerABytes = 16 * kUnitBytes;            // operand tile, 128 channels (input layer: half)
constexpr int kLayerWUnit = kLayerW * 16;                // one 8-channel unit of the weights' rows
constexpr int kLayerWBytes = 16 * kLayerWUnit;           // W: 64 x 128 bf16
constexpr int kLayerSmem = kLayerWBytes + kLayerABytes;

struct LayerArgs {
    const float* h;              // [M][64] fp32 residual stream (input)
    const int32_t* nbr;          // [M][KN]
    const __nv_bfloat16* X;      // input layer: [M][64] features (h and nbr unused), or null:
    const float *state, *r0, *dt, *mean, *inv_std, *geo;   // the features of fvm_corrector_inputs, built
    const int32_t* cell_case;                              // here (C, G columns; base [M][C] is stored)
    float* base;
    __nv_bfloat16* Xout;         // the feature rows formed here, [M][64], or null
    int C, G;
    bool whole;                  // rows of state, r0 and base start on 16-byte boundaries
    float k;
    int M, KN;
    const __nv_bfloat16* Wt;     // [64][128] (input layer: [64][64])
    const float* bias;           // [64]
    float* h_out;                // [M][64] or null (decoder only)
    float* Z;                    // [M][64] pre-activations or null (training)
    __nv_bfloat16* A;            // [M][128] operand rows or null (training)
    const float* Wo;             // [O][64] decoder weights or null
    const float* bo;             // [O]
    int O;
    float* out;                  // [M][O] decoder outputs or null
    int* err;
};

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(d),
        "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

// 32 accumulator columns [c0, c0 + 32) of this warp's TMEM lanes.
__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 16 TMEM lanes x 32 columns as 16x256b blocks: register 4 g + 2 j + e of lane t holds lane 8 j + t / 4,
// column 8 g + 2 (t % 4) + e.  With the operand's columns stored in the order of frag_col, a lane has
// eight neighbouring logical columns of a row and the row's 32 columns lie on four consecutive lanes.
__device__ __forceinline__ void tmem_ld_frag(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
}
__device__ __forceinline__ int frag_col(int m) {   // TMEM column of logical column m
    return (m & ~31) | ((m >> 1) & 3) << 3 | ((m >> 3) & 3) << 1 | (m & 1);
}

// Operand layout of a tile: 16-byte unit u (8 channels) of row r at u * kUnitBytes + 16 r.  Eight
// consecutive rows of a unit are one core matrix, so the tile reads as a K-major operand with the
// channels as K (core matrices of a K step LBO = kUnitBytes apart, 8-row groups SBO = 128 apart).
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
    __align__(16) __nv_bfloat16 a[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) a[e] = __float2bfloat16(v[e]);
    return *reinterpret_cast<const uint4*>(a);
}
// Offset of 16-byte chunk c (0..15) of row r in the fp32 epilogue tile (256 bytes per row): the
// chunk index is xored with the row, so eight rows at one chunk and two rows at four even (or odd)
// chunks both hit every bank once.
__device__ __forceinline__ int epi_off(int r, int c) { return r * 256 + ((c ^ (r & 7)) << 4); }

// A row of zeros: what a missing neighbour, or a row past M, reads (adding +0 leaves a sum that starts
// at +0 unchanged), so the gather needs no selects on the data.
__device__ __align__(256) float g_zero_row[kLayerW];

// A row's features as k_corrector_inputs forms them -- normalised state and baseline k dt r0 (stored to
// base), geometry, zeros -- into the operand tile: the row's thread of the block's first half takes the
// first 16, that of the second half the others, so a thread's loads are all independent.
template <int C>
__device__ __forceinline__ void stage_features(const LayerArgs& g, uint8_t* sA, int64_t row, int r, bool second) {
    const bool valid = row < g.M;
    if (!second) {
        float u[C], b[C], x[16];
        float h = 0.f;
        if (valid) {
            load_row_any<C>(g.state + row * C, g.whole, u);
            load_row_any<C>(g.r0 + row * C, g.whole, b);
            h = g.k * __ldg(g.dt + (g.cell_case ? __ldg(g.cell_case + row) : 0));
        }
#pragma unroll
        for (int c = 2 * C; c < 16; ++c) x[c] = valid && c < 2 * C + g.G ? __ldg(g.geo + row * g.G + c - 2 * C) : 0.f;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            b[c] *= h;
            x[c] = valid ? (u[c] - __ldg(g.mean + c)) * __ldg(g.inv_std + c) : 0.f;
            x[C + c] = valid ? (b[c] - __ldg(g.mean + C + c)) * __ldg(g.inv_std + C + c) : 0.f;
        }
        if (valid) store_row_any<C>(g.base + row * C, g.whole, b);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = x[8 * q + e];
            *reinterpret_cast<uint4*>(sA + q * kUnitBytes + r * 16) = pack8(v);
        }
    } else {
        for (int q = 2; q < 8; ++q) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int c = 8 * q + e;
                v[e] = valid && c < 2 * C + g.G ? __ldg(g.geo + row * g.G + c - 2 * C) : 0.f;
            }
            *reinterpret_cast<uint4*>(sA + q * kUnitBytes + r * 16) = pack8(v);
        }
    }
}

template <bool INPUT>
__global__ void __launch_bounds__(kLayerThreads, layer_ctas(INPUT)) k_mp_layer(LayerArgs g) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sW = smem;                                   // B operand
    uint8_t* sA = smem + kLayerWBytes;                    // A operand, then the epilogue tile
    constexpr int UNITS = INPUT ? 8 : 16;
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t s_taddr;
    __shared__ __align__(16) int s_nb[INPUT ? 4 : TM * 8];
    __shared__ float s_inv[INPUT ? 1 : TM];
    __shared__ __align__(16) float s_bias[kLayerW];
    __shared__ __align__(16) float s_wo[INPUT ? 4 : 8 * kLayerW];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ntiles = (g.M + TM - 1) / TM;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_taddr)),
                     "r"(64u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    dependency_wait();
    for (int t = tid; t < kLayerW * UNITS; t += kLayerThreads) {
        const int r = t / UNITS, u = t % UNITS;
        *reinterpret_cast<uint4*>(sW + u * kLayerWUnit + r * 16) =
            *reinterpret_cast<const uint4*>(g.Wt + (int64_t)r * 8 * UNITS + 8 * u);
    }
    if (tid < kLayerW) s_bias[tid] = g.bias[tid];
    if (!INPUT && g.out)
        for (int t = tid; t < g.O * kLayerW; t += kLayerThreads) s_wo[t] = g.Wo[t];
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t taddr = s_taddr;
    const uint32_t idesc = make_idesc(kLayerW);

    // A thread's share of a tile: the 8-channel unit u of rows r0 + 32 q, q = 0..3.  A warp covers
    // 8 rows x 4 units per q with each row's units on four consecutive lanes: the L1 serves a 256-bit
    // access four lanes at a time, in one cycle when they share a 128-byte line (9 cycles per
    // warp request) and in up to four when they do not (rows on consecutive lanes: 48 cycles, 88 %
    // of the L1 data path's peak and 86 us per layer at 278 k rows).
    const int u = (tid & 3) + 4 * (warp & 1), r0 = (lane >> 2) + 8 * (warp >> 1);
    // Neighbour lists (thread t: row t) are fetched one tile ahead.
    int nxt[8];
    auto fetch_nbr = [&](int tile) {
        const int64_t row = (int64_t)tile * TM + tid;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            nxt[q] = (tid < TM && row < g.M && q < g.KN) ? __ldg(g.nbr + row * g.KN + q) : -1;
    };
    if (!INPUT && (int)blockIdx.x < ntiles) fetch_nbr(blockIdx.x);
    bool ok = true;
    int k = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++k) {
        const int m0 = tile * TM;
        if constexpr (!INPUT) {
            if (tid < TM) {
                int cnt = 0;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    s_nb[tid * 8 + q] = nxt[q];
                    cnt += nxt[q] >= 0;
                }
                s_inv[tid] = cnt > 0 ? 1.f / (float)cnt : 0.f;
            }
            if (tile + (int)gridDim.x < ntiles) fetch_nbr(tile + gridDim.x);
            __syncthreads();
        }
        // A operand.  The neighbour mean is the fp32 sum over the valid neighbours in table order
        // (starting at +0) times 1 / count; with at most four neighbours all loads of a row's unit
        // are issued before any is used.
        if (INPUT && !g.X) {
            const int r = tid & (TM - 1);
            if (g.C == 4) stage_features<4>(g, sA, (int64_t)m0 + r, r, tid >= TM);
            else stage_features<5>(g, sA, (int64_t)m0 + r, r, tid >= TM);
        } else
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
            const int r = r0 + 32 * q;
            const int64_t row = (int64_t)m0 + r;
            const bool valid = row < g.M;
            if constexpr (INPUT) {
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (valid) v = *reinterpret_cast<const uint4*>(g.X + row * kLayerW + 8 * u);
                *reinterpret_cast<uint4*>(sA + u * kUnitBytes + r * 16) = v;
            } else {
                auto src = [&](int64_t j, bool on) { return (on ? g.h + j * kLayerW : (const float*)g_zero_row) + 8 * u; };
                float own[8], acc[8];
                ld8(src(row, valid), own);
                if (g.KN <= 4) {
                    float nb[4][8];
                    const int4 jj = *reinterpret_cast<const int4*>(s_nb + r * 8);
                    ld8(src(jj.x, jj.x >= 0), nb[0]);
                    ld8(src(jj.y, jj.y >= 0), nb[1]);
                    ld8(src(jj.z, jj.z >= 0), nb[2]);
                    if (g.KN == 4) ld8(src(jj.w, jj.w >= 0), nb[3]);
#pragma unroll
                    for (int c = 0; c < 8; ++c) acc[c] = ((0.f + nb[0][c]) + nb[1][c]) + nb[2][c];
                    if (g.KN == 4)
#pragma unroll
                        for (int c = 0; c < 8; ++c) acc[c] += nb[3][c];
                } else {
#pragma unroll
                    for (int c = 0; c < 8; ++c) acc[c] = 0.f;
                    for (int e = 0; e < g.KN; ++e) {
                        const int j = s_nb[r * 8 + e];
                        if (j < 0) continue;
                        float v[8];
                        ld8(g.h + (int64_t)j * kLayerW + 8 * u, v);
#pragma unroll
                        for (int c = 0; c < 8; ++c) acc[c] += v[c];
                    }
                }
                const float inv = s_inv[r];
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[c] *= inv;
                const uint4 a = pack8(own), b = pack8(acc);
                *reinterpret_cast<uint4*>(sA + u * kUnitBytes + r * 16) = a;
                *reinterpret_cast<uint4*>(sA + (8 + u) * kUnitBytes + r * 16) = b;
                if (g.A && valid) {
                    *reinterpret_cast<uint4*>(g.A + row * 2 * kLayerW + 8 * u) = a;
                    *reinterpret_cast<uint4*>(g.A + row * 2 * kLayerW + kLayerW + 8 * u) = b;
                }
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
            for (int q = 0; q < UNITS / 2; ++q)
                tc_mma(taddr, make_desc(smem_u32(sA) + 2 * q * kUnitBytes, kUnitBytes, 128),
                       make_desc(smem_u32(sW) + 2 * q * kLayerWUnit, kLayerWUnit, 128), idesc, q > 0);
            tc_commit(&bar);
        }
        if (INPUT && g.Xout)   // features formed here, out of the operand tile while the products run
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = r0 + 32 * q;
                if (m0 + r < g.M)
                    *reinterpret_cast<uint4*>(g.Xout + (int64_t)(m0 + r) * kLayerW + 8 * u) =
                        *reinterpret_cast<const uint4*>(sA + u * kUnitBytes + r * 16);
            }
        if (!__syncthreads_and(mbar_wait(&bar, (uint32_t)(k & 1)))) {
            ok = false;
            break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        {   // accumulator + bias -> epilogue tile; warp w reads TMEM lanes 32 (w % 4), columns 32 (w / 4)
            const int r = 32 * (warp & 3) + lane, half = warp >> 2;
            uint32_t z[32];
            tmem_ld32(taddr + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(32 * half), z);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float4 bs = *reinterpret_cast<const float4*>(s_bias + 32 * half + 4 * c);
                float4 v;
                v.x = __uint_as_float(z[4 * c]) + bs.x;
                v.y = __uint_as_float(z[4 * c + 1]) + bs.y;
                v.z = __uint_as_float(z[4 * c + 2]) + bs.z;
                v.w = __uint_as_float(z[4 * c + 3]) + bs.w;
                *reinterpret_cast<float4*>(sA + epi_off(r, 8 * half + c)) = v;
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
        // activation and residual, row units as in the gather
#pragma unroll 2
        for (int q = 0; q < 4; ++q) {
            const int r = r0 + 32 * q;
            const int64_t row = (int64_t)m0 + r;
            if (row < g.M) {
                float x[8], v[8];
                if constexpr (!INPUT) ld8(g.h + row * kLayerW + 8 * u, x);
                float4* lo = reinterpret_cast<float4*>(sA + epi_off(r, 2 * u));
                float4* hi = reinterpret_cast<float4*>(sA + epi_off(r, 2 * u + 1));
                const float4 a = *lo, b = *hi;
                v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
                if (g.Z) st8(g.Z + row * kLayerW + 8 * u, v);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    v[c] = silu(v[c]);
                    if constexpr (!INPUT) v[c] = __fadd_rn(v[c], x[c]);
                }
                if (g.h_out) st8(g.h_out + row * kLayerW + 8 * u, v);
                if (!INPUT && g.out) {
                    *lo = make_float4(v[0], v[1], v[2], v[3]);
                    *hi = make_float4(v[4], v[5], v[6], v[7]);
                }
            }
        }
        if (!INPUT && g.out) {   // decoder: thread t takes row t % 128, outputs t / 128, t / 128 + 2, ...
            __syncthreads();
            const int r = tid & (TM - 1);
            if (m0 + r < g.M) {
                float dec[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int o = 2 * e + (tid >> 7);
                    dec[e] = o < g.O ? __ldg(g.bo + o) : 0.f;
                }
#pragma unroll 4
                for (int c = 0; c < 16; ++c) {
                    const float4 v = *reinterpret_cast<const float4*>(sA + epi_off(r, c));
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int o = 2 * e + (tid >> 7);
                        if (o < g.O) {
                            const float4 w = *reinterpret_cast<const float4*>(s_wo + o * kLayerW + 4 * c);
                            dec[e] = fmaf(v.x, w.x, dec[e]);
                            dec[e] = fmaf(v.y, w.y, dec[e]);
                            dec[e] = fmaf(v.z, w.z, dec[e]);
                            dec[e] = fmaf(v.w, w.w, dec[e]);
                        }
                    }
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int o = 2 * e + (tid >> 7);
                    if (o < g.O) g.out[(int64_t)(m0 + r) * g.O + o] = dec[e];
                }
            }
        }
        __syncthreads();                                  // the tile's buffers may be overwritten
    }
    if (!ok && tid == 0) {
        if (g.err) atomicExch(g.err, 1);
        mbar_wait(&bar, (uint32_t)(k & 1));              // a second bounded chance before TMEM is released
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(64u));
}

// Grid: one wave of resident CTAs, or one per tile.
template <bool INPUT>
static int launch_layer(const LayerArgs& g, cudaStream_t s) {
    static int sms[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) {
        launch_status();
        return FVM_E_CUDA;
    }
    if (!sms[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaFuncSetAttribute(k_mp_layer<INPUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kLayerSmem) !=
                cudaSuccess) {
            launch_status();
            return FVM_E_CUDA;
        }
        sms[dev] = n;
    }
    const int ntiles = (g.M + TM - 1) / TM;
    FVM_LAUNCH(KID_CORRECTOR, s, launch(k_mp_layer<INPUT>, dim3((unsigned)std::min(ntiles, layer_ctas(INPUT) * sms[dev])),
                                        dim3(kLayerThreads), kLayerSmem, s, g));
    return launch_status();
}

// Training-path gather with the fused layer's arithmetic: out[i] = [bf16(h_i), bf16(mean_j h_j)]
// from the fp32 residual stream (mean = fp32 sum over the valid neighbours in table order times
// 1 / count); bf16 [N][128].  One thread per (cell, 8-channel unit).
__global__ void k_mp_gather_f32(const float* __restrict__ h, const int32_t* __restrict__ nbr, int N, int KN,
                                __nv_bfloat16* __restrict__ out) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= (int64_t)N * 8) return;
    const int i = (int)(t >> 3), u = (int)(t & 7);
    float own[8], acc[8];
    ld8(h + (int64_t)i * kLayerW + 8 * u, own);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    int cnt = 0;
    for (int k = 0; k < KN; ++k) {
        const int j = __ldg(nbr + (int64_t)i * KN + k);
        cnt += j >= 0;
    }
    const float inv = cnt > 0 ? 1.f / (float)cnt : 0.f;
    for (int k = 0; k < KN && k < 8; ++k) {
        const int j = __ldg(nbr + (int64_t)i * KN + k);
        if (j < 0) continue;
        float v[8];
        ld8(h + (int64_t)j * kLayerW + 8 * u, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += v[e];
    }
    __align__(16) __nv_bfloat16 a[8], b[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        a[e] = __float2bfloat16(own[e]);
        b[e] = __float2bfloat16(acc[e] * inv);
    }
    *reinterpret_cast<uint4*>(out + (int64_t)i * 2 * kLayerW + 8 * u) = *reinterpret_cast<const uint4*>(a);
    *reinterpret_cast<uint4*>(out + (int64_t)i * 2 * kLayerW + kLayerW + 8 * u) = *reinterpret_cast<const uint4*>(b);
}

// Decoder on the fp32 stream with the fused layer's order: out[i][o] = b[o] + sum_c h[i][c] Wo[o][c]
// (fp32 fma over c ascending).
__global__ void k_decoder_f32(const float* __restrict__ h, const float* __restrict__ Wo, const float* __restrict__ bo,
                              int N, int O, float* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    float acc[8];
#pragma unroll
    for (int o = 0; o < 8; ++o) acc[o] = o < O ? bo[o] : 0.f;
    for (int c0 = 0; c0 < kLayerW; c0 += 8) {
        float x[8];
        ld8(h + (int64_t)i * kLayerW + c0, x);
#pragma unroll
        for (int e = 0; e < 8; ++e)
#pragma unroll
            for (int o = 0; o < 8; ++o)
                if (o < O) acc[o] = fmaf(x[e], Wo[o * kLayerW + c0 + e], acc[o]);
    }
    for (int o = 0; o < O; ++o) out[(int64_t)i * O + o] = acc[o];
}

}  // namespace corr
}  // namespace fvm

extern "C" int fvm_mp_layer_train(const float* h, const int32_t* nbr, int32_t M, int32_t KN, const void* Wt,
                                  const float* bias, float* h_out, float* Z, void* A, const float* Wo,
                                  const float* bo, int32_t O, float* out, int32_t* err, void* stream) {
    if (!h || !nbr || !Wt || !bias || M <= 0 || KN <= 0 || KN > 8 || !err) return FVM_E_ARG;
    if (!h_out && !out) return FVM_E_ARG;
    if (out && (!Wo || !bo || O < 1 || O > 8)) return FVM_E_ARG;
    auto a32 = [](const void* p) { return ((uintptr_t)p & 31u) == 0; };
    if (!a32(h) || !a32(h_out) || !a32(Z) || (uintptr_t)Wt % 16 || (uintptr_t)A % 16) return FVM_E_ARG;
    if (h_out == h) return FVM_E_ARG;                    // the neighbours of later tiles read h
    corr::LayerArgs g{};
    g.h = h;
    g.nbr = nbr;
    g.M = M;
    g.KN = KN;
    g.Wt = static_cast<const __nv_bfloat16*>(Wt);
    g.bias = bias;
    g.h_out = h_out;
    g.Z = Z;
    g.A = static_cast<__nv_bfloat16*>(A);
    g.Wo = Wo;
    g.bo = bo;
    g.O = O;
    g.out = out;
    g.err = err;
    return corr::launch_layer<false>(g, (cudaStream_t)stream);
}

extern "C" int fvm_mp_layer(const float* h, const int32_t* nbr, int32_t M, int32_t KN, const void* Wt,
                            const float* bias, float* h_out, const float* Wo, const float* bo, int32_t O, float* out,
                            int32_t* err, void* stream) {
    return fvm_mp_layer_train(h, nbr, M, KN, Wt, bias, h_out, nullptr, nullptr, Wo, bo, O, out, err, stream);
}

extern "C" int fvm_in_layer(const void* X, int32_t M, const void* Wt, const float* bias, float* h_out, float* Z,
                            int32_t* err, void* stream) {
    if (!X || !Wt || !bias || !h_out || M <= 0 || !err) return FVM_E_ARG;
    auto a32 = [](const void* p) { return ((uintptr_t)p & 31u) == 0; };
    if (!a32(h_out) || !a32(Z) || (uintptr_t)X % 16 || (uintptr_t)Wt % 16) return FVM_E_ARG;
    corr::LayerArgs g{};
    g.X = static_cast<const __nv_bfloat16*>(X);
    g.M = M;
    g.Wt = static_cast<const __nv_bfloat16*>(Wt);
    g.bias = bias;
    g.h_out = h_out;
    g.Z = Z;
    g.err = err;
    return corr::launch_layer<true>(g, (cudaStream_t)stream);
}

extern "C" int fvm_corrector_in_layer_keep(const float* state, const float* r0, const float* dt, float k,
                                           const int32_t* cell_case, int32_t N, int32_t C, const float* mean,
                                           const float* inv_std, const float* geo, int32_t G, float* base, void* X,
                                           const void* Wt, const float* bias, float* h_out, int32_t* err,
                                           void* stream) {
    if (!state || !r0 || !dt || !mean || !inv_std || (G > 0 && !geo) || !base || !Wt || !bias || !h_out || !err ||
        N <= 0 || G < 0 || (C != 4 && C != 5) || 2 * C + G > corr::kLayerW)
        return FVM_E_ARG;
    if (((uintptr_t)h_out & 31u) || (uintptr_t)Wt % 16 || (uintptr_t)X % 16) return FVM_E_ARG;
    corr::LayerArgs g{};
    g.M = N;
    g.state = state;
    g.r0 = r0;
    g.dt = dt;
    g.mean = mean;
    g.inv_std = inv_std;
    g.geo = geo;
    g.cell_case = cell_case;
    g.base = base;
    g.Xout = static_cast<__nv_bfloat16*>(X);
    g.C = C;
    g.G = G;
    g.whole = (((uintptr_t)state | (uintptr_t)r0 | (uintptr_t)base) & 15u) == 0;
    g.k = k;
    g.Wt = static_cast<const __nv_bfloat16*>(Wt);
    g.bias = bias;
    g.h_out = h_out;
    g.err = err;
    return corr::launch_layer<true>(g, (cudaStream_t)stream);
}

extern "C" int fvm_corrector_in_layer(const float* state, const float* r0, const float* dt, int32_t k,
                                      const int32_t* cell_case, int32_t N, int32_t C, const float* mean,
                                      const float* inv_std, const float* geo, int32_t G, float* base, const void* Wt,
                                      const float* bias, float* h_out, int32_t* err, void* stream) {
    if (k < 1) return FVM_E_ARG;
    return fvm_corrector_in_layer_keep(state, r0, dt, (float)k, cell_case, N, C, mean, inv_std, geo, G, base, nullptr, Wt, bias,
                                       h_out, err, stream);
}

extern "C" int fvm_mp_gather_f32(const float* h, const int32_t* nbr, int32_t N, int32_t KN, void* out, void* stream) {
    if (!h || !nbr || !out || N <= 0 || KN <= 0 || KN > 8 || ((uintptr_t)h & 31u) || ((uintptr_t)out & 15u))
        return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    FVM_LAUNCH(KID_CORRECTOR, s, corr::k_mp_gather_f32<<<corr::nblk((int64_t)N * 8, 256), 256, 0, s>>>(
                                     h, nbr, N, KN, static_cast<__nv_bfloat16*>(out)));
    return launch_status();
}

extern "C" int fvm_decoder_f32(const float* h, const float* Wo, const float* bo, int32_t N, int32_t O, float* out,
                               void* stream) {
    if (!h || !Wo || !bo || !out || N <= 0 || O < 1 || O > 8 || ((uintptr_t)h & 31u)) return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    FVM_LAUNCH(KID_CORRECTOR, s, corr::k_decoder_f32<<<corr::nblk(N, 256), 256, 0, s>>>(h, Wo, bo, N, O, out));
    return launch_status();
}

// ------------------------------------------------------------------------------------------
// Backward pass of the network (fvm_back_top, fvm_back_layer, fvm_back_gather, fvm_back_bias,
// fvm_back_decoder, fvm_back_finish).
//
// Per layer two kernels walk the cells:
//   * k_back_layer: dA = dZ W (the first 64 columns as they are, the others divided by the row's
//     neighbour count) and dW += dZ^T A, both on tcgen05 from one staged copy of the tile;
//   * k_back_gather: dh_l = dh_{l+1} + dA[:, :64] + sum over neighbours of dA[:, 64:], then
//     dZ = dh_l SiLU'(Z_l) for the layer below.
// Both are bound by memory: 0.9 kB and 1.7 kB per cell and layer (52 and 86 us at 278 k cells, 4.8 and
// 5.4 TB/s).  They replace a SiLU kernel
// with one atomic per element (1178 us per layer at 278 k cells), two transposes, two GEMMs with
// their operands read again and a scatter that counted every neighbour's neighbours.
//
// Column sums (the gradients of the biases and of the decoder) follow one running fp32 accumulator over the
// cells, rounding error included: with terms of one sign that error is systematic (1.6e-4 of the decoder's
// gradient at 278 k cells), and trained weights would move with it if pieces were summed from zero, which
// is closer to the exact sum (5e-7) and would save the second pass.  Rounding a + t depends on a mostly
// through its binade, so a block walks a contiguous range of rows with one accumulator per half-warp, each
// started from the sum of the blocks before it (a first pass over the same terms); what an accumulator
// gained is exact while it stays in its binade.  With 296 blocks of 24 half-warps the result is within
// 3e-6 of the running sum, not equal to it, and it does not depend on scheduling.  The first pass runs in
// the kernel that produces the terms, the second in the next kernel that reads them, and the blocks'
// increments are added up once at the end (k_back_finish).
// ------------------------------------------------------------------------------------------
namespace fvm {
namespace corr {

// A block owns a contiguous range of rows; its half-warps (16 lanes with four channels each) take them in
// turn, a row as one 256-byte piece, with the loads of two to four rows issued together.  At 278 k cells:
// gather 86 us, input bias 29, decoder 31, top 51; with a range per warp and two channels per lane
// (4736 streams, and the compiler's own unrolling) 116, 47, 45 and 65.
constexpr int kSumBlocks = 2 * 148, kSumThreads = 384, kSumParts = kSumThreads / 16;
// One set of 64 column sums: the blocks' sums, the blocks' increments.
constexpr int kSumSet = 2 * kSumBlocks * kLayerW;
static_assert(kSumSet == FVM_BACK_SET, "workspace size");
__host__ __device__ __forceinline__ constexpr int set_block(int b) { return b * kLayerW; }
__host__ __device__ __forceinline__ constexpr int set_delta(int b) { return (kSumBlocks + b) * kLayerW; }

struct Rows {
    int64_t lo, hi;                                      // lo, lo + kSumParts, ... below hi
};
__device__ __forceinline__ Rows part_rows(int N) {
    const int64_t per = ((int64_t)N + kSumBlocks - 1) / kSumBlocks, lo = (int64_t)blockIdx.x * per;
    return Rows{lo + (threadIdx.x >> 4), min(lo + per, (int64_t)N)};
}
__device__ __forceinline__ float4 ldf4(const float* p, int64_t i) { return __ldg(reinterpret_cast<const float4*>(p) + i); }
__device__ __forceinline__ float4 f4(float v) { return make_float4(v, v, v, v); }
__device__ __forceinline__ float4 add4(float4 a, float4 b) {
    return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
}
__device__ __forceinline__ float4 mul4(float d, float4 b) {
    return make_float4(__fmul_rn(d, b.x), __fmul_rn(d, b.y), __fmul_rn(d, b.z), __fmul_rn(d, b.w));
}
__device__ __forceinline__ float4 fma4(float d, float4 b, float4 c) {
    return make_float4(fmaf(d, b.x, c.x), fmaf(d, b.y, c.y), fmaf(d, b.z, c.z), fmaf(d, b.w, c.w));
}

// First pass: this half-warp's sums of channels 4 l .. 4 l + 3 -> the set; block-wide call.
__device__ __forceinline__ void put_sums(float* set, float4 v, float (*smem)[kLayerW]) {
    const int h = threadIdx.x >> 4, l = threadIdx.x & 15;
    __syncthreads();
    reinterpret_cast<float4*>(smem[h])[l] = v;
    __syncthreads();
    if (threadIdx.x < kLayerW) {
        float t = 0.f;
#pragma unroll 8
        for (int q = 0; q < kSumParts; ++q) t += smem[q][threadIdx.x];
        set[set_block(blockIdx.x) + threadIdx.x] = t;
    }
}
// Second pass: the sums of everything before this block's range, for S consecutive sets; block-wide call.
template <int S>
__device__ __forceinline__ void get_prefix(const float* set, float4 (&out)[S], float (*smem)[kLayerW]) {
    const int h = threadIdx.x >> 4, l = threadIdx.x & 15;
    constexpr int kLoads = (kSumBlocks + kSumParts - 1) / kSumParts;
#pragma unroll
    for (int o = 0; o < S; ++o) {
        float4 t = f4(0.f);
#pragma unroll
        for (int j = 0; j < kLoads; ++j) {
            const int b = h + j * kSumParts;
            if (b < (int)blockIdx.x)
                t = add4(t, __ldcg(reinterpret_cast<const float4*>(set + (int64_t)o * kSumSet + set_block(b)) + l));
        }
        __syncthreads();
        reinterpret_cast<float4*>(smem[h])[l] = t;
        __syncthreads();
        t = f4(0.f);
#pragma unroll 8
        for (int q = 0; q < kSumParts; ++q) t = add4(t, reinterpret_cast<const float4*>(smem[q])[l]);
        out[o] = t;
    }
}
// What an accumulator gained; an infinity it started from is an earlier block's, which counted it.
__device__ __forceinline__ float gain(float acc, float start) { return acc == start ? 0.f : acc - start; }
// Second pass: what this half-warp's accumulator gained -> the block's increment; block-wide call.
__device__ __forceinline__ void put_delta(float* set, float4 acc, float4 start, float (*smem)[kLayerW]) {
    const int h = threadIdx.x >> 4, l = threadIdx.x & 15;
    __syncthreads();
    reinterpret_cast<float4*>(smem[h])[l] =
        make_float4(gain(acc.x, start.x), gain(acc.y, start.y), gain(acc.z, start.z), gain(acc.w, start.w));
    __syncthreads();
    if (threadIdx.x < kLayerW) {
        double t = 0.0;
#pragma unroll 8
        for (int q = 0; q < kSumParts; ++q) t += (double)smem[q][threadIdx.x];
        set[set_delta(blockIdx.x) + threadIdx.x] = (float)t;
    }
}

// dh * SiLU'(z)
__device__ __forceinline__ float silu_grad(float dh, float z) {
    const float s = 1.f / (1.f + __expf(-z));
    return dh * s * (1.f + z * (1.f - s));
}
__device__ __forceinline__ float4 silu_grad4(float4 dh, float4 z) {
    return make_float4(silu_grad(dh.x, z.x), silu_grad(dh.y, z.y), silu_grad(dh.z, z.z), silu_grad(dh.w, z.w));
}
__device__ __forceinline__ void st_bf4(__nv_bfloat16* p, int64_t i, float4 v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    reinterpret_cast<uint2*>(p)[i] =
        make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
// Lane l's value of column l (l < 16) <-> columns 4 l .. 4 l + 3 of a set (the others are zero).
__device__ __forceinline__ float4 spread(float v) {
    const int lane = threadIdx.x & 31, l = lane & 15, base = lane & 16;
    float t[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        t[e] = __shfl_sync(0xffffffffu, v, base | ((4 * l + e) & 15));
        if (4 * l + e >= 16) t[e] = 0.f;
    }
    return make_float4(t[0], t[1], t[2], t[3]);
}
__device__ __forceinline__ float pick(float4 v) {
    const int lane = threadIdx.x & 31, l = lane & 15, src = (lane & 16) | (l >> 2);
    const float x = __shfl_sync(0xffffffffu, v.x, src), y = __shfl_sync(0xffffffffu, v.y, src);
    const float z = __shfl_sync(0xffffffffu, v.z, src), w = __shfl_sync(0xffffffffu, v.w, src);
    return (l & 2) ? ((l & 1) ? w : z) : ((l & 1) ? y : x);
}

// Decoder backward and the last layer's dZ: dh = dOut Wo, dZ = dh SiLU'(Z); first pass of the sums of
// dOut^T h, dOut (sets [O] and [1] at `dec`) and dZ (`bias`).
template <int O>
__global__ void __launch_bounds__(kSumThreads, 2) k_back_top(const float* __restrict__ h, const float* __restrict__ Wo,
                                                          const float* __restrict__ dOut, const float* __restrict__ Z,
                                                          int N, float* __restrict__ dh, __nv_bfloat16* __restrict__ dZ,
                                                          float* __restrict__ dec, float* __restrict__ bias) {
    __shared__ __align__(16) float smem[kSumParts][kLayerW];
    __shared__ __align__(16) float s_wo[O][kLayerW];
    const int l = threadIdx.x & 15;
    for (int t = threadIdx.x; t < O * kLayerW; t += kSumThreads) s_wo[t / kLayerW][t % kLayerW] = __ldg(Wo + t);
    __syncthreads();
    float4 aw[O], ab = f4(0.f);
    float ao = 0.f;                                          // column l of dOut
#pragma unroll
    for (int o = 0; o < O; ++o) aw[o] = f4(0.f);
    const Rows r = part_rows(N);
    constexpr int kBatch = 2;                             // rows in flight; past the range they add +0
    for (int64_t i0 = r.lo; i0 < r.hi; i0 += kBatch * kSumParts) {
        float4 x[kBatch], z[kBatch];
        float d[kBatch][O], c[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int64_t i = i0 + u * kSumParts;
            const bool on = i < r.hi;
            x[u] = on ? ldf4(h, i * 16 + l) : f4(0.f);
            z[u] = on ? ldf4(Z, i * 16 + l) : f4(0.f);
            c[u] = on && l < O ? __ldg(dOut + i * O + l) : 0.f;
#pragma unroll
            for (int o = 0; o < O; ++o) d[u][o] = on ? __ldg(dOut + i * O + o) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int64_t i = i0 + u * kSumParts;
            float4 v = f4(0.f);
#pragma unroll
            for (int o = 0; o < O; ++o) {
                v = fma4(d[u][o], reinterpret_cast<const float4*>(s_wo[o])[l], v);
                aw[o] = fma4(d[u][o], x[u], aw[o]);
            }
            ao += c[u];
            const float4 g = silu_grad4(v, z[u]);
            if (i < r.hi) {
                reinterpret_cast<float4*>(dh)[i * 16 + l] = v;
                st_bf4(dZ, i * 16 + l, g);
            }
            ab = add4(ab, g);
        }
    }
#pragma unroll
    for (int o = 0; o < O; ++o) put_sums(dec + (int64_t)o * kSumSet, aw[o], smem);
    put_sums(dec + (int64_t)O * kSumSet, spread(ao), smem);
    put_sums(bias, ab, smem);
}

// Second pass of the decoder's sums.
template <int O>
__global__ void __launch_bounds__(kSumThreads, 2) k_back_decoder(const float* __restrict__ h,
                                                              const float* __restrict__ dOut, int N,
                                                              float* __restrict__ dec) {
    __shared__ __align__(16) float smem[kSumParts][kLayerW];
    const int l = threadIdx.x & 15;
    float4 s0[O + 1], a[O];
    get_prefix<O + 1>(dec, s0, smem);
#pragma unroll
    for (int o = 0; o < O; ++o) a[o] = s0[o];
    const float so = pick(s0[O]);
    float ao = so;                                           // column l of dOut
    const Rows r = part_rows(N);
    constexpr int kBatch = 4;                             // rows in flight; past the range they add +0
    const int h0 = threadIdx.x >> 4;                      // block-uniform trips: the shuffles need both halves
    for (int64_t i0 = r.lo - h0; i0 < r.hi; i0 += kBatch * kSumParts) {
        float4 x[kBatch];
        float c[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int64_t i = i0 + h0 + u * kSumParts;
            x[u] = i < r.hi ? ldf4(h, i * 16 + l) : f4(0.f);
            c[u] = i < r.hi && l < O ? __ldg(dOut + i * O + l) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
#pragma unroll
            for (int o = 0; o < O; ++o)
                a[o] = add4(a[o], mul4(__shfl_sync(0xffffffffu, c[u], (threadIdx.x & 16) | o), x[u]));
            ao = __fadd_rn(ao, c[u]);
        }
    }
#pragma unroll
    for (int o = 0; o < O; ++o) put_delta(dec + (int64_t)o * kSumSet, a[o], s0[o], smem);
    put_delta(dec + (int64_t)O * kSumSet, spread(ao), spread(so), smem);
}

// Second pass of a bias gradient on its own (the input layer's).
__global__ void __launch_bounds__(kSumThreads, 2) k_back_bias(const float* __restrict__ dh, const float* __restrict__ Z,
                                                           int N, float* __restrict__ bias) {
    __shared__ __align__(16) float smem[kSumParts][kLayerW];
    const int l = threadIdx.x & 15;
    float4 s0[1];
    get_prefix<1>(bias, s0, smem);
    float4 a = s0[0];
    const Rows r = part_rows(N);
    constexpr int kBatch = 4;                             // rows in flight; past the range they add +0
    for (int64_t i0 = r.lo; i0 < r.hi; i0 += kBatch * kSumParts) {
        float4 d[kBatch], z[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int64_t i = i0 + u * kSumParts;
            d[u] = i < r.hi ? ldf4(dh, i * 16 + l) : f4(0.f);
            z[u] = i < r.hi ? ldf4(Z, i * 16 + l) : f4(0.f);
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) a = add4(a, silu_grad4(d[u], z[u]));
    }
    put_delta(bias, a, s0[0], smem);
}

// dh = dh_in + dA[:, :64] + sum_{j in nbr} dA[j][64:], in that order; dZ = dh SiLU'(Z) with the first
// pass of its column sums (bias), and the second pass of the layer above's (dh_in, Z_in, bias_in).
// KM bounds the neighbour count at compile time; the lists are fetched a row ahead.
template <int KM>
__global__ void __launch_bounds__(kSumThreads, 2) k_back_gather(
    const float* __restrict__ dA, const int32_t* __restrict__ nbr, int N, int KN, const float* __restrict__ dh_in,
    const float* __restrict__ Z_in, float* __restrict__ bias_in, const float* __restrict__ Z, float* __restrict__ dh,
    __nv_bfloat16* __restrict__ dZ, float* __restrict__ bias) {
    __shared__ __align__(16) float smem[kSumParts][kLayerW], s_start[kSumParts][kLayerW];
    const int l = threadIdx.x & 15;
    float4 s0[1], ab = f4(0.f);
    get_prefix<1>(bias_in, s0, smem);
    float4 a = s0[0];
    float4* start = reinterpret_cast<float4*>(s_start[threadIdx.x >> 4]) + l;   // this thread's own, out of the registers
    *start = a;
    const Rows r = part_rows(N);
    int next[KM];
    auto fetch = [&](int64_t i) {
#pragma unroll
        for (int q = 0; q < KM; ++q) next[q] = q < KN && i < r.hi ? __ldg(nbr + i * KN + q) : -1;
    };
    fetch(r.lo);
    for (int64_t i = r.lo; i < r.hi; i += kSumParts) {
        float4 nb[KM];
#pragma unroll
        for (int q = 0; q < KM; ++q) nb[q] = next[q] >= 0 ? ldf4(dA, (int64_t)next[q] * 32 + 16 + l) : f4(0.f);
        const float4 own = ldf4(dA, i * 32 + l), up = ldf4(dh_in, i * 16 + l);
        const float4 zi = ldf4(Z_in, i * 16 + l), z = ldf4(Z, i * 16 + l);
        fetch(i + kSumParts);
        a = add4(a, silu_grad4(up, zi));
        float4 v = add4(own, up);
#pragma unroll
        for (int q = 0; q < KM; ++q) v = add4(v, nb[q]);
        reinterpret_cast<float4*>(dh)[i * 16 + l] = v;
        const float4 g = silu_grad4(v, z);
        st_bf4(dZ, i * 16 + l, g);
        ab = add4(ab, g);
    }
    put_delta(bias_in, a, *start, smem);
    put_sums(bias, ab, smem);
}

struct FinishArgs {
    const float* set[32];
    float* dst[32];
    int n[32];
};
// dst[c] += the sum of a set's block increments (one block per set).
__global__ void __launch_bounds__(256) k_back_finish(FinishArgs f) {
    __shared__ double part[4][kLayerW];
    const int c = threadIdx.x & 63, q = threadIdx.x >> 6;
    const float* set = f.set[blockIdx.x];
    double t = 0.0;
#pragma unroll 8
    for (int b = q; b < kSumBlocks; b += 4) t += (double)set[set_delta(b) + c];
    part[q][c] = t;
    __syncthreads();
    if (q == 0 && c < f.n[blockIdx.x])
        f.dst[blockIdx.x][c] += (float)((part[0][c] + part[1][c]) + (part[2][c] + part[3][c]));
}

// One layer's products over the cells, a persistent kernel (one CTA per SM, 128-row tiles):
//   warp 8 copies the tile's dZ (128 x 64) and A (128 x 128, two halves) into a four-stage ring with
//   TMA in the 128-byte swizzle (64 channels of a row = one swizzled line; rows past N read as zero);
//   warp 9 issues the MMAs
//     dA  [128 x 128] = dZ . W       (K-major dZ and W^T; two accumulators)
//     dW^T [128 x 64] += A^T . dZ    (the same copies read MN-major, the tile's rows as K; two
//                                     accumulators for chunks of four tiles in turn);
//   warps 0-7 read dA (warp w: TMEM lanes 32 (w % 4), columns 64 (w / 4)), divide the neighbour half
//   by the row's neighbour count and store it, a row's 32 columns on four lanes as one 128-byte line.
//   After each chunk they also add its dW^T to their registers, and at the end the CTA's sum to dW.
// The chunks are there for accuracy: the tensor core's fp32 accumulator does not round to nearest, and its
// error grows with the rows it has taken.  Relative error of one-signed sums at 278 k and 4.1 M rows: one
// accumulator for the whole run 5.0e-6 and 1.4e-4, split-K products over 512 ranges 1.1e-6 and 3.5e-5, chunks
// of 512 rows summed in registers 8.4e-7 and 9.1e-7 (at less than 1 % of a training step).
// Without dA (the input layer) A is the [N][64] feature rows and only dW is formed.
// Bound by memory, 0.9 kB per row.  Copies by four warps' cp.async into no-swizzle operands held the L1's
// path for 3000 cycles per tile, and their warp also issued the MMAs (2200 cycles per tile); with stores
// of one row per lane that took 75 us per layer at 278 k rows.
constexpr int kBackThreads = 320, kBackStages = 4;
constexpr int kChunkTiles = 4;                                                   // tiles per dW^T accumulation
constexpr int kBackHalf = TM * kLayerW * 2;                                      // 128 rows x 64 channels
constexpr int kBackStage = 3 * kBackHalf;                                        // dZ and A of one tile
constexpr int kBackSmem = 1024 + kBackStages * kBackStage + 8 * kUnitBytes;      // + alignment, W^T (128 x 64)

// 128-byte-swizzled operand: atoms of 8 rows x 128 bytes, 1024 bytes apart along the rows; `lbo` apart
// along the channels (MN-major reads of more than 64 channels).
__device__ __forceinline__ uint64_t make_desc_sw(uint32_t saddr, uint32_t lbo) {
    return make_desc(saddr, lbo, 1024) | (uint64_t)2 << 61;
}
__device__ __forceinline__ void tma_tile(uint32_t dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

template <bool LAYER>
__global__ void __launch_bounds__(kBackThreads, 1) k_back_layer(const __grid_constant__ CUtensorMap map_z,
                                                                const __grid_constant__ CUtensorMap map_a,
                                                                const __nv_bfloat16* __restrict__ WT,
                                                                const int32_t* __restrict__ nbr, int KN, int N,
                                                                float* __restrict__ dA, float* __restrict__ dW,
                                                                int* __restrict__ err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    uint8_t* sW = smem + kBackStages * kBackStage;
    __shared__ __align__(8) uint64_t bar_load[kBackStages], bar_free[kBackStages], bar_full[2], bar_empty[2];
    __shared__ __align__(8) uint64_t bar_wfull[2], bar_wfree[2], bar_done;
    __shared__ uint32_t s_taddr;
    __shared__ int s_fail;
    constexpr int AU = LAYER ? 16 : 8;                    // 8-channel units of an A row
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ntiles = (N + TM - 1) / TM;
    const int nlocal = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_taddr)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int b = 0; b < kBackStages; ++b) {
            mbar_init(&bar_load[b], 1);
            mbar_init(&bar_free[b], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&bar_full[b], 1);
            mbar_init(&bar_empty[b], 8);
            mbar_init(&bar_wfull[b], 1);
            mbar_init(&bar_wfree[b], 8);
        }
        mbar_init(&bar_done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
        s_fail = 0;
    }
    if (LAYER) {
        for (int t = tid; t < TM * 8; t += kBackThreads)
            *reinterpret_cast<uint4*>(sW + (t & 7) * kUnitBytes + frag_col(t >> 3) * 16) =
                *reinterpret_cast<const uint4*>(WT + (int64_t)(t >> 3) * kLayerW + 8 * (t & 7));
    } else {   // rows 64..127 of the input layer's dW^T read zeros
        for (int st = 0; st < kBackStages; ++st)
            for (int t = tid; t < kBackHalf / 16; t += kBackThreads)
                reinterpret_cast<uint4*>(smem + st * kBackStage + 2 * kBackHalf)[t] = make_uint4(0u, 0u, 0u, 0u);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t taddr = s_taddr, tw = taddr + 256;     // dA: columns 0..255, dW^T: 256..383
    const uint32_t id_a = make_idesc(TM);
    const uint32_t id_w = make_idesc(kLayerW) | (1u << 15) | (1u << 16);   // both operands MN-major
    float sum[32];                                        // warps 0-7: dW^T, input channel 32 (w % 4) + lane,
#pragma unroll                                            // output channels 32 (w / 4) ..
    for (int n = 0; n < 32; ++n) sum[n] = 0.f;
    // Chunk c's dW^T -> the sums (warps 0-7, all lanes).
    auto take = [&](int c) {
        const bool ok = mbar_wait(&bar_wfull[c & 1], (uint32_t)((c >> 1) & 1));
        if (!__all_sync(0xffffffffu, ok)) {
            if (lane == 0) atomicExch(&s_fail, 1);
            return false;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        uint32_t v[32];
        tmem_ld32(tw + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(kLayerW * (c & 1) + 32 * (warp >> 2)), v);
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_wfree[c & 1]);
#pragma unroll
        for (int n = 0; n < 32; ++n) sum[n] += __uint_as_float(v[n]);
        return true;
    };

    if (warp == 8) {
        if (lane == 0) {
            int k = 0;
            for (; k < nlocal; ++k) {
                const int st = k % kBackStages, m0 = ((int)blockIdx.x + k * (int)gridDim.x) * TM;
                if (k >= kBackStages && !mbar_wait(&bar_free[st], (uint32_t)((k / kBackStages - 1) & 1))) {
                    atomicExch(&s_fail, 1);
                    break;
                }
                const uint32_t sz = smem_u32(smem + st * kBackStage);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&bar_load[st])),
                             "r"((LAYER ? 3 : 2) * kBackHalf)
                             : "memory");
                tma_tile(sz, &map_z, 0, m0, &bar_load[st]);
                tma_tile(sz + kBackHalf, &map_a, 0, m0, &bar_load[st]);
                if (LAYER) tma_tile(sz + 2 * kBackHalf, &map_a, kLayerW, m0, &bar_load[st]);
            }
            // no copy outlives the CTA, also when a wait gave up
            for (int j = max(0, k - kBackStages); j < k; ++j)
                if (!mbar_wait(&bar_load[j % kBackStages], (uint32_t)((j / kBackStages) & 1))) atomicExch(&s_fail, 1);
        }
    } else if (warp == 9) {
        if (lane == 0) {
            for (int k = 0; k < nlocal; ++k) {
                const int a = k & 1, st = k % kBackStages, c = k / kChunkTiles;
                const bool first = k % kChunkTiles == 0, last = (k + 1) % kChunkTiles == 0 || k + 1 == nlocal;
                if (!mbar_wait(&bar_load[st], (uint32_t)((k / kBackStages) & 1)) ||
                    (LAYER && k >= 2 && !mbar_wait(&bar_empty[a], (uint32_t)(((k >> 1) - 1) & 1))) ||
                    (first && c >= 2 && !mbar_wait(&bar_wfree[c & 1], (uint32_t)(((c >> 1) - 1) & 1)))) {
                    atomicExch(&s_fail, 1);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
                const uint32_t sz = smem_u32(smem + st * kBackStage), sa = sz + kBackHalf;
                if (LAYER)
#pragma unroll
                    for (int q = 0; q < kLayerW / 16; ++q)
                        tc_mma(taddr + a * TM, make_desc_sw(sz + 32 * q, 16),
                               make_desc(smem_u32(sW) + 2 * q * kUnitBytes, kUnitBytes, 128), id_a, q > 0);
#pragma unroll
                for (int q = 0; q < TM / 16; ++q)
                    tc_mma(tw + kLayerW * (c & 1), make_desc_sw(sa + 2048 * q, kBackHalf),
                           make_desc_sw(sz + 2048 * q, kBackHalf), id_w, !first || q > 0);
                tc_commit(&bar_free[st]);
                if (LAYER) tc_commit(&bar_full[a]);
                if (last) tc_commit(&bar_wfull[c & 1]);
            }
            // Covers every MMA issued, also when a wait gave up.  A barrier of its own, completed once: of
            // bar_full several phases can be open where no reader follows them (the input layer), and a
            // parity then says nothing about the last one.
            tc_commit(&bar_done);
        }
    } else if (LAYER) {
        const int half = warp >> 2;
        int next[8];                                      // row `lane`'s neighbours, fetched a tile ahead
        auto fetch = [&](int k) {
            const int64_t row = (int64_t)((int)blockIdx.x + k * (int)gridDim.x) * TM + 32 * (warp & 3) + lane;
#pragma unroll
            for (int q = 0; q < 8; ++q) next[q] = half && k < nlocal && row < N && q < KN ? __ldg(nbr + row * KN + q) : -1;
        };
        fetch(0);
        for (int k = 0; k < nlocal; ++k) {
            const int a = k & 1;
            const int64_t m0 = (int64_t)((int)blockIdx.x + k * (int)gridDim.x) * TM + 32 * (warp & 3);
            int deg = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) deg += next[q] >= 0;
            fetch(k + 1);
            const bool ok = mbar_wait(&bar_full[a], (uint32_t)((k >> 1) & 1));
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) atomicExch(&s_fail, 1);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            uint32_t v[2][2][16];                         // 16-row group, 32-column group
            const uint32_t base = taddr + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(a * TM + 64 * half);
#pragma unroll
            for (int t = 0; t < 4; ++t) tmem_ld_frag(base + ((uint32_t)(16 * (t >> 1)) << 16) + 32 * (t & 1), v[t >> 1][t & 1]);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;");
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_empty[a]);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int r = 8 * t + (lane >> 2);
                const float d = (float)max(__shfl_sync(0xffffffffu, deg, r), 1);
                if (m0 + r < N) {
                    float* dst = dA + (m0 + r) * TM + 64 * half + 8 * (lane & 3);
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        float x[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            x[e] = __uint_as_float(v[t >> 1][c][4 * (e >> 1) + 2 * (t & 1) + (e & 1)]);
                            if (half) x[e] = x[e] / d;
                        }
                        st8(dst + 32 * c, x);
                    }
                }
            }
            if (((k + 1) % kChunkTiles == 0 || k + 1 == nlocal) && !take(k / kChunkTiles)) break;
        }
    } else {
        for (int c = 0; c * kChunkTiles < nlocal; ++c)
            if (!take(c)) break;
    }
    __syncthreads();
    // no MMA is in flight past this point (a second bounded chance before tensor memory is released)
    const bool done = mbar_wait(&bar_done, 0u);
    if (!__syncthreads_and(done) || s_fail) {
        if (tid == 0) atomicExch(err, 1);
        if (!done) mbar_wait(&bar_done, 0u);
    } else if (warp < 8) {
        const int in = 32 * (warp & 3) + lane;            // input channel
        if (in < 8 * AU)
#pragma unroll
            for (int n = 0; n < 32; ++n) atomicAdd(dW + (int64_t)(32 * (warp >> 2) + n) * (8 * AU) + in, sum[n]);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(512u));
}

// Tensor map of bf16 rows [N][cols] in boxes of 128 rows x 64 columns, 128-byte swizzle.
static bool tile_map(CUtensorMap* map, const void* base, int cols, int N) {
    using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<Encode>(f);
    }();
    if (!encode) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)N}, strides[1] = {(cuuint64_t)cols * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kLayerW, (cuuint32_t)TM}, step[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, step,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool LAYER>
static int launch_back_layer(const void* dZ, const void* A, const void* WT, const int32_t* nbr, int KN, int N,
                             float* dA, float* dW, int* err, cudaStream_t s) {
    static int sms[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) {
        launch_status();
        return FVM_E_CUDA;
    }
    if (!sms[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaFuncSetAttribute(k_back_layer<LAYER>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBackSmem) !=
                cudaSuccess) {
            launch_status();
            return FVM_E_CUDA;
        }
        sms[dev] = n;
    }
    CUtensorMap map_z, map_a;
    if (!tile_map(&map_z, dZ, kLayerW, N) || !tile_map(&map_a, A, LAYER ? 2 * kLayerW : kLayerW, N)) return FVM_E_CUDA;
    const unsigned grid = (unsigned)std::min((N + TM - 1) / TM, sms[dev]);
    FVM_LAUNCH(KID_CORRECTOR, s, k_back_layer<LAYER><<<grid, kBackThreads, kBackSmem, s>>>(
                                     map_z, map_a, static_cast<const __nv_bfloat16*>(WT), nbr, KN, N, dA, dW, err));
    return launch_status();
}

static inline bool aligned(const void* p, int b) { return ((uintptr_t)p & (b - 1)) == 0; }

}  // namespace corr
}  // namespace fvm

#define FVM_BY_OUTPUTS(O, CALL)  \
    switch (O) {                 \
        case 1: CALL(1); break;  \
        case 2: CALL(2); break;  \
        case 3: CALL(3); break;  \
        case 4: CALL(4); break;  \
        case 5: CALL(5); break;  \
        case 6: CALL(6); break;  \
        case 7: CALL(7); break;  \
        default: CALL(8); break; \
    }

extern "C" int fvm_back_top(const float* h, const float* Wo, const float* dOut, const float* Z, int32_t N, int32_t O,
                            float* dh, void* dZ, float* dec, float* bias, void* stream) {
    if (!h || !Wo || !dOut || !Z || !dh || !dZ || !dec || !bias || N <= 0 || O < 1 || O > 8) return FVM_E_ARG;
    if (!corr::aligned(h, 16) || !corr::aligned(Z, 16) || !corr::aligned(dh, 16) || !corr::aligned(dZ, 8) ||
        !corr::aligned(dec, 16) || !corr::aligned(bias, 16))
        return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    __nv_bfloat16* z = static_cast<__nv_bfloat16*>(dZ);
#define FVM_CALL(OO) FVM_LAUNCH(KID_CORRECTOR, s, corr::k_back_top<OO><<<corr::kSumBlocks, corr::kSumThreads, 0, s>>>( \
                                    h, Wo, dOut, Z, N, dh, z, dec, bias))
    FVM_BY_OUTPUTS(O, FVM_CALL)
#undef FVM_CALL
    return launch_status();
}

extern "C" int fvm_back_decoder(const float* h, const float* dOut, int32_t N, int32_t O, float* dec, void* stream) {
    if (!h || !dOut || !dec || N <= 0 || O < 1 || O > 8 || !corr::aligned(h, 16) || !corr::aligned(dec, 16))
        return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
#define FVM_CALL(OO) FVM_LAUNCH(KID_CORRECTOR, s, corr::k_back_decoder<OO><<<corr::kSumBlocks, corr::kSumThreads, 0, s>>>( \
                                    h, dOut, N, dec))
    FVM_BY_OUTPUTS(O, FVM_CALL)
#undef FVM_CALL
    return launch_status();
}

extern "C" int fvm_back_layer(const void* dZ, const void* A, const void* WT, const int32_t* nbr, int32_t KN, int32_t N,
                              float* dA, float* dW, int32_t* err, void* stream) {
    if (!dZ || !A || !dW || !err || N <= 0 || !corr::aligned(dZ, 16) || !corr::aligned(A, 16)) return FVM_E_ARG;
    if (dA && (!WT || !nbr || KN <= 0 || KN > 8 || !corr::aligned(dA, 32) || !corr::aligned(WT, 16))) return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    return dA ? corr::launch_back_layer<true>(dZ, A, WT, nbr, KN, N, dA, dW, err, s)
              : corr::launch_back_layer<false>(dZ, A, nullptr, nullptr, 0, N, nullptr, dW, err, s);
}

extern "C" int fvm_back_gather(const float* dA, const int32_t* nbr, int32_t N, int32_t KN, const float* dh_in,
                               const float* Z_in, float* bias_in, const float* Z, float* dh, void* dZ, float* bias,
                               void* stream) {
    if (!dA || !nbr || !dh_in || !Z_in || !bias_in || !Z || !dh || !dZ || !bias || N <= 0 || KN <= 0 || KN > 8 ||
        dh == dh_in)
        return FVM_E_ARG;
    if (!corr::aligned(dA, 16) || !corr::aligned(dh_in, 16) || !corr::aligned(Z_in, 16) || !corr::aligned(Z, 16) ||
        !corr::aligned(dh, 16) || !corr::aligned(dZ, 8) || !corr::aligned(bias_in, 16) || !corr::aligned(bias, 16))
        return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    __nv_bfloat16* z = static_cast<__nv_bfloat16*>(dZ);
#define FVM_CALL(KM) FVM_LAUNCH(KID_CORRECTOR, s, corr::k_back_gather<KM><<<corr::kSumBlocks, corr::kSumThreads, 0, s>>>( \
                                    dA, nbr, N, KN, dh_in, Z_in, bias_in, Z, dh, z, bias))
    if (KN <= 3) FVM_CALL(3);
    else if (KN == 4) FVM_CALL(4);
    else FVM_CALL(8);
#undef FVM_CALL
    return launch_status();
}

extern "C" int fvm_back_bias(const float* dh, const float* Z, int32_t N, float* bias, void* stream) {
    if (!dh || !Z || !bias || N <= 0 || !corr::aligned(dh, 16) || !corr::aligned(Z, 16) || !corr::aligned(bias, 16))
        return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    FVM_LAUNCH(KID_CORRECTOR, s, corr::k_back_bias<<<corr::kSumBlocks, corr::kSumThreads, 0, s>>>(dh, Z, N, bias));
    return launch_status();
}

extern "C" int fvm_back_finish(int32_t n_sets, const float* const* sets, float* const* dst, const int32_t* n,
                               void* stream) {
    if (n_sets < 1 || n_sets > 32 || !sets || !dst || !n) return FVM_E_ARG;
    corr::FinishArgs f{};
    for (int q = 0; q < n_sets; ++q) {
        if (!sets[q] || !dst[q] || n[q] < 1 || n[q] > corr::kLayerW) return FVM_E_ARG;
        f.set[q] = sets[q];
        f.dst[q] = dst[q];
        f.n[q] = n[q];
    }
    cudaStream_t s = (cudaStream_t)stream;
    FVM_LAUNCH(KID_CORRECTOR, s, corr::k_back_finish<<<n_sets, 256, 0, s>>>(f));
    return launch_status();
}

// ------------------------------------------------------------------------------------------
// Acceptance checks of a corrector proposal, per case, in two launches (fvm_corrector_checks).
//   sums[c] (FP64, 3C + 4 slots): sum vol U, sum vol P, sum vol r0 (C each), sum vol |r0|^2,
//   sum vol |r1|^2, number of inadmissible cells of P (rho <= 0, internal energy <= 0 or not finite),
//   sum vol |P - U - k dt_c (r0 + r1) / 2|^2 (the proposal against the trapezoidal rule over the
//   window).  ok[c] = drift <= tol && |r1|^2 <= ratio^2 |r0|^2 && drift finite && no inadmissible
//   cell [&& trapezoid distance <= consistency * k dt_c |r0| when consistency > 0], with drift =
//   max over mass and energy of |sum vol P - (sum vol U + k dt_c sum vol r0)| / |sum vol U|.
// The reduction walks one contiguous chunk of cells per warp and flushes per case change (cells of
// a case are contiguous), as the conservation sums do; the verdict kernel clears the sums after
// reading them, so the pair can be replayed from a CUDA graph.
// ------------------------------------------------------------------------------------------
namespace fvm {
namespace corr {

template <int C>
__global__ void k_checks_reduce(const float* __restrict__ U, const float* __restrict__ P,
                                const float* __restrict__ r0, const float* __restrict__ r1,
                                const float* __restrict__ vol, const int32_t* __restrict__ cell_case, int N,
                                const float* __restrict__ dt, int k, double* __restrict__ sums) {
    constexpr int DIM = C - 2, NS = 3 * C + 4;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t chunk = (((int64_t)N + warps - 1) / warps + 31) & ~(int64_t)31;
    const int64_t beg = w * chunk, end = beg + chunk < N ? beg + chunk : (int64_t)N;
    int cur = -1;
    double acc[NS];
#pragma unroll
    for (int q = 0; q < NS; ++q) acc[q] = 0.0;
    auto flush = [&]() {
        if (cur < 0) return;
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            double v = acc[q];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(full, v, o);
            if (lane == 0) atomicAdd(sums + (int64_t)cur * NS + q, v);
            acc[q] = 0.0;
        }
    };
    for (int64_t i0 = beg; i0 < end; i0 += 32) {
        const int64_t i = i0 + lane;
        const bool live = i < end;
        const int cse = live ? __ldg(cell_case + i) : -1;
        double v[NS];
#pragma unroll
        for (int q = 0; q < NS; ++q) v[q] = 0.0;
        if (live) {
            const double vo = (double)__ldg(vol + i);
            float u[C], pp[C], a[C], b[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                u[c] = __ldg(U + i * C + c);
                pp[c] = __ldg(P + i * C + c);
                a[c] = __ldg(r0 + i * C + c);
                b[c] = __ldg(r1 + i * C + c);
            }
            const double half_kdt = 0.5 * (double)k * (double)__ldg(dt + cse);
            double n0 = 0.0, n1 = 0.0, e2 = 0.0;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                v[c] = vo * (double)u[c];
                v[C + c] = vo * (double)pp[c];
                v[2 * C + c] = vo * (double)a[c];
                n0 += vo * (double)(a[c] * a[c]);
                n1 += vo * (double)(b[c] * b[c]);
                const double e = ((double)pp[c] - (double)u[c]) - half_kdt * ((double)a[c] + (double)b[c]);
                e2 += vo * (e * e);
            }
            v[3 * C + 3] = e2;
            v[3 * C] = n0;
            v[3 * C + 1] = n1;
            const float rho = pp[DIM];
            float k2 = 0.f;
#pragma unroll
            for (int d = 0; d < DIM; ++d) k2 += pp[d] * pp[d];
            const float e_int = pp[DIM + 1] - 0.5f * k2 / rho;
            v[3 * C + 2] = (rho <= 0.f || e_int <= 0.f || !isfinite(e_int)) ? 1.0 : 0.0;
        }
        unsigned pending = __ballot_sync(full, live);
        while (pending) {
            const int lc = __shfl_sync(full, cse, __ffs(pending) - 1);
            if (lc != cur) {
                flush();
                cur = lc;
            }
            const bool mine = live && cse == lc;
            if (mine)
#pragma unroll
                for (int q = 0; q < NS; ++q) acc[q] += v[q];
            pending &= ~__ballot_sync(full, mine);
        }
    }
    flush();
}

__global__ void k_checks_verdict(double* __restrict__ sums, int n_cases, int C, const float* __restrict__ dt, int k,
                                 double tol, double ratio2, double consistency, uint8_t* __restrict__ ok,
                                 double* __restrict__ keep) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_cases) return;
    const int NS = 3 * C + 4, DIM = C - 2;
    double* s = sums + (int64_t)c * NS;
    const double kdt = (double)k * (double)dt[c];
    double drift = 0.0;
    for (int q = DIM; q < DIM + 2; ++q) {
        const double m0 = s[q], mp = s[C + q], r = s[2 * C + q];
        const double d = fabs(mp - (m0 + kdt * r)) / fabs(m0);
        drift = (d > drift || isnan(d)) ? d : drift;
    }
    const bool near_trapezoid = consistency <= 0.0 || s[3 * C + 3] <= consistency * consistency * kdt * kdt * s[3 * C];
    ok[c] = (drift <= tol && s[3 * C + 1] <= ratio2 * s[3 * C] && isfinite(drift) && s[3 * C + 2] == 0.0 &&
             near_trapezoid) ? 1 : 0;
    for (int q = 0; q < NS; ++q) {
        if (keep) keep[(int64_t)c * NS + q] = s[q];
        s[q] = 0.0;
    }
}

}  // namespace corr
}  // namespace fvm

extern "C" int fvm_corrector_checks(const float* U, const float* P, const float* r0, const float* r1,
                                    const float* volumes, const int32_t* cell_case, int32_t N, int32_t C,
                                    int32_t n_cases, const float* dt, int32_t k, double drift_tol, double ratio,
                                    double consistency, double* sums, uint8_t* ok, double* keep, void* stream) {
    if (!U || !P || !r0 || !r1 || !volumes || !cell_case || !dt || !sums || !ok || N <= 0 || n_cases <= 0 ||
        (C != 4 && C != 5) || k < 1)
        return FVM_E_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) !=
                                                      cudaSuccess) {
            launch_status();
            return FVM_E_CUDA;
        }
    }
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(4LL * sms, ((int64_t)N + 255) / 256));
    if (C == 4)
        FVM_LAUNCH(KID_CORRECTOR, s, corr::k_checks_reduce<4><<<grid, 256, 0, s>>>(U, P, r0, r1, volumes, cell_case, N,
                                                                                    dt, k, sums));
    else
        FVM_LAUNCH(KID_CORRECTOR, s, corr::k_checks_reduce<5><<<grid, 256, 0, s>>>(U, P, r0, r1, volumes, cell_case, N,
                                                                                    dt, k, sums));
    int rc = launch_status();
    if (rc) return rc;
    FVM_LAUNCH(KID_CORRECTOR, s, corr::k_checks_verdict<<<(n_cases + 127) / 128, 128, 0, s>>>(
                                     sums, n_cases, C, dt, k, drift_tol, ratio * ratio, consistency, ok, keep));
    return launch_status();
}
