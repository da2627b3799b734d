// ELL sparse operators: y = A x (+ b), Y = A X (+ b).
//
// Replaces the Triton kernels of the reference (time_fvm/utils/ell_kernel.py:25-80 ell_spmm_kernel,
// :100-132 _ell_spmv_kernel) and their wrappers (:135-210).  Differences by design:
//  * ELL is slot-major (vals[k][row]) with int32 columns: a warp reading slot k of 32 consecutive
//    rows issues one 128-byte transaction for the values and one for the columns, where the
//    reference's row-major layout strides K * 4 (8 for int64) bytes between lanes;
//  * SpMM with few columns (B = 4 or 5 conserved variables) gives each thread a whole row and up to
//    8 columns, so no lanes are masked (the reference's BLOCK_B >= 16 masks >= 69 % of them);
//  * SpMV of a multi-column x is one launch, not one launch per column (ell_kernel.py:157-165);
//  * the bias is added in-kernel after the K-slot accumulation (same order as the reference);
//  * the slot loop is unrolled to a compile-time bound (K <= FVM_MAX_ELL_K = 16), so a row's
//    gathers are issued together instead of one dependent load chain per slot.
#include "fvm_common.cuh"

namespace fvm {

// Every kernel is templated on an upper bound KT of the slot count (2, 4, 5, 6, 8, 12 or 16; five slots are the
// widest rows of the residual's operators on the reference's stencil) and unrolls the
// slot loop, so the values, columns and gathers of all slots of a row are in flight together (one
// dependent round trip per row instead of K); slots are summed in order k = 0, 1, ...
//
// The products are bound by memory (8 K bytes of values and columns per row), but with a row or two
// per thread and one block after the other they ran at the pace of the two round trips: 22 us for
// 1.3 M rows of five slots whose bytes take 9.  So one wave of blocks walks the rows (kEllBlocks per SM)
// and a thread loads the values and columns of its next RT rows (a block apart, so that each access
// stays contiguous over the warp) before it gathers for the current ones.  On the operators of a
// 438 k-tet box: facet gradient (4.4 M rows of two slots) 41 -> 22 us, cell gradient (1.3 M rows of
// five) 21 -> 14 us, with five columns 26 -> 19 us, divergence with five columns 14 -> 11 us.
//
// Rows of more than five slots, and most products with several columns, take one row per thread and no look
// ahead (the *_once kernels, all slots loaded before the first gather): a second set of that many slots leaves
// 8 to 32 warps per SM or spills, and more warps hide the two round trips better.  M rows of K slots with B
// columns, look ahead against once, in us, operator in the L2 / not there: 240 k x 6 (B 1) 5.1 / 5.6 against
// 3.5 / 5.1; 240 k x 10 (B 1) 9.4 / 11.8 against 5.2 / 7.2; 1.3 M x 16 (B 1) 43 / 45 against 35 / 36;
// 240 k x 10 (B 5) 20.9 / 24.0 against 15.9 / 17.2; 1.3 M x 5 (B 2) 28.8 / 31.0 against 22.3 / 24.8;
// 1.3 M x 16 (B 9) 373 / 376 against 272 / 274.
constexpr int kEllBlocks = 4;

template <int KT, int RT>
struct EllRows {
    float v[RT][KT];
    int c[RT][KT];
    __device__ __forceinline__ void load(const float* __restrict__ vals, const int32_t* __restrict__ cols, int64_t M,
                                         int K, int64_t r0) {
#pragma unroll
        for (int j = 0; j < RT; ++j)
#pragma unroll
            for (int k = 0; k < KT; ++k) {
                const int64_t r = r0 + j * kBlock;
                const bool on = k < K && r < M;
                v[j][k] = on ? __ldg(vals + k * M + r) : 0.f;
                c[j][k] = on ? __ldg(cols + k * M + r) : 0;
            }
    }
};

template <int KT, int RT>
__global__ void __launch_bounds__(kBlock, kEllBlocks) k_ell_spmv(const float* __restrict__ vals,
                                                                  const int32_t* __restrict__ cols, int64_t M,
                                                                  int K, const float* __restrict__ x,
                                                                  int64_t incx, const float* __restrict__ bias,
                                                                  float* __restrict__ y, int64_t incy) {
    const int64_t step = (int64_t)gridDim.x * (kBlock * RT);
    int64_t r0 = blockIdx.x * (int64_t)(kBlock * RT) + threadIdx.x;
    EllRows<KT, RT> next;
    next.load(vals, cols, M, K, r0);
    for (; r0 < M; r0 += step) {
        const EllRows<KT, RT> cur = next;
        float xv[RT][KT], b[RT];
#pragma unroll
        for (int j = 0; j < RT; ++j) {
            const bool on = r0 + j * kBlock < M;
            b[j] = on && bias ? __ldg(bias + r0 + j * kBlock) : 0.f;
#pragma unroll
            for (int k = 0; k < KT; ++k) xv[j][k] = on && k < K ? __ldg(x + (int64_t)cur.c[j][k] * incx) : 0.f;
        }
        next.load(vals, cols, M, K, r0 + step);
#pragma unroll
        for (int j = 0; j < RT; ++j) {
            const int64_t r = r0 + j * kBlock;
            if (r >= M) break;
            float acc = 0.f;
#pragma unroll
            for (int k = 0; k < KT; ++k)
                if (k < K) acc = fmaf(cur.v[j][k], xv[j][k], acc);
            if (bias) acc += b[j];
            y[r * incy] = acc;
        }
    }
}

template <int KT>
__global__ void __launch_bounds__(kBlock) k_ell_spmv_once(const float* __restrict__ vals,
                                                          const int32_t* __restrict__ cols, int64_t M,
                                                          int K, const float* __restrict__ x,
                                                          int64_t incx, const float* __restrict__ bias,
                                                          float* __restrict__ y, int64_t incy) {
    const int64_t r = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (r >= M) return;
    float v[KT], xv[KT];
    int c[KT];
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        v[k] = k < K ? __ldg(vals + k * M + r) : 0.f;
        c[k] = k < K ? __ldg(cols + k * M + r) : 0;
    }
    const float b = bias ? __ldg(bias + r) : 0.f;
#pragma unroll
    for (int k = 0; k < KT; ++k) xv[k] = k < K ? __ldg(x + (int64_t)c[k] * incx) : 0.f;
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < KT; ++k)
        if (k < K) acc = fmaf(v[k], xv[k], acc);
    if (bias) acc += b;
    y[r * incy] = acc;
}

// One thread per (row, group of CB columns).
template <int KT, int CB>
__global__ void __launch_bounds__(kBlock) k_ell_spmm_once(const float* __restrict__ vals,
                                                          const int32_t* __restrict__ cols, int64_t M,
                                                          int K, const float* __restrict__ X,
                                                          int64_t ldx, int B,
                                                          const float* __restrict__ bias,
                                                          float* __restrict__ Y, int64_t ldy) {
    const int64_t r = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (r >= M) return;
    const int c0 = blockIdx.y * CB;
    const int nb = min(CB, B - c0);
    float v[KT];
    int c[KT];
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        v[k] = k < K ? __ldg(vals + k * M + r) : 0.f;
        c[k] = k < K ? __ldg(cols + k * M + r) : 0;
    }
    float acc[CB];
#pragma unroll
    for (int j = 0; j < CB; ++j) acc[j] = 0.f;
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        if (k >= K) break;
        float xr[CB];
        const float* xk = X + (int64_t)c[k] * ldx + c0;
#pragma unroll
        for (int j = 0; j < CB; ++j) xr[j] = j < nb ? __ldg(xk + j) : 0.f;
#pragma unroll
        for (int j = 0; j < CB; ++j)
            if (j < nb) acc[j] = fmaf(v[k], xr[j], acc[j]);
    }
    const float b = bias ? __ldg(bias + r) : 0.f;
    float* yr = Y + r * ldy + c0;
#pragma unroll
    for (int j = 0; j < CB; ++j)
        if (j < nb) yr[j] = bias ? acc[j] + b : acc[j];
}

// The same for groups of CB whole columns (B a multiple of CB), with the look ahead.
template <int KT, int CB>
__global__ void __launch_bounds__(kBlock, kEllBlocks) k_ell_spmm(const float* __restrict__ vals,
                                                      const int32_t* __restrict__ cols, int64_t M,
                                                      int K, const float* __restrict__ X,
                                                      int64_t ldx,
                                                      const float* __restrict__ bias,
                                                      float* __restrict__ Y, int64_t ldy) {
    const int64_t step = (int64_t)gridDim.x * kBlock;
    int64_t r = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    const int c0 = blockIdx.y * CB;
    EllRows<KT, 1> next;
    next.load(vals, cols, M, K, r);
    for (; r < M; r += step) {
        const EllRows<KT, 1> cur = next;
        next.load(vals, cols, M, K, r + step);
        float acc[CB];
#pragma unroll
        for (int j = 0; j < CB; ++j) acc[j] = 0.f;
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            if (k >= K) break;
            float xr[CB];
            const float* xk = X + (int64_t)cur.c[0][k] * ldx + c0;
#pragma unroll
            for (int j = 0; j < CB; ++j) xr[j] = __ldg(xk + j);
#pragma unroll
            for (int j = 0; j < CB; ++j) acc[j] = fmaf(cur.v[0][k], xr[j], acc[j]);
        }
        const float b = bias ? __ldg(bias + r) : 0.f;
        float* yr = Y + r * ldy + c0;
#pragma unroll
        for (int j = 0; j < CB; ++j) yr[j] = bias ? acc[j] + b : acc[j];
    }
}

// Five columns (the 3D variables).  A slot's five floats start on any 4-byte boundary; they lie in two
// consecutive 16-byte words, which are loaded whole and shifted into place: five scalar gathers per
// slot cost the L1 41-70 cycles per warp (rows in random order), the two words 17-21.  Both words hold
// at least one of the five floats, so neither leaves the memory the row itself lies in.
constexpr int spmm5_blocks(int KT) { return KT <= 4 ? 3 : 2; }   // per SM: 40 gathered floats of a row in registers

template <int KT>
__global__ void __launch_bounds__(kBlock, spmm5_blocks(KT)) k_ell_spmm5(const float* __restrict__ vals,
                                                         const int32_t* __restrict__ cols, int64_t M,
                                                         int K, const float* __restrict__ X, int64_t ldx,
                                                         const float* __restrict__ bias,
                                                         float* __restrict__ Y, int64_t ldy) {
    const int64_t step = (int64_t)gridDim.x * kBlock;
    int64_t r = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    EllRows<KT, 1> next;
    next.load(vals, cols, M, K, r);
    for (; r < M; r += step) {
        const EllRows<KT, 1> cur = next;
        float4 w[KT][2];
        int sh[KT];
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            const uintptr_t a = reinterpret_cast<uintptr_t>(X + (int64_t)cur.c[0][k] * ldx);
            const float4* q = reinterpret_cast<const float4*>(a & ~(uintptr_t)15);
            sh[k] = (int)(a >> 2) & 3;
            w[k][0] = k < K ? __ldg(q) : make_float4(0.f, 0.f, 0.f, 0.f);
            w[k][1] = k < K ? __ldg(q + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        next.load(vals, cols, M, K, r + step);
        const float b = bias ? __ldg(bias + r) : 0.f;
        float acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            if (k >= K) break;
            const float f[8] = {w[k][0].x, w[k][0].y, w[k][0].z, w[k][0].w, w[k][1].x, w[k][1].y, w[k][1].z, w[k][1].w};
            float t[7];
#pragma unroll
            for (int j = 0; j < 7; ++j) t[j] = sh[k] & 1 ? f[j + 1] : f[j];
#pragma unroll
            for (int j = 0; j < 5; ++j) acc[j] = fmaf(cur.v[0][k], sh[k] & 2 ? t[j + 2] : t[j], acc[j]);
        }
        float* yr = Y + r * ldy;
#pragma unroll
        for (int j = 0; j < 5; ++j) yr[j] = bias ? acc[j] + b : acc[j];
    }
}

// Specialisation for 4 contiguous, 16-byte aligned columns: one float4 gather per slot.
template <int KT>
__global__ void __launch_bounds__(kBlock) k_ell_spmm4(const float* __restrict__ vals,
                                                       const int32_t* __restrict__ cols, int64_t M,
                                                       int K, const float* __restrict__ X,
                                                       const float* __restrict__ bias,
                                                       float* __restrict__ Y) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= M) return;
    float v[KT], x[KT][4];
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        v[k] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) x[k][j] = 0.f;
        if (k < K) {
            v[k] = __ldg(vals + k * M + r);
            load_row<4>(X + 4 * (int64_t)__ldg(cols + k * M + r), x[k]);
        }
    }
    float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < KT; ++k)
        if (k < K)
#pragma unroll
            for (int j = 0; j < 4; ++j) a[j] = fmaf(v[k], x[k][j], a[j]);
    if (bias) {
        const float b = __ldg(bias + r);
#pragma unroll
        for (int j = 0; j < 4; ++j) a[j] += b;
    }
    store_row<4>(Y + 4 * r, a);
}

}  // namespace fvm

#include <vector>

namespace fvm {
static thread_local int g_last_cuda_error = 0;

struct ProfState {
    bool on = false;
    int cap = 0, n = 0;
    bool overflow = false;
    std::vector<cudaEvent_t> ev;   // 2 per launch
    std::vector<int> ids;
};
static ProfState g_prof;

void prof_begin(int kid, cudaStream_t s) {
    if (!g_prof.on) return;
    if (g_prof.n >= g_prof.cap) {
        g_prof.overflow = true;
        return;
    }
    g_prof.ids[g_prof.n] = kid;
    cudaEventRecord(g_prof.ev[2 * g_prof.n], s);
}

void prof_end(cudaStream_t s) {
    if (!g_prof.on || g_prof.n >= g_prof.cap) return;
    cudaEventRecord(g_prof.ev[2 * g_prof.n + 1], s);
    ++g_prof.n;
}

int g_launch_overlap = 1;
static thread_local cudaError_t g_pending_launch_error = cudaSuccess;

void note_launch_error(cudaError_t e) {
    if (g_pending_launch_error == cudaSuccess) g_pending_launch_error = e;
}

int launch_status() {
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = g_pending_launch_error;
    g_pending_launch_error = cudaSuccess;
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return FVM_E_CUDA;
    }
    return FVM_OK;
}
}  // namespace fvm

extern "C" int fvm_set_launch_overlap(int32_t on) {
    if (on != 0 && on != 1) return FVM_E_ARG;
    fvm::g_launch_overlap = on;
    return FVM_OK;
}

extern "C" int fvm_last_cuda_error(void) { return fvm::g_last_cuda_error; }

extern "C" int fvm_profile_start(int32_t capacity) {
    using fvm::g_prof;
    if (capacity <= 0 || g_prof.on) return FVM_E_ARG;
    if ((int)g_prof.ids.size() < capacity) {
        const size_t have = g_prof.ev.size();
        g_prof.ev.resize(2 * (size_t)capacity);
        for (size_t i = have; i < g_prof.ev.size(); ++i)
            if (cudaEventCreate(&g_prof.ev[i]) != cudaSuccess) return fvm::launch_status();
        g_prof.ids.resize(capacity);
    }
    g_prof.cap = capacity;
    g_prof.n = 0;
    g_prof.overflow = false;
    g_prof.on = true;
    return FVM_OK;
}

extern "C" int fvm_profile_stop(void) {
    using fvm::g_prof;
    g_prof.on = false;
    return g_prof.overflow ? FVM_E_ARG : g_prof.n;
}

extern "C" int fvm_profile_read(int32_t n, int32_t* ids, float* ms) {
    using fvm::g_prof;
    if (n < 0 || n > g_prof.n || !ids || !ms) return FVM_E_ARG;
    for (int i = 0; i < n; ++i) {
        ids[i] = g_prof.ids[i];
        if (cudaEventSynchronize(g_prof.ev[2 * i + 1]) != cudaSuccess ||
            cudaEventElapsedTime(&ms[i], g_prof.ev[2 * i], g_prof.ev[2 * i + 1]) != cudaSuccess) {
            fvm::launch_status();
            return FVM_E_CUDA;
        }
    }
    return n;
}

extern "C" const char* fvm_version(void) { return "fvm_b200 1.0 sm_100a"; }

using fvm::launch_status;

// SMs of the current device (0: no device).
static int64_t ell_wave() {
    static int sms[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (!sms[dev] && cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return sms[dev];
}
// One wave of `per_sm` blocks on each of `sms` SMs over M rows, `rows` per thread.
static unsigned ell_grid(int64_t M, int rows, int64_t sms, int per_sm) {
    const int64_t all = (M + (int64_t)fvm::kBlock * rows - 1) / ((int64_t)fvm::kBlock * rows);
    return (unsigned)(all < sms * per_sm ? all : sms * per_sm);
}

extern "C" int fvm_ell_spmv(const float* vals, const int32_t* cols, int64_t M, int32_t K,
                            const float* x, int64_t incx, const float* bias, float* y, int64_t incy,
                            void* stream) {
    if (M < 0 || K < 0 || (M > 0 && (!vals && K > 0)) || (M > 0 && (!x || !y))) return FVM_E_ARG;
    if (M == 0) return FVM_OK;
    if (K > FVM_MAX_ELL_K) return FVM_E_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t wave = ell_wave();
    if (wave < 1) {
        launch_status();
        return FVM_E_CUDA;
    }
    // several rows per thread only where every SM still gets its blocks
#define FVM_SPMV_R(KT, RT) FVM_LAUNCH(fvm::KID_ELL_SPMV, s, fvm::k_ell_spmv<KT, RT><<<ell_grid(M, RT, wave, fvm::kEllBlocks), \
                                      fvm::kBlock, 0, s>>>(vals, cols, M, K, x, incx, bias, y, incy))
#define FVM_SPMV_1(KT) FVM_LAUNCH(fvm::KID_ELL_SPMV, s, fvm::k_ell_spmv_once<KT><<<(unsigned)((M + fvm::kBlock - 1) / fvm::kBlock), \
                                  fvm::kBlock, 0, s>>>(vals, cols, M, K, x, incx, bias, y, incy))
#define FVM_SPMV(KT, RT)                                                                                \
    do {                                                                                                \
        if (RT > 1 && M >= wave * fvm::kEllBlocks * fvm::kBlock * RT) FVM_SPMV_R(KT, RT);              \
        else FVM_SPMV_R(KT, 1);                                                                         \
    } while (0)
    if (K <= 2) FVM_SPMV(2, 4);
    else if (K <= 4) FVM_SPMV(4, 2);
    else if (K <= 5) FVM_SPMV(5, 1);
    else if (K <= 6) FVM_SPMV_1(6);
    else if (K <= 8) FVM_SPMV_1(8);
    else if (K <= 12) FVM_SPMV_1(12);
    else FVM_SPMV_1(16);
#undef FVM_SPMV_1
#undef FVM_SPMV_R
#undef FVM_SPMV
    return launch_status();
}

extern "C" int fvm_ell_spmm(const float* vals, const int32_t* cols, int64_t M, int32_t K,
                            const float* X, int64_t ldx, int32_t B, const float* bias, float* Y,
                            int64_t ldy, void* stream) {
    if (M < 0 || K < 0 || B < 0 || (M > 0 && B > 0 && (!X || !Y || (K > 0 && !vals))))
        return FVM_E_ARG;
    if (M == 0 || B == 0) return FVM_OK;
    const int64_t gx = (M + fvm::kBlock - 1) / fvm::kBlock;
    cudaStream_t s = (cudaStream_t)stream;
    if (K > FVM_MAX_ELL_K) return FVM_E_UNSUPPORTED;
    const int64_t wave = ell_wave();
    if (wave < 1) {
        launch_status();
        return FVM_E_CUDA;
    }
    const bool aligned = ((uintptr_t)X % 16 == 0) && ((uintptr_t)Y % 16 == 0);
    if (B == 4 && ldx == 4 && ldy == 4 && aligned) {
#define FVM_SPMM4(KT) FVM_LAUNCH(fvm::KID_ELL_SPMM, s, fvm::k_ell_spmm4<KT><<<(unsigned)gx, fvm::kBlock, 0, s>>>( \
                                     vals, cols, M, K, X, bias, Y))
        if (K <= 4) FVM_SPMM4(4);
        else if (K <= 8) FVM_SPMM4(8);
        else FVM_SPMM4(16);
#undef FVM_SPMM4
    } else if (B == 5 && K <= 5) {
#define FVM_SPMM5(KT) FVM_LAUNCH(fvm::KID_ELL_SPMM, s, fvm::k_ell_spmm5<KT><<<ell_grid(M, 1, wave, fvm::spmm5_blocks(KT)), \
                                     fvm::kBlock, 0, s>>>(vals, cols, M, K, X, ldx, bias, Y, ldy))
        if (K <= 4) FVM_SPMM5(4);
        else FVM_SPMM5(5);
#undef FVM_SPMM5
    } else {
        const unsigned gy = (unsigned)((B + 7) / 8);
#define FVM_SPMM_1(KT) FVM_LAUNCH(fvm::KID_ELL_SPMM, s, fvm::k_ell_spmm_once<KT, 8><<<dim3((unsigned)gx, gy), fvm::kBlock, 0, s>>>( \
                                      vals, cols, M, K, X, ldx, B, bias, Y, ldy))
        if (B % 8 == 0 && K > 4 && K <= 8)   // whole groups: 1.3 M rows of six slots with eight columns 112 against 129 us
            FVM_LAUNCH(fvm::KID_ELL_SPMM, s, fvm::k_ell_spmm<8, 8><<<dim3(ell_grid(M, 1, wave, fvm::kEllBlocks), gy),
                                                                    fvm::kBlock, 0, s>>>(vals, cols, M, K, X, ldx, bias, Y, ldy));
        else if (K <= 4) FVM_SPMM_1(4);
        else if (K <= 5) FVM_SPMM_1(5);
        else if (K <= 6) FVM_SPMM_1(6);
        else if (K <= 8) FVM_SPMM_1(8);
        else if (K <= 12) FVM_SPMM_1(12);
        else FVM_SPMM_1(16);
#undef FVM_SPMM_1
    }
    return launch_status();
}
