// dgemm.cu -- batched FP64 GEMM on the sm_100a FP64 tensor-core path.
//
// Two kernels by the batch's largest M: thin (M <= 16, 16 x 64 tiles) and
// ring (64 x 64 tiles fed by a cp.async ring).  Transposes are resolved at
// load time (opA, opB template flags), so A^T B, A B^T, ... need no extra
// pass.
//
// Entries flagged sym (a symmetric product added to a symmetric C) compute
// only the lower-triangle tiles and mirror each result.
//
// This is the contraction engine behind the Schur complement
// S = A - (B D^-1) B^T, the W^-1 blocks (Sinv B, B^T Sinv B), the dipole /
// overlap row sweeps and the outer-region products.
#include "common.cuh"

#include <atomic>
#include <cstdint>

namespace scatt {

namespace {

constexpr int PAD = 4;
constexpr int THREADS = 128;

__device__ __forceinline__ void dmma_16x8x8(double (&c)[4], double a0, double a1, double a2, double a3, double b0,
                                            double b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

// Thin products (every entry M <= 16: the dipole / overlap row sweeps
// G(n) = G(n-1) Rinv(n) and their W^-1 terms, K_rows x N_t x N_t).  A
// 64-row tile would spend three quarters of its DMMAs on zero rows and make
// these HBM-bound sweeps compute-bound; here a CTA computes 16 x 64 of C (16 x
// 32 where the grid is small) with four warps and streams op(B) through a
// cp.async ring of 32-deep k stages, 16-byte copies where op(B) = B allows
// them: a single matrix of order 1046 is a chain of 33 loads, 36 us with one
// stage in flight, 14 us with three.
constexpr int TBM = 16, TBK = 32;
constexpr int T_AKM = TBM + PAD;             // A as [k][m]
constexpr int T_MK = TBK + PAD;              // A as [m][k], B as [n][k]

__device__ __forceinline__ void ring_cp8(double* sdst, const double* gsrc, bool pred) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(sdst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" :: "r"(sa), "l"(gsrc), "r"(pred ? 8 : 0));
}
__device__ __forceinline__ void ring_cp16(double* sdst, const double* gsrc, bool pred) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(sdst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" :: "r"(sa), "l"(gsrc), "r"(pred ? 16 : 0));
}

template <int OPA, int OPB, int TBN>
struct ThinLayout {
    static constexpr int STAGES = TBN == 64 ? 3 : 4;
    static constexpr int BKN = TBN + PAD;    // B as [k][n]
    static constexpr int A_ELEMS = OPA == 0 ? TBK * T_AKM : TBM * T_MK;
    static constexpr int B_ELEMS = OPB == 0 ? TBN * T_MK : TBK * BKN;
    static constexpr int STAGE = A_ELEMS + B_ELEMS;
    static constexpr size_t SMEM = STAGES * (size_t)STAGE * sizeof(double);
};

template <int OPA, int OPB, int TBN>
__global__ void __launch_bounds__(THREADS)
gemm_thin_kernel(const GemmEntry* entries) {
    dep_sync();
    using L = ThinLayout<OPA, OPB, TBN>;
    constexpr int NB = TBN / 32;                // 8-column blocks of a warp
    const GemmEntry e = entries[blockIdx.z];
    const int n0 = blockIdx.y * TBN;
    if (e.M <= 0 || n0 >= e.N) return;
    const bool sym = e.sym != 0;                // M = N <= 16: one tile holds the lower triangle

    extern __shared__ double tsmem[];
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int nk = (e.K + TBK - 1) / TBK;
    const bool b16 = OPB == 0 && e.ldb % 2 == 0 && e.K % 2 == 0 && (reinterpret_cast<uintptr_t>(e.B) & 15) == 0;
    auto issue = [&](int kt, int slot) {
        if (kt < nk) {
            double* As = tsmem + slot * L::STAGE;
            double* Bs = As + L::A_ELEMS;
            const int k0 = kt * TBK;
#pragma unroll
            for (int u = 0; u < TBM * TBK / THREADS; ++u) {
                const int idx = tid + u * THREADS;
                const int m = OPA == 0 ? idx & 15 : idx >> 5, k = OPA == 0 ? idx >> 4 : idx & 31;
                const bool ok = m < e.M && k0 + k < e.K;
                const size_t at = OPA == 0 ? m + (size_t)(k0 + k) * e.lda : (k0 + k) + (size_t)m * e.lda;
                ring_cp8(As + (OPA == 0 ? k * T_AKM + m : m * T_MK + k), e.A + (ok ? at : 0), ok);
            }
            if (b16) {
#pragma unroll
                for (int u = 0; u < TBN * TBK / 2 / THREADS; ++u) {
                    const int idx = tid + u * THREADS;
                    const int n = idx >> 4, k = 2 * (idx & 15);
                    const bool ok = n0 + n < e.N && k0 + k < e.K;
                    ring_cp16(Bs + n * T_MK + k, e.B + (ok ? (k0 + k) + (size_t)(n0 + n) * e.ldb : 0), ok);
                }
            } else {
#pragma unroll
                for (int u = 0; u < TBN * TBK / THREADS; ++u) {
                    const int idx = tid + u * THREADS;
                    const int n = OPB == 0 ? idx >> 5 : idx % TBN, k = OPB == 0 ? idx & 31 : idx / TBN;
                    const bool ok = n0 + n < e.N && k0 + k < e.K;
                    const size_t at = OPB == 0 ? (k0 + k) + (size_t)(n0 + n) * e.ldb : (n0 + n) + (size_t)(k0 + k) * e.ldb;
                    ring_cp8(Bs + (OPB == 0 ? n * T_MK + k : k * L::BKN + n), e.B + (ok ? at : 0), ok);
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    double acc[NB][4];
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[j][v] = 0.0;
#pragma unroll
    for (int p = 0; p < L::STAGES - 1; ++p) issue(p, p);
    int slot = 0;
#pragma unroll 1
    for (int kt = 0; kt < nk; ++kt) {
        asm volatile("cp.async.wait_group %0;\n" :: "n"(L::STAGES - 2) : "memory");
        __syncthreads();                        // stage kt is in, and every warp is done with stage kt - 1
        issue(kt + L::STAGES - 1, slot == 0 ? L::STAGES - 1 : slot - 1);
        const double* As = tsmem + slot * L::STAGE;
        const double* Bs = As + L::A_ELEMS;
#pragma unroll
        for (int kk = 0; kk < TBK; kk += 8) {
            double a[4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = kk + t + 4 * h;
                a[2 * h] = OPA == 0 ? As[k * T_AKM + g] : As[g * T_MK + k];
                a[2 * h + 1] = OPA == 0 ? As[k * T_AKM + g + 8] : As[(g + 8) * T_MK + k];
            }
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                const int c = (warp * NB + j) * 8 + g, k = kk + t;
                const double b0 = OPB == 0 ? Bs[c * T_MK + k] : Bs[k * L::BKN + c];
                const double b1 = OPB == 0 ? Bs[c * T_MK + k + 4] : Bs[(k + 4) * L::BKN + c];
                dmma_16x8x8(acc[j], a[0], a[1], a[2], a[3], b0, b1);
            }
        }
        slot = slot == L::STAGES - 1 ? 0 : slot + 1;
    }
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int row = g + ((v >> 1) << 3);
            const int col = n0 + (warp * NB + j) * 8 + 2 * t + (v & 1);
            if (row < e.M && col < e.N && !(sym && col > row)) {
                double* c = e.C + row + (size_t)col * e.ldc;
                double r = e.alpha * acc[j][v];
                if (e.beta != 0.0) r += e.beta * *c;
                *c = r;
                if (sym && col != row) e.C[col + (size_t)row * e.ldc] = r;
            }
        }
}

// Everything else (some entry M > 16: the Schur update B D^-1 B^T, T = Sinv
// Bs, F = Bs^T T, the fit rows): 64 x 64 tiles, eight warps of 16 x 32,
// three CTAs per SM.  k streams through a three- or eight-stage cp.async
// ring of 16-deep stages with one barrier per stage.  Each operand is staged in the
// layout its global storage is contiguous in (A as [k][m] for op N, [m][k]
// for op T; B as [n][k] for op N, [k][n] for op T), so every copy is a
// contiguous run: 16-byte copies where the leading dimension, the contiguous
// extent and the base allow, 8-byte otherwise.  Row strides are 4 mod 16
// doubles, which keeps the fragment reads free of bank conflicts in every
// layout.  The 64-row tile, rather than 128, follows from the orders met
// (441 and 605 rows fill 7 and 10 of them to 0.98 and 0.95, but 4 and 5 of
// 128 to 0.86 and 0.95) and from the symmetric products, whose diagonal tiles
// waste half.
constexpr int RB = 64, RK = 16, RTHREADS = 256;
constexpr int R_KM = RB + PAD;               // [k][m] rows
constexpr int R_MK = RK + PAD;               // [m][k] rows

template <int OPA, int OPB>
struct RingLayout {
    static constexpr int A_ELEMS = OPA == 0 ? RK * R_KM : RB * R_MK;
    static constexpr int B_ELEMS = OPB == 0 ? RB * R_MK : RK * R_KM;
    static constexpr int STAGE = A_ELEMS + B_ELEMS;
};

// One operand's stage: RB rows x (of extent nx) by RK k (of extent nk), stored
// x-contiguous (XC: X[x + k ld], staged [k][x]) or k-contiguous (staged [x][k]).
template <bool XC>
__device__ __forceinline__ void ring_copy(double* sm, const double* X, int ld, int x0, int nx, int k0, int nk,
                                          bool wide, int tid) {
    if (wide) {
#pragma unroll
        for (int u = 0; u < RB * RK / 2 / RTHREADS; ++u) {
            const int idx = tid + u * RTHREADS;
            const int x = XC ? 2 * (idx & 31) : idx >> 3, k = XC ? idx >> 5 : 2 * (idx & 7);
            const bool ok = x0 + x < nx && k0 + k < nk;
            const long g = XC ? (x0 + x) + (long)(k0 + k) * ld : (k0 + k) + (long)(x0 + x) * ld;
            ring_cp16(sm + (XC ? k * R_KM + x : x * R_MK + k), X + (ok ? g : 0), ok);
        }
    } else {
#pragma unroll
        for (int u = 0; u < RB * RK / RTHREADS; ++u) {
            const int idx = tid + u * RTHREADS;
            const int x = XC ? idx & 63 : idx >> 4, k = XC ? idx >> 6 : idx & 15;
            const bool ok = x0 + x < nx && k0 + k < nk;
            const size_t g = XC ? (x0 + x) + (size_t)(k0 + k) * ld : (k0 + k) + (size_t)(x0 + x) * ld;
            ring_cp8(sm + (XC ? k * R_KM + x : x * R_MK + k), X + (ok ? g : 0), ok);
        }
    }
}

template <int OPA, int OPB, int RSTAGES>
__global__ void __launch_bounds__(RTHREADS, 3)
gemm_ring_kernel(const GemmEntry* entries) {
    dep_sync();
    using L = RingLayout<OPA, OPB>;
    const GemmEntry e = entries[blockIdx.z];
    const int m0 = blockIdx.x * RB;
    const int n0 = blockIdx.y * RB;
    if (m0 >= e.M || n0 >= e.N) return;
    const bool sym = e.sym != 0;
    if (sym && n0 > m0) return;                 // strictly upper tiles come from the mirror

    extern __shared__ double rsmem[];
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int wm = (warp & 3) * 16, wn = (warp >> 2) * 32;
    // 16-byte copies: even leading dimension, even contiguous extent, 16-byte aligned base
    const bool a16 = (e.lda % 2 == 0) && ((OPA == 0 ? e.M : e.K) % 2 == 0) &&
                     ((reinterpret_cast<uintptr_t>(e.A) & 15) == 0);
    const bool b16 = (e.ldb % 2 == 0) && ((OPB == 0 ? e.K : e.N) % 2 == 0) &&
                     ((reinterpret_cast<uintptr_t>(e.B) & 15) == 0);
    const int nk = (e.K + RK - 1) / RK;
    auto issue = [&](int kt, int slot) {
        if (kt < nk) {
            double* As = rsmem + slot * L::STAGE;
            ring_copy<OPA == 0>(As, e.A, e.lda, m0, e.M, kt * RK, e.K, a16, tid);
            ring_copy<OPB == 1>(As + L::A_ELEMS, e.B, e.ldb, n0, e.N, kt * RK, e.K, b16, tid);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };

    double acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[j][v] = 0.0;

#pragma unroll
    for (int p = 0; p < RSTAGES - 1; ++p) issue(p, p);
    int slot = 0;
#pragma unroll 1
    for (int kt = 0; kt < nk; ++kt) {
        asm volatile("cp.async.wait_group %0;\n" :: "n"(RSTAGES - 2) : "memory");
        __syncthreads();                        // stage kt is in, and every warp is done with stage kt - 1
        issue(kt + RSTAGES - 1, slot == 0 ? RSTAGES - 1 : slot - 1);
        const double* As = rsmem + slot * L::STAGE;
        const double* Bs = As + L::A_ELEMS;
#pragma unroll
        for (int kk = 0; kk < RK; kk += 8) {
            double a[4];
            const int r = wm + g;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = kk + t + 4 * h;
                a[2 * h] = OPA == 0 ? As[k * R_KM + r] : As[r * R_MK + k];
                a[2 * h + 1] = OPA == 0 ? As[k * R_KM + r + 8] : As[(r + 8) * R_MK + k];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c = wn + j * 8 + g;
                const double b0 = OPB == 0 ? Bs[c * R_MK + kk + t] : Bs[(kk + t) * R_KM + c];
                const double b1 = OPB == 0 ? Bs[c * R_MK + kk + t + 4] : Bs[(kk + t + 4) * R_KM + c];
                dmma_16x8x8(acc[j], a[0], a[1], a[2], a[3], b0, b1);
            }
        }
        slot = slot == RSTAGES - 1 ? 0 : slot + 1;
    }

    // C = alpha * acc + beta * C
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int row = m0 + wm + g + ((v >> 1) << 3);
            const int col = n0 + wn + j * 8 + 2 * t + (v & 1);
            if (row < e.M && col < e.N && !(sym && col > row)) {
                double* c = e.C + row + (size_t)col * e.ldc;
                double r = e.alpha * acc[j][v];
                if (e.beta != 0.0) r += e.beta * *c;
                *c = r;
                if (sym && col != row) e.C[col + (size_t)row * e.ldc] = r;
            }
        }
}

template <class Kernel>
int launch_stages(Kernel kernel, std::atomic<unsigned long long>& done, dim3 grid, int threads, size_t smem,
                  const GemmEntry* entries_dev, cudaStream_t stream) {
    int dev = 0;
    SCATT_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !(done.load() & (1ull << dev))) {
        SCATT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (dev >= 0 && dev < 64) done.fetch_or(1ull << dev);
    }
    return SCATT_CUDA_TRY_RET(launch_dep(kernel, grid, dim3(threads), smem, stream, entries_dev));
}

template <int OPA, int OPB>
int launch_ring(const GemmEntry* entries_dev, int count, int maxM, int maxN, cudaStream_t stream) {
    constexpr size_t stage = RingLayout<OPA, OPB>::STAGE * sizeof(double);
    static_assert(3 * stage <= 75 * 1024, "three CTAs per SM");
    static std::atomic<unsigned long long> done3{0}, done8{0};
    const dim3 grid((maxM + RB - 1) / RB, (maxN + RB - 1) / RB, count);
    // A grid that leaves each SM one CTA is a chain of loads: eight stages in
    // flight instead of three (which let three CTAs share an SM).
    if ((long)grid.x * grid.y * count <= 148)
        return launch_stages(gemm_ring_kernel<OPA, OPB, 8>, done8, grid, RTHREADS, 8 * stage, entries_dev, stream);
    return launch_stages(gemm_ring_kernel<OPA, OPB, 3>, done3, grid, RTHREADS, 3 * stage, entries_dev, stream);
}

template <int OPA, int OPB>
int launch_thin(const GemmEntry* entries_dev, int count, int maxN, cudaStream_t stream) {
    static std::atomic<unsigned long long> done32{0}, done64{0};
    // 32 columns a CTA spread a grid of at most two waves over more SMs; past that they only read A twice as often
    if ((long)((maxN + 63) / 64) * count <= 296)
        return launch_stages(gemm_thin_kernel<OPA, OPB, 32>, done32, dim3(1, (maxN + 31) / 32, count), THREADS,
                             ThinLayout<OPA, OPB, 32>::SMEM, entries_dev, stream);
    return launch_stages(gemm_thin_kernel<OPA, OPB, 64>, done64, dim3(1, (maxN + 63) / 64, count), THREADS,
                         ThinLayout<OPA, OPB, 64>::SMEM, entries_dev, stream);
}

}  // namespace

int gemm_batched(const GemmEntry* entries_dev, int count, int maxM, int maxN,
                 int opA, int opB, cudaStream_t stream) {
    if (count <= 0 || maxM <= 0 || maxN <= 0) return SCATT_OK;
    if (count > 65535) {
        set_last_error("gemm_batched: batch count exceeds 65535");
        return SCATT_ERR_ARG;
    }
    if (maxM <= TBM) {
        if (opA == 0 && opB == 0)      SCATT_TRY((launch_thin<0, 0>(entries_dev, count, maxN, stream)));
        else if (opA == 1 && opB == 0) SCATT_TRY((launch_thin<1, 0>(entries_dev, count, maxN, stream)));
        else if (opA == 0 && opB == 1) SCATT_TRY((launch_thin<0, 1>(entries_dev, count, maxN, stream)));
        else                           SCATT_TRY((launch_thin<1, 1>(entries_dev, count, maxN, stream)));
        SCATT_COUNT_LAUNCH(1);
        return SCATT_OK;
    }
    if (opA == 0 && opB == 0)      SCATT_TRY((launch_ring<0, 0>(entries_dev, count, maxM, maxN, stream)));
    else if (opA == 1 && opB == 0) SCATT_TRY((launch_ring<1, 0>(entries_dev, count, maxM, maxN, stream)));
    else if (opA == 0 && opB == 1) SCATT_TRY((launch_ring<0, 1>(entries_dev, count, maxM, maxN, stream)));
    else                           SCATT_TRY((launch_ring<1, 1>(entries_dev, count, maxM, maxN, stream)));
    SCATT_COUNT_LAUNCH(1);
    return SCATT_OK;
}

}  // namespace scatt
