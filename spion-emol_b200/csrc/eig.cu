// eig.cu -- eigenvalues of symmetric matrices on the device.
//
// Used for (a) the Johnson stability shift of SchurInverter
// (SchurInverter.cpp:44-59: smallest eigenvalue when the Gershgorin bound is
// inconclusive; the reference calls Eigen's SelfAdjointEigenSolver on the
// lower triangle) and (b) the eigenphases atan(eig K) of
// KMatrixExtractor.cpp:185-191 / AsymptoticAmplitudes.cpp:340-344.
//
// Method: Householder reduction to tridiagonal form (one cluster of CTAs per
// matrix, reading only the lower triangle, in place in global memory), then
// Sturm-sequence bisection for the requested eigenvalues.  Both steps are
// backward stable, so eigenvalues are accurate to O(eps ||M||), the same
// guarantee the reference's QR-based solver gives.
#include <cmath>

#include "common.cuh"
#include "eig.cuh"

namespace scatt {

namespace {

constexpr int ET = 256;

// Sum over the CTA, the same value (and bits) in every thread.
__device__ double block_sum(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < ET / 32; ++i) s += red[i];
    return s;
}

// One matrix on a cluster of EC CTAs, in place in global memory (it stays in
// L2).  Columns are dealt to the cluster's warps; every CTA forms the
// Householder vector of each step itself.  A step's rank-2 update is applied
// in the next step's pass over the matrix, which also forms that step's
// product A v, so that the trailing matrix is passed once and the cluster
// meets once per step (to exchange p = beta A v, double-buffered in the work
// array); the one column that the others read next is not written in that
// pass.  Bound by the chain of n steps, each a few L2 latencies: order 441,
// 99.3 ms with one CTA per matrix, two passes and a matrix-vector product of
// one row per thread.
constexpr int EC = 8;

__global__ void __cluster_dims__(EC, 1, 1) __launch_bounds__(ET)
tridiag_kernel(const EigEntry* entries) {
    const EigEntry en = entries[blockIdx.x / EC];
    const int n = en.n, ld = en.ld;
    double* M = en.M;
    double *d = en.d, *e = en.e;
    extern __shared__ double esm[];
    double* v = esm;              // Householder vector of the last step, rows below it
    double* w = esm + n;          // its partner in the pending update A -= v w^T + w v^T
    double* x = esm + 2 * n;      // vector of this step
    __shared__ double red[ET / 32];
    const int tid = threadIdx.x, lane = tid & 31;
    const int rank = blockIdx.x % EC, gw = rank * (ET / 32) + (tid >> 5);
    constexpr int GW = EC * ET / 32;
    auto meet = [] {
        asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    };
    // only the lower triangle is read: mirror it into the upper triangle first
    for (int j = gw; j < n; j += GW)
        for (int i = j + 1 + lane; i < n; i += 32) M[j + (size_t)i * ld] = M[i + (size_t)j * ld];
    for (int i = tid; i < n; i += ET) v[i] = w[i] = 0.0;
    meet();
    for (int k = 0; k + 2 < n; ++k) {
        // column k with the pending update: x below the diagonal
        const double vk = v[k], wk = w[k];
        double ss = 0.0;
        for (int i = k + 1 + tid; i < n; i += ET) {
            const double c = __ldcg(&M[i + (size_t)k * ld]) - (v[i] * wk + w[i] * vk);
            x[i] = c;
            ss += c * c;
        }
        const double nrm2 = block_sum(ss, red);
        const double x0 = x[k + 1];
        double alpha = x0 > 0.0 ? -sqrt(nrm2) : sqrt(nrm2), beta = 0.0;    // beta = 2 / (v^T v)
        if (nrm2 > 0.0) {
            const double vtv = nrm2 - x0 * x0 + (x0 - alpha) * (x0 - alpha);
            beta = vtv > 0.0 ? 2.0 / vtv : 0.0;
        } else {
            alpha = 0.0;
        }
        if (rank == 0 && tid == 0) {
            d[k] = __ldcg(&M[k + (size_t)k * ld]) - 2.0 * vk * wk;
            e[k] = alpha;
        }
        __syncthreads();                           // every thread has read x[k + 1]
        if (tid == 0) x[k + 1] = x0 - alpha;
        __syncthreads();
        // pending update and p = beta A x on this warp's columns
        double* p = en.work + (size_t)(k & 1) * n;
        for (int j = k + 1 + gw; j < n; j += GW) {
            double* col = M + (size_t)j * ld;
            const double vj = v[j], wj = w[j];
            double s = 0.0;
            for (int i = k + 1 + lane; i < n; i += 32) {
                const double c = col[i] - (v[i] * wj + w[i] * vj);
                col[i] = c;
                s += c * x[i];
            }
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (lane == 0) p[j] = beta * s;
        }
        meet();
        // w = p - (beta / 2) (p^T x) x; x becomes v
        double pv = 0.0;
        for (int i = k + 1 + tid; i < n; i += ET) {
            const double c = __ldcg(&p[i]);
            w[i] = c;
            pv += c * x[i];
        }
        const double K = 0.5 * beta * block_sum(pv, red);
        for (int i = k + 1 + tid; i < n; i += ET) {
            w[i] = beta == 0.0 ? 0.0 : w[i] - K * x[i];
            v[i] = x[i];
        }
        __syncthreads();
    }
    if (rank == 0 && tid == 0) {
        auto at = [&](int i, int j) { return __ldcg(&M[i + (size_t)j * ld]) - (v[i] * w[j] + w[i] * v[j]); };
        if (n >= 2) {
            d[n - 2] = at(n - 2, n - 2);
            e[n - 2] = at(n - 1, n - 2);
        }
        d[n - 1] = at(n - 1, n - 1);
    }
    meet();                                        // no CTA leaves while another may still read its columns
}

// Sturm count: number of eigenvalues of the tridiagonal (d, e^2) below x.
__device__ int sturm_count(const double* d, const double* e2, int n, double x) {
    int cnt = 0;
    double q = d[0] - x;
    if (q < 0.0) ++cnt;
    for (int i = 1; i < n; ++i) {
        if (q == 0.0) q = 1e-300;
        q = (d[i] - x) - e2[i - 1] / q;
        if (q < 0.0) ++cnt;
    }
    return cnt;
}

__device__ double bisect_kth(const double* d, const double* e2, int n, int kth, double lo, double hi) {
    // smallest x with count(x) > kth
    for (int it = 0; it < 200; ++it) {
        const double mid = 0.5 * (lo + hi);
        if (mid <= lo || mid >= hi) break;
        if (sturm_count(d, e2, n, mid) > kth) hi = mid; else lo = mid;
    }
    return 0.5 * (lo + hi);
}

// eigenvalues by bisection: one thread per requested eigenvalue index, the
// tridiagonal matrix in shared memory (each count is a chain of n divisions;
// 13.2 ms at order 441 with its elements read from global memory)
constexpr int BT = 32;

__global__ void __launch_bounds__(BT)
bisect_kernel(const EigEntry* entries, int nwant) {
    extern __shared__ double esm[];
    const EigEntry en = entries[blockIdx.y];
    const int n = en.n;
    const int want = nwant > 0 ? min(nwant, n) : n;
    if ((int)(blockIdx.x * BT) >= want) return;
    double *d = esm, *e2 = esm + n;
    double lo = INFINITY, hi = -INFINITY;
    for (int i = threadIdx.x; i < n; i += BT) {
        const double di = en.d[i], ei = i + 1 < n ? en.e[i] : 0.0;
        const double r = (i > 0 ? fabs(en.e[i - 1]) : 0.0) + fabs(ei);
        d[i] = di;
        e2[i] = ei * ei;
        lo = fmin(lo, di - r);
        hi = fmax(hi, di + r);
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    __syncwarp();
    const int kth = blockIdx.x * BT + threadIdx.x;
    if (kth >= want) return;
    const double pad = 1e-12 * fmax(fabs(lo), fabs(hi)) + 1e-300;
    en.out[kth] = bisect_kth(d, e2, n, kth, lo - pad, hi + pad);
}

}  // namespace

int sym_eigvals_batched(const EigEntry* entries_dev, int count, int nmax, int nwant,
                        cudaStream_t stream) {
    if (count <= 0 || nmax <= 0) return SCATT_OK;
    // orders of S(n) and K, whose inverses end at 8192
    constexpr size_t order_max = 8533;
    static_assert(3 * order_max * sizeof(double) <= 200 * 1024, "one CTA's shared memory");
    if ((size_t)nmax > order_max) {
        set_last_error("sym_eigvals_batched: order above 8533");
        return SCATT_ERR_SIZE;
    }
    static std::atomic<unsigned long long> tridiag_done{0}, bisect_done{0};
    SCATT_TRY(allow_smem(tridiag_kernel, 3 * order_max * sizeof(double), tridiag_done));
    SCATT_TRY(allow_smem(bisect_kernel, 2 * order_max * sizeof(double), bisect_done));
    const size_t ts = 3 * (size_t)nmax * sizeof(double), bs = 2 * (size_t)nmax * sizeof(double);
    tridiag_kernel<<<count * EC, ET, ts, stream>>>(entries_dev);
    const int want = nwant > 0 ? nwant : nmax;
    bisect_kernel<<<dim3((want + BT - 1) / BT, count), BT, bs, stream>>>(entries_dev, nwant);
    SCATT_CUDA_TRY(cudaGetLastError());
    SCATT_COUNT_LAUNCH(2);
    return SCATT_OK;
}

}  // namespace scatt
