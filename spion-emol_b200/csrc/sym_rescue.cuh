// sym_rescue.cuh -- what follows a symmetric sweep whose intermediate
// inverses grew (see sym_inverse.cu): one launch per batch, which returns at
// once when no entry needs it.
//
// A sweep's error grows with g, the larger of max|D_i| / max|A^-1| and of the
// Schur complements' largest element over A's, each within a tile row i (over
// the whole matrix, a large element of another block would hide the growth of
// this one: blocks of delta I and I / delta beside one with a pivot tile of
// delta = 1e-4 give 1, and an error of 1.5e-12 in that block), the largest of
// the rows'.  The inverse takes a Newton step
// X <- X (2 I - A X), two products over the whole grid for that entry alone,
// which squares the relative error, where g > 3 (rare in a radial sweep, and
// rarer the finer the grid), and a second one above g = 1e3.  Not elsewhere: the step leaves rounding of
// kappa eps, which a sweep of a graded matrix (large diagonal elements near
// the origin) stays ten times below.  A step too where max|D| times A's
// largest element off the diagonal tiles is above 2e4: one dominant direction
// that every tile has a part of.  (By sym_skew above 1e3 instead, the dipoles of
// a sweep at l_cont 11, N_t 386, came out ten times worse, 8.4e-10 off the
// oracle's.)
// Measured on the matrices of one sweep (order 1046, kappa = max|A| max|X|),
// relative errors:
//              g       kappa   sweep    Newton   LU       Gauss-Jordan, pivoted
//              1200    21      3.9e-11  7.7e-16  8.4e-16  1.1e-14
//              0.94    2.1e6   3.1e-9   8.2e-13  1.9e-12  2.7e-13
//              15      1.4e3   7.7e-13  7.0e-15  3.9e-13  7.4e-13
//   median     1       20      7e-16             6e-16
// The steps' changes tell whether they converge: a step more is taken while
// one is above 1e-6, three at most.  Where they grow instead (condition numbers
// past 1e9 beside a growth of 1e5), past g = 1e6, and on zero and non-finite
// pivots, to report them, the entry takes a pivoted elimination by one CTA:
// slow, and not met in normal running.
#pragma once

#include "sym_tiles.cuh"

namespace scatt {

// Barrier over the grid's CTAs, all resident (cooperative launch): `turn`
// counts the barriers passed on this counter, which starts at zero.  The wait
// is bounded (about 10 s); false: it ran out.
__device__ __forceinline__ bool sym_grid_barrier(unsigned* counter, unsigned& turn) {
    __shared__ int s_ok;
    __syncthreads();
    ++turn;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(counter, 1u);
        const unsigned want = turn * gridDim.x;
        int ok = 0;
        for (unsigned spin = 0; spin < (1u << 26); ++spin) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
            if (v >= want) { ok = 1; break; }
            __nanosleep(100);
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Tile (i, j) of alpha A^T B, all of order n and column-major (A^T read by
// columns of A); the 64 x 64 result in the accumulator layout of sym_tile_mma.
__device__ __forceinline__ void sym_product_tile(double (&acc)[4][4], const double* A, int lda, const double* B,
                                                 int ldb, int n, int i, int j, double* smem) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *As = smem, *Bs = smem + SYM_TILE;
#pragma unroll
    for (int nb = 0; nb < 4; ++nb)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[nb][v] = 0.0;
    for (int kb = 0; kb < n; kb += SYM_NB) {
        __syncthreads();
#pragma unroll 4
        for (int u = 0; u < 16; ++u) {
            const int x = warp * 8 + (u >> 1), k = lane + 32 * (u & 1), gk = kb + k;
            const int ra = i * SYM_NB + x, rb = j * SYM_NB + x;
            As[sym_pos(x, k)] = (ra < n && gk < n) ? A[gk + (size_t)ra * lda] : 0.0;
            Bs[sym_pos(x, k)] = (rb < n && gk < n) ? B[gk + (size_t)rb * ldb] : 0.0;
        }
        __syncthreads();
        sym_tile_mma(acc, As, Bs, warp & 3, warp >> 2, lane, 0, 8);
    }
}

struct SymPivotShared {
    unsigned long long best[32];
    int row[32];
    int p, stop;
};

// Gauss-Jordan elimination with partial pivoting of e.A by one CTA (rows stay
// in place, as in sym_diag_invert; the pivot row and column go through e.W)
// into e.out, symmetrised; e.status gets the first zero or non-finite pivot.
__device__ __forceinline__ void sym_pivoted(const SymEntry& e, SymPivotShared& sh) {
    const int n = e.n, tid = threadIdx.x;
    double* A = e.A;
    double* row = e.W;                // n doubles
    double* col = e.W + n;            // n doubles
    double* X = e.out;
    // step of each row's pivot (-1: unused) and row of each step
    double* step_of_row = reinterpret_cast<double*>(e.M);
    double* row_of_step = reinterpret_cast<double*>(e.P);
    for (int r = tid; r < n; r += blockDim.x) step_of_row[r] = -1.0;
    if (tid == 0) sh.stop = 0;
    __syncthreads();
    for (int k = 0; k < n; ++k) {
        unsigned long long b = 0;
        int br = n;
        for (int r = tid; r < n; r += blockDim.x) {
            const double v = A[r + (size_t)k * n];
            col[r] = v;
            if (step_of_row[r] < 0.0) {
                const unsigned long long key = (unsigned long long)__double_as_longlong(fabs(v));
                if (br == n || key > b) { b = key; br = r; }
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long ob = __shfl_xor_sync(0xffffffffu, b, o);
            const int orow = __shfl_xor_sync(0xffffffffu, br, o);
            if (orow < n && (br == n || ob > b || (ob == b && orow < br))) { b = ob; br = orow; }
        }
        if ((tid & 31) == 0) { sh.best[tid >> 5] = b; sh.row[tid >> 5] = br; }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
                if (sh.row[w] < n && (br == n || sh.best[w] > b || (sh.best[w] == b && sh.row[w] < br))) {
                    b = sh.best[w];
                    br = sh.row[w];
                }
            sh.p = br;
            const double v = __longlong_as_double((long long)b);
            if (!isfinite(v) || v == 0.0) {
                e.status[0] = isfinite(v) ? DEV_SINGULAR : DEV_NONFINITE;
                e.status[1] = k;
                sh.stop = 1;
            }
            step_of_row[br] = k;
            row_of_step[k] = br;
        }
        __syncthreads();
        if (sh.stop) break;
        const int p = sh.p;
        for (int c = tid; c < n; c += blockDim.x) row[c] = A[p + (size_t)c * n];
        __syncthreads();
        const double rp = 1.0 / col[p];
        for (long u = tid; u < (long)n * n; u += blockDim.x) {
            const int r = (int)(u % n), c = (int)(u / n);
            double v;
            if (r == p) v = c == k ? rp : row[c] * rp;
            else v = c == k ? -col[r] * rp : A[u] - (col[r] * rp) * row[c];
            A[u] = v;
        }
        __syncthreads();
    }
    if (sh.stop) {
        const double bad = __longlong_as_double(0x7ff8000000000000ll);
        for (long u = tid; u < (long)n * n; u += blockDim.x) X[(u % n) + (size_t)(u / n) * e.ldo] = bad;
        return;
    }
    // A[p_k][j] = inv[k][p_j]
    for (long u = tid; u < (long)n * n; u += blockDim.x) {
        const int r = (int)(u % n), c = (int)(u / n);
        X[(int)step_of_row[r] + (size_t)(int)row_of_step[c] * e.ldo] = A[u];
    }
    __syncthreads();
    for (long u = tid; u < (long)n * n; u += blockDim.x) {
        const int r = (int)(u % n), c = (int)(u / n);
        if (c >= r) continue;
        const double v = 0.5 * (X[r + (size_t)c * e.ldo] + X[c + (size_t)r * e.ldo]);
        X[r + (size_t)c * e.ldo] = v;
        X[c + (size_t)r * e.ldo] = v;
    }
}

constexpr int SYM_RESCUE_LIST = 256;          // entries looked at in one pass

// `source` fills rows and columns of entry.A from what the caller still has
// (index, entry, first element, stride); entry.A may also have been kept.
// The status words come in cleared and are only ever set here, each entry's by
// one CTA: passes over the list are not ordered between the CTAs.
template <class Source>
__global__ void __launch_bounds__(SYM_THREADS, 1)
sym_rescue_kernel(const SymEntry* entries, int count, unsigned* barrier, double* scratch, Source source) {
    extern __shared__ double smem[];
    __shared__ int s_mode[SYM_RESCUE_LIST];
    __shared__ SymPivotShared s_piv;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wr = warp & 3, wc = warp >> 2, g = lane >> 2, t = lane & 3;
    unsigned turn = 0;
    bool alive = true;
    for (int base = 0; base < count; base += SYM_RESCUE_LIST) {
        const int m = min(SYM_RESCUE_LIST, count - base);
        int any = 0;
        // four lanes an entry, every load of a lane in flight together: this stands in each step's chain
        for (int k = tid >> 2; k < ((m + 7) & ~7); k += SYM_THREADS / 4) {
            const int n = k < m ? entries[base + k].n : 0;
            unsigned* stat = entries[base + min(k, m - 1)].stat;
            double gr = 0.0, dm = 0.0;
            bool bad = false;
#pragma unroll 5
            for (int i = tid & 3; i < sym_tiles_of(n); i += 4) {
                const uint4 w = reinterpret_cast<const uint4*>(stat + SYM_STAT_HEAD)[i];
                const double a = __hiloint2double((int)w.x, 0), s = __hiloint2double((int)w.y, 0);
                const double d = __hiloint2double((int)w.z, 0), x = __hiloint2double((int)w.w, 0);
                gr = fmax(gr, fmax(d / x, s / a));
                dm = fmax(dm, d);
                bad |= !isfinite(a) || !isfinite(s) || !isfinite(d) || !isfinite(x) || !(a > 0.0) || !(x > 0.0);
            }
            for (int o = 1; o <= 2; o <<= 1) {
                gr = fmax(gr, __shfl_xor_sync(0xffffffffu, gr, o));
                dm = fmax(dm, __shfl_xor_sync(0xffffffffu, dm, o));
            }
            const double off = n > SYM_NB ? __hiloint2double((int)stat[SYM_STAT_OFF], 0) : 0.0;
            const unsigned quad = __ballot_sync(0xffffffffu, bad) >> (lane & ~3) & 15u;
            // one tile is pivoted throughout
            const int mode = n == 0 ? 0 : quad || !(gr <= 1e6) ? 3 : n <= SYM_NB ? 0 : gr > 1e3 ? 2 : gr > 3.0 || off * dm > 2e4 ? 1 : 0;
            if (k < m && (tid & 3) == 0) {
                s_mode[k] = mode;
                if (n > 0 && blockIdx.x == 0) stat[0] = (unsigned)mode;
            }
            any |= mode;
        }
        if (!__syncthreads_or(any)) continue;
        // Newton steps, entry by entry over the whole grid
        for (int k = 0; k < m && alive; ++k) {
            const int mode = s_mode[k];
            if (mode != 1 && mode != 2) continue;
            const SymEntry e = entries[base + k];
            const int n = e.n, T = sym_tiles_of(n);
            source(base + k, e, blockIdx.x * SYM_THREADS + tid, gridDim.x * SYM_THREADS);
            alive = sym_grid_barrier(barrier, turn);
            double last = INFINITY;                 // change of the step before
            for (int step = 0; alive; ++step) {
                for (int half = 0; half < 2 && alive; ++half) {
                    // scratch = A X, then its second half = X scratch (A and X are symmetric)
                    for (int u = blockIdx.x; u < T * T; u += gridDim.x) {
                        const int i = u % T, j = u / T;
                        double acc[4][4];
                        if (half == 0) sym_product_tile(acc, e.A, n, e.out, e.ldo, n, i, j, smem);
                        else sym_product_tile(acc, e.out, e.ldo, scratch, n, n, i, j, smem);
                        double* C = half == 0 ? scratch : scratch + (size_t)n * n;
#pragma unroll
                        for (int nb = 0; nb < 4; ++nb)
#pragma unroll
                            for (int v = 0; v < 4; ++v) {
                                const int r = i * SYM_NB + wr * 16 + g + ((v >> 1) << 3);
                                const int c = j * SYM_NB + wc * 32 + nb * 8 + 2 * t + (v & 1);
                                if (r < n && c < n) C[r + (size_t)c * n] = acc[nb][v];
                            }
                    }
                    alive = sym_grid_barrier(barrier, turn);
                }
                if (!alive) break;
                const double* Z = scratch + (size_t)n * n;
                double ch = 0.0;                    // largest change over the smaller of its two tile rows' maxima
                for (long u = blockIdx.x * (long)SYM_THREADS + tid; u < (long)n * n; u += (long)gridDim.x * SYM_THREADS) {
                    const int r = (int)(u % n), c = (int)(u / n);
                    if (c > r) continue;
                    const double z = 0.5 * (Z[r + (size_t)c * n] + Z[c + (size_t)r * n]);
                    const double x0 = e.out[r + (size_t)c * e.ldo], x = 2.0 * x0 - z;
                    e.out[r + (size_t)c * e.ldo] = x;
                    e.out[c + (size_t)r * e.ldo] = x;
                    const unsigned row = min(*sym_stat(e, r / SYM_NB, SYM_OF_X), *sym_stat(e, c / SYM_NB, SYM_OF_X));
                    const double q = fabs(x - x0) / __hiloint2double((int)row, 0);
                    ch = q <= ch ? ch : q;          // a NaN stays
                }
                const unsigned hi = __reduce_max_sync(0xffffffffu, sym_hi(ch));
                if (lane == 0) atomicMax(e.stat + 1 + step, hi);
                alive = sym_grid_barrier(barrier, turn);
                ch = __hiloint2double((int)__ldcg(e.stat + 1 + step), 0);
                // not contracting: the elimination below (every CTA decides the same)
                if (!(ch <= 0.1) || (ch > 1e-6 && (ch > last || step + 1 == SYM_STEPS))) {
                    __syncthreads();                // s_mode[k] has been read
                    if (tid == 0) s_mode[k] = 3;
                    if (blockIdx.x == 0 && tid == 0) e.stat[0] = 3;
                    break;
                }
                if (step + 1 >= mode && ch <= 1e-6) break;
                last = ch;
            }
            if (!alive && blockIdx.x == 0 && tid == 0) e.status[0] = DEV_NONFINITE;
        }
        __syncthreads();
        // pivoted eliminations, one CTA each
        for (int k = 0; k < m; ++k) {
            if (s_mode[k] != 3 || (base + k) % (int)gridDim.x != (int)blockIdx.x) continue;
            const SymEntry e = entries[base + k];
            source(base + k, e, tid, SYM_THREADS);
            __syncthreads();
            sym_pivoted(e, s_piv);
            __syncthreads();
        }
        __syncthreads();                        // s_mode is rewritten
    }
}

template <class Source>
int sym_rescue_launch(const SymEntry* entries_dev, int count, unsigned* barrier, double* scratch, Source source,
                      cudaStream_t stream) {
    if (count <= 0) return SCATT_OK;
    int dev = 0, sms = 0;
    SCATT_CUDA_TRY(cudaGetDevice(&dev));
    static std::atomic<int> grid_of[64];
    const size_t smem = 2 * SYM_TILE * sizeof(double);
    sms = dev >= 0 && dev < 64 ? grid_of[dev].load() : 0;
    if (sms == 0) {
        SCATT_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        SCATT_CUDA_TRY(cudaFuncSetAttribute(sym_rescue_kernel<Source>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)smem));
        if (dev >= 0 && dev < 64) grid_of[dev].store(sms);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sms);
    cfg.blockDim = dim3(SYM_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    SCATT_CUDA_TRY(cudaLaunchKernelEx(&cfg, sym_rescue_kernel<Source>, entries_dev, count, barrier, scratch, source));
    SCATT_COUNT_LAUNCH(1);
    return SCATT_OK;
}

// For callers whose entry.A is intact; barrier: one zeroed word; scratch: sym_scratch_doubles of the largest order.
int sym_rescue_batched(const SymEntry* entries_dev, int count, unsigned* barrier, double* scratch, cudaStream_t stream);

}  // namespace scatt
