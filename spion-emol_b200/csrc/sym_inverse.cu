// sym_inverse.cu -- batched inverse of symmetric matrices by a blocked
// symmetric sweep on 64 x 64 tiles.
//
// The Schur complements S(n) and the matrices R(n) of the R-ratio recurrence
// are symmetric, so their inverses need n^3 flops, half of a Gauss-Jordan
// elimination's, and only the lower triangle's traffic.  Pivot tile by pivot
// tile (K = 0 .. T - 1), with D = A_KK^-1 and P_i = A_iK:
//     A_ij -= P_i D P_j^T (i, j != K),   A_iK = P_i D,   A_KK = -D,
// which after the last K leaves -A^-1.  Two kernels per K:
//   panel   one CTA per tile row: P_i (copied, transposed above K) and
//           -P_i D by DMMA, and the pivot column's new tiles;
//   update  one CTA per tile of the triangle: 64 x 64 x 64 DMMAs onto the
//           accumulator loaded from the tile, operands by cp.async in four
//           k stages, three CTAs per SM.  The CTA of the next pivot tile goes
//           first and inverts it after its update (sym_diag_invert), so the
//           serial pivot chain (about 20 us a tile) hides behind the other tiles.
// The last K writes the inverse itself, both triangles.
// Bound by the DMMA pipe where the batch fills the chip, by the chain of pivot
// tiles where it does not.  R^-1 of order 1046, B200, against the pivoted
// Gauss-Jordan elimination: 128 matrices 18.9 -> 6.8 ms, 1 matrix 2.60 -> 0.75 ms.
// Tiles of 64: a 128-wide pivot would halve the triangle's traffic (which the
// DMMAs still cover) and double the panel's flops and the serial chain.
//
// There is no column of pivots down the whole matrix: pivoting is partial
// inside a pivot tile only.  What a leading block much closer to singular
// than the matrix does to the result, and how it is mended, is in
// sym_rescue.cuh.
#include "sym_rescue.cuh"

namespace scatt {

namespace {

__device__ __forceinline__ void cp16(double* sdst, const double* gsrc) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(sdst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" :: "r"(sa), "l"(gsrc));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" :: "n"(N) : "memory"); }

// -acc into out (both triangles): tile rows from r0, columns from c0.
__device__ __forceinline__ void store_out(const SymEntry& e, const double (&acc)[4][4], int r0, int c0, int wr, int wc,
                                          int lane) {
    unsigned m = 0;
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int nb = 0; nb < 4; ++nb)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int r = r0 + wr * 16 + g + ((v >> 1) << 3), c = c0 + wc * 32 + nb * 8 + 2 * t + (v & 1);
            if (r >= e.n || c >= e.n || (r0 == c0 && c > r)) continue;
            const double x = -acc[nb][v];
            e.out[r + (size_t)c * e.ldo] = x;
            if (r != c) e.out[c + (size_t)r * e.ldo] = x;
            m = max(m, sym_hi(x));
        }
    sym_track(e, m, r0 / SYM_NB, c0 / SYM_NB, SYM_OF_X);
}

__global__ void __launch_bounds__(SYM_THREADS, 3)
sym_pack_kernel(const SymEntry* entries, int count, int nt) {
    dep_sync();
    extern __shared__ double smem[];
    int ent, t;
    sym_pack_index(blockIdx.x, count, nt, ent, t);
    const SymEntry e = entries[ent];
    const int T = sym_tiles_of(e.n);
    if (t >= T * (T + 1) / 2) return;
    sym_pack_tile(e, t, *reinterpret_cast<SymDiagShared*>(smem), [&e](int gi, int gj, bool in) {
        return in ? e.A[gj + (size_t)gi * e.n] : 0.0;
    });
}

// acc (16 x 16 of a 32 x 64 product, warp (wr, wc)) += A B^T over the shared half tile As and tile Bs.
__device__ __forceinline__ void sym_half_mma(double (&acc)[2][4], const double* As, const double* Bs, int wr, int wc,
                                             int lane) {
#pragma unroll
    for (int kc = 0; kc < 8; ++kc) {
        const double2 alo = *reinterpret_cast<const double2*>(As + ((2 * wr) * 8 + kc) * 64 + 2 * lane);
        const double2 ahi = *reinterpret_cast<const double2*>(As + ((2 * wr + 1) * 8 + kc) * 64 + 2 * lane);
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
            const double2 b = *reinterpret_cast<const double2*>(Bs + ((2 * wc + nb) * 8 + kc) * 64 + 2 * lane);
            sym_dmma(acc[nb], alo, ahi, b);
        }
    }
}

constexpr int PANEL_ROWS = 32;
constexpr size_t PANEL_SMEM = (SYM_TILE + PANEL_ROWS * SYM_NB) * sizeof(double);

// Grid (half tile rows, entries): 32 rows of the pivot column a CTA.  Whole
// tiles leave a small batch fewer CTAs with a longer chain each, and at 28
// matrices of order 1046 run as a full wave and a sliver (22 us a launch).
//
// L = P D takes over D's error, kappa(A_KK) eps, and the update L P^T multiplies
// it by P again, where the Schur complement may cancel to a small part of
// P D P^T: a matrix with one dominant direction (c / n v v^T beside a part of
// norm 1, c = 1e5, order 196) lost four digits, 1.6e-9 against the pivoted
// elimination's 5.5e-13.  Where the tile's skew tells of it, one step by the
// tile itself, L += (P - L A_KK) D, leaves the row residual at rounding
// whatever kappa: 8.6e-13.  Only there: two products more of 64 x 64 a CTA.
// Telling costs the inverse 1 % (order 1046: 28 matrices 1.765 -> 1.781 ms, one
// 0.597 -> 0.605), most of it the sums of |A_KK o D| at the end of each pivot
// tile's chain.
__global__ void __launch_bounds__(SYM_THREADS, 3)
sym_panel_kernel(const SymEntry* entries, int K) {
    dep_sync();
    extern __shared__ double smem[];
    const SymEntry e = entries[blockIdx.y];
    const int T = sym_tiles_of(e.n), i = blockIdx.x >> 1, half = blockIdx.x & 1;
    if (i >= T || K >= T) return;
    const bool last = K == T - 1;
    double* Ds = smem;
    double* Ps = smem + SYM_TILE;                // 32 x 64: sub-block rows 4 half .. 4 half + 3 of the tile
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wr = warp & 1, wc = warp >> 1;     // 16 rows, 16 columns
    if (i == K) {
        if (!last || half) return;
        unsigned m = 0;
        for (int u = tid; u < SYM_TILE; u += SYM_THREADS) {
            const int r = u & 63, c = u >> 6;
            const int gr = K * SYM_NB + r, gc = K * SYM_NB + c;
            if (gr >= e.n || gc >= e.n) continue;
            const double x = e.D[r >= c ? sym_pos(r, c) : sym_pos(c, r)];
            e.out[gr + (size_t)gc * e.ldo] = x;
            m = max(m, sym_hi(x));
        }
        sym_track(e, m, K, K, SYM_OF_X);
        return;
    }
    constexpr int HALF = PANEL_ROWS * SYM_NB;    // doubles
    double* Wt = e.W + (i > K ? sym_tile_index(i, K) : sym_tile_index(K, i)) * SYM_TILE;
    if (i > K) {
        for (int u = tid; u < HALF / 2; u += SYM_THREADS) cp16(Ps + 2 * u, Wt + half * HALF + 2 * u);
    } else {
        // rows of the transpose: sub-block columns 4 half .. of tile (K, i)
#pragma unroll
        for (int q = 0; q < HALF / 2 / SYM_THREADS; ++q) {
            const int u = tid + q * SYM_THREADS;                 // sub-block u / 32 of the 8 x 4 read
            const int sr = u >> 7, sc = (u >> 5) & 3, row = (u & 31) >> 2, col = (u & 3) * 2;
            const double2 v = *reinterpret_cast<const double2*>(Wt + (sr * 8 + 4 * half + sc) * 64 + row * 8 + col);
            double* d = Ps + (sc * 8 + sr) * 64 + row;
            d[col * 8] = v.x;
            d[col * 8 + 8] = v.y;
        }
    }
    for (int u = tid; u < SYM_TILE / 2; u += SYM_THREADS) cp16(Ds + 2 * u, e.D + 2 * u);
    cp_commit();
    // read by one warp of the CTA: read by all, 272 warps at order 1046 queue for one line (0.5 us)
    const bool skewed = tid < SYM_THREADS / 32 && sym_skew(e)[tid] > e.skew_max;
    cp_wait<0>();
    const bool refine = __syncthreads_or(skewed);
    double acc[2][4];
#pragma unroll
    for (int nb = 0; nb < 2; ++nb)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[nb][v] = 0.0;
    sym_half_mma(acc, Ps, Ds, wr, wc, lane);
    double* Pg = e.P + (size_t)i * SYM_TILE + half * HALF;
    double* Mg = e.M + (size_t)i * SYM_TILE + half * HALF;
    for (int u = tid; u < HALF / 2; u += SYM_THREADS)
        reinterpret_cast<double2*>(Pg)[u] = reinterpret_cast<const double2*>(Ps)[u];
    if (refine) {
        double res[2][4];                        // P - L A_KK
        const double2 *A2 = reinterpret_cast<const double2*>(sym_tile_of_D(e)), *D2 = reinterpret_cast<const double2*>(e.D);
        __syncthreads();                         // Ps and Ds are read by every warp above
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double2* p = reinterpret_cast<double2*>(Ps + ((2 * wr + h) * 8 + 2 * wc + nb) * 64 + 2 * lane);
                res[nb][2 * h] = p->x;
                res[nb][2 * h + 1] = p->y;
                *p = make_double2(-acc[nb][2 * h], -acc[nb][2 * h + 1]);
            }
        for (int u = tid; u < SYM_TILE / 2; u += SYM_THREADS) reinterpret_cast<double2*>(Ds)[u] = A2[u];
        __syncthreads();
        sym_half_mma(res, Ps, Ds, wr, wc, lane);
        __syncthreads();
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<double2*>(Ps + ((2 * wr + h) * 8 + 2 * wc + nb) * 64 + 2 * lane) =
                    make_double2(res[nb][2 * h], res[nb][2 * h + 1]);
        for (int u = tid; u < SYM_TILE / 2; u += SYM_THREADS) reinterpret_cast<double2*>(Ds)[u] = D2[u];
        __syncthreads();
        sym_half_mma(acc, Ps, Ds, wr, wc, lane);
    }
    if (last) {
        // the inverse's tile (i, K) is -L_i
        unsigned m = 0;
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int r = i * SYM_NB + half * PANEL_ROWS + wr * 16 + g + ((v >> 1) << 3);
                const int c = K * SYM_NB + wc * 16 + nb * 8 + 2 * t + (v & 1);
                if (r >= e.n || c >= e.n) continue;
                const double x = -acc[nb][v];
                e.out[r + (size_t)c * e.ldo] = x;
                e.out[c + (size_t)r * e.ldo] = x;
                m = max(m, sym_hi(x));
            }
        sym_track(e, m, i, K, SYM_OF_X);
    }
#pragma unroll
    for (int nb = 0; nb < 2; ++nb)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int off = ((2 * wr + h) * 8 + 2 * wc + nb) * 64 + 2 * lane;
            *reinterpret_cast<double2*>(Mg + off) = make_double2(-acc[nb][2 * h], -acc[nb][2 * h + 1]);
            if (i > K)
                *reinterpret_cast<double2*>(Wt + half * HALF + off) = make_double2(acc[nb][2 * h], acc[nb][2 * h + 1]);
        }
    if (i < K) {
        __syncthreads();                         // Ps is read by every warp above
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                // element (row, col) of L_i goes to (col, row) of tile (K, i): sub-block (col / 8, row / 8) of 8 x 4
                double* d = Ps + ((2 * wc + nb) * 4 + 2 * wr + (v >> 1)) * 64;
                d[(2 * t + (v & 1)) * 8 + g] = acc[nb][v];
            }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < HALF / 2 / SYM_THREADS; ++q) {
            const int u = tid + q * SYM_THREADS;
            *reinterpret_cast<double2*>(Wt + ((u >> 7) * 8 + 4 * half + ((u >> 5) & 3)) * 64 + (u & 31) * 2) =
                reinterpret_cast<const double2*>(Ps)[u];
        }
    }
}

// Tile pair of index u among the lower triangle without row and column K.
__device__ __forceinline__ void tile_of(int u, int K, int& i, int& j) {
    int a = (int)((sqrtf(8.0f * (float)u + 1.0f) - 1.0f) * 0.5f);
    while ((a + 1) * (a + 2) / 2 <= u) ++a;
    while (a * (a + 1) / 2 > u) --a;
    const int b = u - a * (a + 1) / 2;
    i = a + (a >= K ? 1 : 0);
    j = b + (b >= K ? 1 : 0);
}

constexpr size_t UPDATE_SMEM = 2 * SYM_TILE * sizeof(double);
static_assert(sizeof(SymDiagShared) <= UPDATE_SMEM, "the pivot tile's inversion reuses the operands' shared memory");

// One CTA per tile; `nu` tiles of the largest entry.  With ud >= 0 the first
// `count` CTAs take each entry's next pivot tile (index ud).
__global__ void __launch_bounds__(SYM_THREADS, 3)
sym_update_kernel(const SymEntry* entries, int count, int K, int nu, int ud) {
    dep_sync();
    extern __shared__ double smem[];
    const int bid = blockIdx.x;
    int ent, u;
    if (ud < 0) {
        ent = bid / nu;
        u = bid - ent * nu;
    } else if (bid < count) {
        ent = bid;
        u = ud;
    } else {
        ent = (bid - count) / (nu - 1);
        u = (bid - count) - ent * (nu - 1);
        if (u >= ud) ++u;
    }
    int i, j;
    tile_of(u, K, i, j);
    const SymEntry e = entries[ent];
    const int T = sym_tiles_of(e.n);
    if (i >= T || K >= T) return;
    const bool last = K == T - 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wr = warp & 3, wc = warp >> 2;
    double* Ms = smem;
    double* Ps = smem + SYM_TILE;
    const double* Mg = e.M + (size_t)i * SYM_TILE;
    const double* Pg = e.P + (size_t)j * SYM_TILE;
    // four k stages of two sub-block columns: 8 runs of 128 doubles per operand
#pragma unroll
    for (int st = 0; st < 4; ++st) {
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const int x = tid + w * SYM_THREADS;           // 512 16-byte pieces
            const int off = (x >> 6) * 512 + st * 128 + (x & 63) * 2;
            cp16(Ms + off, Mg + off);
            cp16(Ps + off, Pg + off);
        }
        cp_commit();
    }
    double* Wt = e.W + sym_tile_index(i, j) * SYM_TILE;
    double acc[4][4];
#pragma unroll
    for (int nb = 0; nb < 4; ++nb)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const double2 v = *reinterpret_cast<const double2*>(Wt + ((2 * wr + h) * 8 + 4 * wc + nb) * 64 + 2 * lane);
            acc[nb][2 * h] = v.x;
            acc[nb][2 * h + 1] = v.y;
        }
    cp_wait<3>();
    __syncthreads();
    sym_tile_mma(acc, Ms, Ps, wr, wc, lane, 0, 2);
    cp_wait<2>();
    __syncthreads();
    sym_tile_mma(acc, Ms, Ps, wr, wc, lane, 2, 4);
    cp_wait<1>();
    __syncthreads();
    sym_tile_mma(acc, Ms, Ps, wr, wc, lane, 4, 6);
    cp_wait<0>();
    __syncthreads();
    sym_tile_mma(acc, Ms, Ps, wr, wc, lane, 6, 8);
    if (last) {
        store_out(e, acc, i * SYM_NB, j * SYM_NB, wr, wc, lane);
        return;
    }
    if (j > K) {                                 // a tile of the Schur complement: its growth
        const int lim = i == T - 1 ? e.n - i * SYM_NB - wr * 16 - (lane >> 2) : SYM_NB;   // rows inside the order
        unsigned m = 0;
#pragma unroll
        for (int nb = 0; nb < 4; ++nb)
#pragma unroll
            for (int v = 0; v < 4; ++v)
                if ((v >> 1) * 8 < lim) m = max(m, sym_hi(acc[nb][v]));
        sym_track(e, m, i, j, SYM_OF_SCHUR);
    }
    if (i == K + 1 && j == K + 1) {
        SymDiagShared& sh = *reinterpret_cast<SymDiagShared*>(smem);
        __syncthreads();                         // every warp has read its operands
#pragma unroll
        for (int nb = 0; nb < 4; ++nb)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int R = 2 * wr + h, S = 4 * wc + nb;
                const double2 x = make_double2(acc[nb][2 * h], acc[nb][2 * h + 1]);
                *reinterpret_cast<double2*>(sh.X + (R * 8 + S) * 64 + 2 * lane) = x;
                *reinterpret_cast<double2*>(sym_tile_of_D(e) + (R * 8 + S) * 64 + 2 * lane) = x;
                if (R >= S) *reinterpret_cast<double2*>(sh.low + (R * (R + 1) / 2 + S) * 64 + 2 * lane) = x;
            }
        __syncthreads();
        sym_diag_invert(sh);
        sym_diag_store(e, K + 1, sh);
        return;
    }
#pragma unroll
    for (int nb = 0; nb < 4; ++nb)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            *reinterpret_cast<double2*>(Wt + ((2 * wr + h) * 8 + 4 * wc + nb) * 64 + 2 * lane) =
                make_double2(acc[nb][2 * h], acc[nb][2 * h + 1]);
}

}  // namespace

int sym_pack_batched(const SymEntry* entries_dev, int count, int nmax, cudaStream_t stream) {
    if (count <= 0 || nmax <= 0) return SCATT_OK;
    const int T = sym_tiles_of(nmax);
    const int nt = T * (T + 1) / 2;
    static std::atomic<unsigned long long> done{0};
    SCATT_TRY(allow_smem(sym_pack_kernel, sizeof(SymDiagShared), done));
    SCATT_CUDA_TRY(launch_dep(sym_pack_kernel, count * nt, SYM_THREADS, sizeof(SymDiagShared), stream, entries_dev, count, nt));
    SCATT_COUNT_LAUNCH(1);
    return SCATT_OK;
}

int sym_sweep_batched(const SymEntry* entries_dev, int count, int nmax, cudaStream_t stream) {
    if (count <= 0 || nmax <= 0) return SCATT_OK;
    if (count > 65535) {
        set_last_error("sym_sweep_batched: batch count exceeds 65535");
        return SCATT_ERR_ARG;
    }
    if (nmax > SYM_ORDER_MAX) {
        set_last_error("sym_sweep_batched: order " + std::to_string(nmax) + " exceeds " + std::to_string(SYM_ORDER_MAX));
        return SCATT_ERR_SIZE;
    }
    static std::atomic<unsigned long long> panel_done{0}, update_done{0};
    SCATT_TRY(allow_smem(sym_panel_kernel, PANEL_SMEM, panel_done));
    SCATT_TRY(allow_smem(sym_update_kernel, UPDATE_SMEM, update_done));
    const int T = sym_tiles_of(nmax), nu = T * (T - 1) / 2;
    for (int K = 0; K < T; ++K) {
        SCATT_CUDA_TRY(launch_dep(sym_panel_kernel, dim3(2 * T, count), SYM_THREADS, PANEL_SMEM, stream, entries_dev, K));
        SCATT_COUNT_LAUNCH(1);
        if (nu > 0) {
            const int ud = K + 1 < T ? K * (K + 1) / 2 + K : -1;
            SCATT_CUDA_TRY(launch_dep(sym_update_kernel, count * nu, SYM_THREADS, UPDATE_SMEM, stream, entries_dev, count, K, nu, ud));
            SCATT_COUNT_LAUNCH(1);
        }
    }
    return SCATT_OK;
}

namespace {
// The caller's matrices are still in entry.A.
struct KeptSource {
    __device__ void operator()(int, const SymEntry&, int, int) const {}
};
}  // namespace

int sym_rescue_batched(const SymEntry* entries_dev, int count, unsigned* barrier, double* scratch, cudaStream_t stream) {
    return sym_rescue_launch(entries_dev, count, barrier, scratch, KeptSource{}, stream);
}

}  // namespace scatt
