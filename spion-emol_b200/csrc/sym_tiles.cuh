// sym_tiles.cuh -- tile layout and device pieces of the symmetric batched
// inverse (sym_inverse.cu): a symmetric matrix of order n is held as the
// lower triangle of its T x T grid of 64 x 64 tiles (T = ceil(n / 64), the
// rows past n padded by the identity), tile (i, j) at index i (i + 1) / 2 + j.
//
// Inside a tile the elements lie as 8 x 8 sub-blocks of 64 contiguous,
// row-major doubles, sub-block (R, C) at 8 R + C.  A warp's 16-byte accesses
// of one sub-block (lane 4 g + t: row g, columns 2 t and 2 t + 1) are then
// 512 contiguous bytes and are the f64 mma fragments as they stand: the
// accumulator pair (g, 2 t .. 2 t + 1), and, as the summation index may be
// taken in any order that both operands share, the operand pair too.
#pragma once

#include <cstddef>

#include "common.cuh"

namespace scatt {

constexpr int SYM_NB = 64;                   // tile order
constexpr int SYM_TILE = SYM_NB * SYM_NB;    // doubles of a tile
constexpr int SYM_THREADS = 256;
constexpr int SYM_ORDER_MAX = 8192;          // the general inverse's limit too

// One matrix of a batched symmetric inverse (a device array of these).
struct SymEntry {
    double* A;              // n x n, ld n (both triangles): rebuilt or kept for the rescue, then its scratch
    double* W;              // T (T + 1) / 2 tiles
    double *P, *M;          // T tiles each: the pivot column block and its negated product with D
    double* D;              // the inverse of the pivot tile, the pivot tile itself, and sym_skew of the two
    double* out;            // n x n, ld ldo: the inverse, both triangles
    unsigned* stat;         // sym_stat_words(n) words, zero before the sweep: [0] how it was finished, [1 ..] SYM_STEPS Newton
                            // steps' changes, [4] the largest element of A off the
                            // diagonal tiles (high word), SYM_STAT_HEAD on sym_stat
    int* status;            // DeviceStatus, first failing column; zero before the sweep
    int n, ldo;
    double skew_max;        // SYM_SKEW_MAX, or infinity: no rows refined
};

__host__ __device__ inline int sym_tiles_of(int n) { return (n + SYM_NB - 1) / SYM_NB; }
__host__ __device__ inline size_t sym_tile_index(int i, int j) { return (size_t)i * (i + 1) / 2 + j; }
// Doubles that W needs for order n, and those of P, M and D together (D: two tiles and a word).
inline size_t sym_work_doubles(int n) {
    const size_t T = sym_tiles_of(n);
    return T * (T + 1) / 2 * SYM_TILE;
}
inline size_t sym_panel_doubles(int n) { return (2 * (size_t)sym_tiles_of(n) + 2) * SYM_TILE + 32; }
// Doubles of the rescue's scratch, one for all entries of a batch (it takes one at a time).
inline size_t sym_scratch_doubles(int n) { return 2 * (size_t)n * n; }

__device__ __forceinline__ int sym_pos(int r, int c) {
    return (((r >> 3) << 3) + (c >> 3)) * 64 + ((r & 7) << 3) + (c & 7);
}

// Reciprocal by two Newton-Raphson steps from the hardware's approximation, 20
// bits of it: 2^-40 after the first, and after the second the rounding of its
// last operation alone (half an ulp, as a division's).  Outside sym_rcp_range
// the approximation flushes x or its reciprocal to zero, and x is scaled first.
// A division, of every pivot or of those alone, made the chain longer by 80
// cycles a pivot (R^-1 of order 1046 alone 0.591 -> 0.638 and 0.633 ms).
__device__ __forceinline__ double sym_rcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    y = fma(y, fma(-x, y, 1.0), y);
    return fma(y, fma(-x, y, 1.0), y);
}

// High word of |x| of a normal number below 2^1022.
__device__ __forceinline__ bool sym_rcp_range(unsigned hi) { return hi - 0x00100000u < 0x7fd00000u - 0x00100000u; }

constexpr int SYM_PANEL_LD = 10;   // doubles of a panel row: 16-byte rows apart by 5 mod 8, no bank conflicts

__device__ __forceinline__ int sym_low_pos(int r, int c) {      // in SymDiagShared::low
    return ((r >> 3) * ((r >> 3) + 1) / 2 + (c >> 3)) * 64 + ((r & 7) << 3) + (c & 7);
}
__device__ __forceinline__ unsigned sym_hi(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }

// What a sweep records of tile row i, as the high words of magnitudes (in
// order as integers, a NaN above every number): the largest element of A's
// tile row, of that row in any Schur complement, of the pivot tile's inverse
// D_i, and of the inverse's tile row.
enum SymStat { SYM_OF_A = 0, SYM_OF_SCHUR = 1, SYM_OF_D = 2, SYM_OF_X = 3 };
constexpr int SYM_STEPS = 3, SYM_STAT_OFF = 4, SYM_STAT_HEAD = 8;
__host__ __device__ inline size_t sym_stat_words(int n) { return SYM_STAT_HEAD + 4 * (size_t)sym_tiles_of(n); }
__device__ __forceinline__ unsigned* sym_stat(const SymEntry& e, int i, SymStat q) { return e.stat + SYM_STAT_HEAD + 4 * i + q; }
// A warp's part of an element block of tile (i, j): it counts for both tile rows.
__device__ __forceinline__ void sym_track(const SymEntry& e, unsigned m, int i, int j, SymStat q) {
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(sym_stat(e, i, q), m);
        if (i != j) atomicMax(sym_stat(e, j, q), m);
    }
}

struct SymDiagShared {
    double X[SYM_TILE];                          // the tile in (lower triangle), its inverse out
    double panel[2][SYM_PANEL_LD * SYM_NB];      // a factored panel: 64 rows by 8 columns, by parity
    double row[8];                               // pivot row of the panel
    unsigned long long used;                     // rows taken as pivots
    unsigned long long took[2];                  // those of the last panel, by parity
    int prow[SYM_NB];                            // row of each step's pivot
    int krow[SYM_NB];                            // step at which each row was the pivot
    alignas(16) double low[36 * 64];             // the tile's sub-blocks (R, C), R >= C, at R (R + 1) / 2 + C
};

static_assert(offsetof(SymDiagShared, panel) % 16 == 0 && offsetof(SymDiagShared, row) % 16 == 0 &&
              offsetof(SymDiagShared, low) % 16 == 0, "read and written in 16-byte pieces");

// Pivot tiles whose largest column sum of |A_ij D_ij| (A the tile, D its
// inverse; sym_skew holds the largest of each warp's columns) is above this
// have their rows L = P D refined (sym_panel_kernel).  The sum is 1 for a
// diagonal or a well-conditioned dominant tile, does not change when rows and
// columns are scaled alike (a tile graded by its centrifugal terms has a
// condition number of 1e3 and a sum below 1.4), and grows with the rounding
// that D brings into L P^T.  Up to 4, sweeps without the refinement stayed
// within 1.5 of the general inverse's error over the matrices of radial sweeps
// (orders 162 and 196, 20 and 50 bohr); above, they did not always.  At 1.4
// bohr no tile is above it; at 20 bohr and order 1046 one in 50.
constexpr double SYM_SKEW_MAX = 3.0;
__device__ __forceinline__ double* sym_tile_of_D(const SymEntry& e) { return e.D + SYM_TILE; }
__device__ __forceinline__ double* sym_skew(const SymEntry& e) { return e.D + 2 * SYM_TILE; }

__device__ __forceinline__ void sym_dmma(double (&c)[4], const double2& alo, const double2& ahi, const double2& b);

// x = keep ? x : 0, by a predicated move.
__device__ __forceinline__ void sym_zero_unless(double& x, int keep) {
    asm("{\n .reg .pred p;\n setp.eq.s32 p, %1, 0;\n @p mov.f64 %0, 0d0000000000000000;\n}\n" : "+d"(x) : "r"(keep));
}

// The eight pivots of column block c by one warp, two rows per lane.  The
// diagonal's row is published before it is known to be the pivot, so that its
// reciprocal and the largest candidate are found side by side.
__device__ __forceinline__ void sym_diag_panel(SymDiagShared& sh, int c, int lane) {
    double a0[8], a1[8];                         // rows lane and lane + 32
    double* blk0 = sh.X + ((lane >> 3) * 8 + c) * 64 + (lane & 7) * 8;
    double* blk1 = blk0 + 4 * 8 * 64;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const double2 x = reinterpret_cast<const double2*>(blk0)[m], y = reinterpret_cast<const double2*>(blk1)[m];
        a0[2 * m] = x.x;
        a0[2 * m + 1] = x.y;
        a1[2 * m] = y.x;
        a1[2 * m + 1] = y.y;
    }
    unsigned long long used = sh.used;
    const unsigned long long before = used;
    unsigned long long took = 0;                 // the panel's pivot rows, a byte each
    bool u0 = (used >> lane) & 1ull, u1 = (used >> (lane + 32)) & 1ull;
    double2* row = reinterpret_cast<double2*>(sh.row);
    double x[8];
    // row p to every lane, through shared memory (16 shuffles a pivot instead: 43,400 cycles a tile for 40,100)
    auto publish = [&](int p) {
        if (lane == (p & 31)) {
            if (p < 32) {
#pragma unroll
                for (int m = 0; m < 4; ++m) row[m] = make_double2(a0[2 * m], a0[2 * m + 1]);
            } else {
#pragma unroll
                for (int m = 0; m < 4; ++m) row[m] = make_double2(a1[2 * m], a1[2 * m + 1]);
            }
        }
        __syncwarp();
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const double2 v = row[m];
            x[2 * m] = v.x;
            x[2 * m + 1] = v.y;
        }
        __syncwarp();
    };
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int d = 8 * c + k;                 // the diagonal's row
        publish(d);
        double rp = sym_rcp(x[k]);
        // candidate keys: magnitude (the low 6 bits of the high word give way to the row)
        const unsigned h0 = (unsigned)__double2hiint(a0[k]) & 0x7fffffc0u, h1 = (unsigned)__double2hiint(a1[k]) & 0x7fffffc0u;
        const unsigned c0 = u0 ? 0u : (0x80000000u | h0 | (unsigned)(63 - lane));
        const unsigned c1 = u1 ? 0u : (0x80000000u | h1 | (unsigned)(31 - lane));
        const unsigned best = __reduce_max_sync(0xffffffffu, c0 > c1 ? c0 : c1);
        const unsigned hd = (unsigned)__double2hiint(x[k]) & 0x7fffffffu;
        int p = d;
        if (((used >> d) & 1ull) || hd < (best & 0x7fffffc0u) || !sym_rcp_range(hd)) {
            p = 63 - (int)(best & 63u);
            publish(p);
            const unsigned hp = (unsigned)__double2hiint(x[k]) & 0x7fffffffu;
            const double scale = sym_rcp_range(hp) ? 1.0 : hp < 0x00100000u ? 0x1p600 : 0x1p-600;
            rp = sym_rcp(scale * x[k]) * scale;
        }
        used |= 1ull << p;
        const bool here = lane == (p & 31);
        double g0 = -(a0[k] * rp), g1 = -(a1[k] * rp);
        // the pivot row becomes 0 + rp x
        const int keep = here ? 0 : 1;
        if (p < 32) {
            u0 |= here;
            g0 = here ? rp : g0;
#pragma unroll
            for (int m = 0; m < 8; ++m) sym_zero_unless(a0[m], keep);
        } else {
            u1 |= here;
            g1 = here ? rp : g1;
#pragma unroll
            for (int m = 0; m < 8; ++m) sym_zero_unless(a1[m], keep);
        }
        took |= (unsigned long long)p << (8 * k);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            if (m == k) continue;
            a0[m] = fma(g0, x[m], a0[m]);
            a1[m] = fma(g1, x[m], a1[m]);
        }
        a0[k] = g0;
        a1[k] = g1;
    }
    double* pan = sh.panel[c & 1];
    double2 *p0 = reinterpret_cast<double2*>(pan + lane * SYM_PANEL_LD);
    double2 *p1 = reinterpret_cast<double2*>(pan + (lane + 32) * SYM_PANEL_LD);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const double2 v = make_double2(a0[2 * m], a0[2 * m + 1]), w = make_double2(a1[2 * m], a1[2 * m + 1]);
        p0[m] = v;
        p1[m] = w;
        reinterpret_cast<double2*>(blk0)[m] = v;
        reinterpret_cast<double2*>(blk1)[m] = w;
    }
    if (lane < 8) {
        const int p = (int)((took >> (8 * lane)) & 0xffull);
        sh.prow[8 * c + lane] = p;
        sh.krow[p] = 8 * c + lane;
    }
    if (lane == 0) {
        sh.used = used;
        sh.took[c & 1] = used & ~before;
    }
}

// Inverse of the 64 x 64 symmetric tile in sh.X (lower triangle read), by
// Gauss-Jordan elimination with pivoting inside the tile, one CTA of 256
// threads.  Warp w owns the 64 x 8 column block w.  At panel c warp c alone
// takes the block's eight pivots and publishes the block; then warp c + 1
// applies it to its own block by DMMAs and goes on to the next panel, and the
// other warps apply it meanwhile.  Rows are not moved: row p_k of step k ends
// as row k of the inverse, whose column p_j sits in column j.  The result is
// symmetrised and left in sh.X.
//
// Bound by the chain of 64 pivots, each of which stays inside a warp.  A form
// with the rows spread over the CTA, and one or two barriers a pivot, took
// 55,000 cycles, this one 40,100 (20 us; 48,000 where every pivot is off the
// diagonal).  Pivoting is partial, inside the tile: without it (pivots in
// order) the growth of the intermediate inverses reaches 1e3 to 1e4 and the
// solver's results lose one to four digits; with it the growth seen is mostly
// below 2.
__device__ __forceinline__ void sym_diag_invert(SymDiagShared& sh) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    // a lane's element (r, c) of the warp's u-th 8 x 4 patch, and its mirror image: at most four-way conflicts
    auto patch = [&](int u, int& r, int& c) {
        const int q = u * 8 + warp;              // 128 patches
        r = (q >> 4) * 8 + g;
        c = (q & 15) * 4 + t;
    };
#pragma unroll 4
    for (int u = 0; u < 16; ++u) {
        int r, c;
        patch(u, r, c);
        if (c > r) sh.X[sym_pos(r, c)] = sh.X[sym_pos(c, r)];
    }
    if (tid == 0) sh.used = 0;
    __syncthreads();
    // block <- (block with the panel's pivot rows zeroed) + panel * (pivot rows of the block)
    auto apply = [&](int c) {
        const double* pan = sh.panel[c & 1];
        const int p0 = sh.prow[8 * c + 2 * t], p1 = sh.prow[8 * c + 2 * t + 1];
        const unsigned long long took = sh.took[c & 1];
        const double2 b = make_double2(sh.X[sym_pos(p0, 8 * warp + g)], sh.X[sym_pos(p1, 8 * warp + g)]);
        double acc[4][4];
        double2 alo[4], ahi[4];
        double2* xb = reinterpret_cast<double2*>(sh.X + warp * 64 + 2 * lane);
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
            const int r0 = mt * 16 + g, r1 = r0 + 8;
            const double2 v = xb[(2 * mt) * 256], w = xb[(2 * mt + 1) * 256];
            const bool z0 = (took >> r0) & 1ull, z1 = (took >> r1) & 1ull;
            acc[mt][0] = z0 ? 0.0 : v.x;
            acc[mt][1] = z0 ? 0.0 : v.y;
            acc[mt][2] = z1 ? 0.0 : w.x;
            acc[mt][3] = z1 ? 0.0 : w.y;
            alo[mt] = *reinterpret_cast<const double2*>(pan + r0 * SYM_PANEL_LD + 2 * t);
            ahi[mt] = *reinterpret_cast<const double2*>(pan + r1 * SYM_PANEL_LD + 2 * t);
        }
        __syncwarp();
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) sym_dmma(acc[mt], alo[mt], ahi[mt], b);
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
            xb[(2 * mt) * 256] = make_double2(acc[mt][0], acc[mt][1]);
            xb[(2 * mt + 1) * 256] = make_double2(acc[mt][2], acc[mt][3]);
        }
        __syncwarp();
    };
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {
        if (warp == c) sym_diag_panel(sh, c, lane);
        __syncthreads();
        // the next panel's warp first, alone with the shared memory's bandwidth; the others beside its pivots
        if (warp == c + 1) apply(c);
        __syncthreads();
        if (warp != c && warp != c + 1) apply(c);
    }
    __syncthreads();
    // inverse(r, c) = X(p_r, step of c), symmetrised
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        int r, c;
        patch(u, r, c);
        v[u] = 0.5 * (sh.X[sym_pos(sh.prow[r], sh.krow[c])] + sh.X[sym_pos(sh.prow[c], sh.krow[r])]);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        int r, c;
        patch(u, r, c);
        sh.X[sym_pos(r, c)] = v[u];
    }
    __syncthreads();
}

__device__ __forceinline__ void sym_dmma(double (&c)[4], const double2& alo, const double2& ahi, const double2& b) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(alo.x), "d"(ahi.x), "d"(alo.y), "d"(ahi.y), "d"(b.x), "d"(b.y));
}

// acc (16 x 32 of a 64 x 64 product, warp (wr, wc)) += A B^T over sub-block
// columns [k0, k1) of the shared tiles As, Bs.
__device__ __forceinline__ void sym_tile_mma(double (&acc)[4][4], const double* As, const double* Bs, int wr, int wc,
                                         int lane, int k0, int k1) {
#pragma unroll
    for (int kc = k0; kc < k1; ++kc) {
        const double2 alo = *reinterpret_cast<const double2*>(As + ((2 * wr) * 8 + kc) * 64 + 2 * lane);
        const double2 ahi = *reinterpret_cast<const double2*>(As + ((2 * wr + 1) * 8 + kc) * 64 + 2 * lane);
#pragma unroll
        for (int nb = 0; nb < 4; ++nb) {
            const double2 b = *reinterpret_cast<const double2*>(Bs + ((4 * wc + nb) * 8 + kc) * 64 + 2 * lane);
            sym_dmma(acc[nb], alo, ahi, b);
        }
    }
}

// Writes the inverse of pivot tile K (in sh.X) to D and, negated, to the
// matrix, tracks its largest element inside the order, and writes sym_skew from
// the tile in sh.low.
__device__ __forceinline__ void sym_diag_store(const SymEntry& e, int K, const SymDiagShared& sh) {
    double2* D = reinterpret_cast<double2*>(e.D);
    double2* W = reinterpret_cast<double2*>(e.W + sym_tile_index(K, K) * SYM_TILE);
    const double2* X = reinterpret_cast<const double2*>(sh.X);
    unsigned m = 0;
    double s0 = 0.0, s1 = 0.0;               // of the lane's two columns
    const int lane = threadIdx.x & 31, C = threadIdx.x >> 5;
#pragma unroll
    for (int R = 0; R < 8; ++R) {
        const int u = threadIdx.x + R * SYM_THREADS;
        const double2 v = X[u];
        const double* low = sh.low + (R >= C ? R * (R + 1) / 2 + C : C * (C + 1) / 2 + R) * 64;
        const int g = lane >> 2, t = lane & 3;
        s0 += fabs(v.x * low[R >= C ? 2 * lane : 16 * t + g]);
        s1 += fabs(v.y * low[R >= C ? 2 * lane + 1 : 16 * t + 8 + g]);
        D[u] = v;
        W[u] = make_double2(-v.x, -v.y);
        // pair u: sub-block u / 32, row (u % 32) / 4
        const int row = K * SYM_NB + (u >> 8) * 8 + ((u & 31) >> 2);
        const int col = K * SYM_NB + ((u >> 5) & 7) * 8 + (u & 3) * 2;
        if (row < e.n && col < e.n) m = max(m, sym_hi(v.x));
        if (row < e.n && col + 1 < e.n) m = max(m, sym_hi(v.y));
    }
    sym_track(e, m, K, K, SYM_OF_D);
#pragma unroll
    for (int o = 16; o >= 4; o >>= 1) {
        s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    }
    s0 = fmax(s0, s1);
#pragma unroll
    for (int o = 2; o >= 1; o >>= 1) s0 = fmax(s0, __shfl_xor_sync(0xffffffffu, s0, o));
    if (lane == 0) sym_skew(e)[C] = s0;
}

// Packs tile t of entry e from elem(row, column, inside) (the element of a
// symmetric matrix, consecutive columns on consecutive lanes; anything where
// !inside, without reading) and, for tile 0, inverts the first pivot tile.
// elem reads under predicates, not branches, so that a thread's 16 elements
// are in flight together; one after another they made this pass four times
// slower than its traffic.
template <class Elem>
__device__ __forceinline__ void sym_pack_tile(const SymEntry& e, int t, SymDiagShared& sh, Elem elem) {
    int i = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((size_t)(i + 1) * (i + 2) / 2 <= (size_t)t) ++i;
    while ((size_t)i * (i + 1) / 2 > (size_t)t) --i;
    const int j = t - i * (i + 1) / 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool first = t == 0;
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const int gi = i * SYM_NB + warp * 8 + (u >> 1), gj = j * SYM_NB + lane + 32 * (u & 1);
        v[u] = elem(gi, gj, gi < e.n && gj < e.n);
    }
    unsigned m = 0;
    double* W = first ? sh.X : e.W + (size_t)t * SYM_TILE;
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const int r = warp * 8 + (u >> 1), c = lane + 32 * (u & 1);
        const int gi = i * SYM_NB + r, gj = j * SYM_NB + c;
        const bool in = gi < e.n && gj < e.n;
        if (in) m = max(m, sym_hi(v[u]));
        const double x = in ? v[u] : gi == gj ? 1.0 : 0.0;
        W[sym_pos(r, c)] = x;
        if (first) {
            sym_tile_of_D(e)[sym_pos(r, c)] = x;
            if (r >> 3 >= c >> 3) sh.low[sym_low_pos(r, c)] = x;
        }
    }
    sym_track(e, m, i, j, SYM_OF_A);
    if (i != j) {
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) atomicMax(e.stat + SYM_STAT_OFF, m);
    }
    if (first) {
        __syncthreads();
        sym_diag_invert(sh);
        sym_diag_store(e, 0, sh);
    }
}

// Entry and tile of CTA bid among count entries of nt tiles: the first tiles,
// whose pivots are inverted, of all entries come first.
__device__ __forceinline__ void sym_pack_index(int bid, int count, int nt, int& ent, int& t) {
    if (bid < count) {
        ent = bid;
        t = 0;
    } else {
        ent = (bid - count) / (nt - 1);
        t = 1 + (bid - count) - ent * (nt - 1);
    }
}

// Sweeps a packed batch (pivot tile 0 already inverted) to the inverses, all
// entries of order <= nmax; entries of order 0 are skipped.
int sym_sweep_batched(const SymEntry* entries_dev, int count, int nmax, cudaStream_t stream);
// Packs full symmetric matrices (entry.A) for sym_sweep_batched; stat and status must be zero.
int sym_pack_batched(const SymEntry* entries_dev, int count, int nmax, cudaStream_t stream);

}  // namespace scatt
