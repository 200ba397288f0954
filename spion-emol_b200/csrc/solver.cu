// solver.cu -- the per-energy scattering path, batched over energies and
// resident in HBM.  Host orchestration + per-step kernels.
//
// One radial step n (all energies of the batch, lock-step):
//   k_build_V / k_build_B  V(n) from V_sigma by the Gaunt pair list, the
//                          exchange block B(n) = h^2/12 Q(n) from chi(n) by the
//                          G_combined CSR, Bs = B D^-1, D^-1 (shared by energies)
//   k_init_S               A = (1 + h^2 E/6) I - h^2/6 V(n)          (SchurInverter.cpp:253-261)
//   k_stab                 Johnson shift of A, n < 60               (SchurInverter.cpp:264-272)
//   gemm                   S = A - Bs B^T, n < n_tr                  (SchurInverter.cpp:347-351)
//   k_stab                 shift of S (n < 60)                       (SchurInverter.cpp:364-371)
//   gj_inverse             Sinv(n) = sym(S^-1)  (inverse_symmetric_indefinite, Eigen build,
//                          LapackInverse.hpp:166-176)
//   gemm x2                T = Sinv Bs, F = Bs^T T   (W^-1 = [[Sinv, -T], [-T^T, D^-1 + F]],
//                          WInverseOperator.cpp:75-128 applied to I)
//   k_assemble_R           R = 12 W^-1 - 10 I - Rinv_{n-1}           (ForwardRPropagator.cpp:332-334)
//   gj_inverse             Rinv_n = sym(R^-1)                        (ForwardRPropagator.cpp:357-358)
//   gemm x3                dipole / overlap sweep: G_n = (G_{n-1} + C_n E_psi^T W_n^-1) Rinv_n
//
// The backward sweep Z_n = Rinv_n Z_{n+1} of BackPropagator.cpp:603-703
// is never run over the whole grid: the dipole and overlap integrals are
// linear in psi_n = (W_n^-1 Z_n)_psi, so the Simpson-weighted rows C_n of the
// integrands are propagated forward instead (G_n above) and contracted with
// Z_N once K is known.  Only the asymptotic window (<= 300 points) is swept
// backward, from stored Rinv_n, to give the psi the amplitude fit needs.
// This removes the Nr x N_t^2 storage of R^-1 (105 GB per energy at
// N_t = 1046, Nr = 12001) and the second pass over it.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <deque>
#include <map>
#include <string>
#include <vector>

#include "angular.hpp"
#include "common.cuh"
#include "devbuf.cuh"
#include "eig.cuh"
#include "riccati.cuh"
#include "scan.cuh"
#include "step_kernels.cuh"
#include "sym_rescue.cuh"
#include "tables.hpp"

namespace scatt {

namespace {

constexpr int TPB = 256;

inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

// ================================================================ step kernels

// Radial step of slot d at position j of its group's current chunk, or -1
// when the slot has none (empty slot, idle group, j past the chunk's end).
__device__ __forceinline__ int step_of(const BatchDev& b, const EnergyDev& d, int j) {
    if (!d.live) return -1;
    const GroupDev& g = b.grp[d.grp];
    return (g.n0 >= 0 && j < g.C) ? g.n0 + j : -1;
}

__device__ __forceinline__ size_t bslot(const BatchDev& b) { return (size_t)b.Np_max * (b.Nf > 0 ? b.Nf : 1); }
__device__ __forceinline__ const double* V_of(const BatchDev& b, const EnergyDev& d, int j) {
    return b.grp[d.grp].Vc + (size_t)j * b.Np_max * b.Np_max;
}
__device__ __forceinline__ const double* B_of(const BatchDev& b, const EnergyDev& d, int j) {
    return b.grp[d.grp].Bc + (size_t)j * bslot(b);
}
__device__ __forceinline__ const double* Bs_of(const BatchDev& b, const EnergyDev& d, int j) {
    return b.grp[d.grp].Bsc + (size_t)j * bslot(b);
}
__device__ __forceinline__ const double* Dinv_of(const BatchDev& b, const EnergyDev& d, int j) {
    return b.grp[d.grp].Dinvc + (size_t)j * (b.Nf > 0 ? b.Nf : 1);
}

__device__ __forceinline__ double vpol_at(const BatchDev& b, double r) {
    double vpol = 0.0;
    if (b.alpha_pol != 0.0 && r >= 1.0e-6) {
        if (b.pol_form == 0) {
            const double u = r / b.r_c;
            const double u6 = u * u * u * u * u * u;
            const double damp = 1.0 - exp(-u6);
            vpol = -0.5 * b.alpha_pol * (damp * damp) / (r * r * r * r);
        } else {
            const double s = r * r + b.r_c * b.r_c;
            vpol = -b.alpha_pol / (2.0 * (s * s));
        }
    }
    return vpol;
}

// V(n) pair p (row <= col of the upper triangle); Potentials.cpp:324-340.
__device__ __forceinline__ void build_V_pair(const BatchDev& b, int p, int n, double* V) {
    const int row = b.pair_row[p], col = b.pair_col[p];
    const double r = n * b.dr;
    double v = 0.0;
    if (r > 1e-14) {
        const double* vs = b.vsig + (size_t)n * b.n_exp;
        for (int k = b.pair_ptr[p]; k < b.pair_ptr[p + 1]; ++k) v += b.pair_G[k] * vs[b.pair_sig[k]];
        if (row == col) {
            const int l = b.l_of_mu[row];
            const double inv_r2 = 1.0 / (r * r);
            v = (v + vpol_at(b, r)) + l * (l + 1.0) * 0.5 * inv_r2;
        }
    }
    if (b.dV) v += b.dV[(size_t)n * b.Np_max * b.Np_max + row + (size_t)col * b.Np_max];
    V[row + (size_t)col * b.Np_max] = v;
    V[col + (size_t)row * b.Np_max] = v;
}

// V of every group's chunk: grid (pairs, groups, SCHUR_CHUNK), one thread per
// channel pair (mu' <= mu).
__global__ void k_build_V(BatchDev b) {
    dep_sync();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const GroupDev& g = b.grp[blockIdx.y];
    const int j = blockIdx.z;
    if (p >= b.n_pairs || g.n0 < 0 || j >= g.C) return;
    build_V_pair(b, p, g.n0 + j, g.Vc + (size_t)j * b.Np_max * b.Np_max);
}

// V(n) into one given buffer (post stages).
__global__ void k_build_V_at(BatchDev b, int n, double* V) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < b.n_pairs) build_V_pair(b, p, n, V);
}

// diagonal of V(n + 1) for the groups whose step n = n0 + j is inside the
// analytic start of the recurrence: grid (channels, groups).
__global__ void k_vdiag(BatchDev b, int j) {
    dep_sync();
    const int mu = blockIdx.x * blockDim.x + threadIdx.x;
    const GroupDev& g = b.grp[blockIdx.y];
    if (mu >= b.Np_max || g.n0 < 0 || j >= g.C || g.n0 + j >= b.n_start) return;
    const int n = g.n0 + j + 1;
    // pair index of (mu, mu) in the row-major upper triangle
    const long p = (long)mu * b.Np_max - ((long)mu * (mu - 1)) / 2;
    const double r = n * b.dr;
    double v = 0.0;
    if (r > 1e-14) {
        const double* vs = b.vsig + (size_t)n * b.n_exp;
        for (int k = b.pair_ptr[p]; k < b.pair_ptr[p + 1]; ++k) v += b.pair_G[k] * vs[b.pair_sig[k]];
        const int l = b.l_of_mu[mu];
        const double inv_r2 = 1.0 / (r * r);
        v = (v + vpol_at(b, r)) + l * (l + 1.0) * 0.5 * inv_r2;
    }
    if (b.dV) v += b.dV[(size_t)n * b.Np_max * b.Np_max + mu + (size_t)mu * b.Np_max];
    g.vdiag1[mu] = v;
}

__device__ __forceinline__ double dinv_of(const BatchDev& b, int l, int n) {
    // r = r_min + n dr with r_min = dr (WavefunctionSetup.cpp:327)
    const double r = b.dr + n * b.dr;
    const double r2 = r * r;
    const double cent = (r2 > 1e-30) ? ((double)l * (l + 1)) / r2 : 0.0;
    double Df = 1.0 - b.h2_12 * cent;
    if (Df < b.W_min) Df = b.W_min;
    return 1.0 / Df;
}

// B(n) = h^2/12 * (2 sqrt(2 pi) / r) * sum_lambda G chi, r = n dr, one
// thread per row mu * n_sigma + sigma; Bs = B D^-1 (ExchangeCoupling.cpp:65-136).
__device__ __forceinline__ void build_B_row(const BatchDev& b, int row, int n, double* B, double* Bs,
                                            double* Dinv) {
    const int rows = b.Np_max * b.n_sigma;
    if (row < b.Nf) Dinv[row] = dinv_of(b, b.l_sigma[row % b.n_sigma], n);
    if (row >= rows) return;
    const int mu = row / b.n_sigma, sigma = row % b.n_sigma;
    const double r = n * b.dr;
    const bool on = (n < b.n_tr) && !(r < 1e-10);
    const double factor = on ? 2.0 * sqrt(2.0 * M_PI) / r : 0.0;
    double acc[64];
    const int no = b.n_occ;
    for (int i = 0; i < no && i < 64; ++i) acc[i] = 0.0;
    if (on) {
        const double* ch = b.chi + (size_t)n * b.n_lambda * no;
        for (int k = b.ex_ptr[row]; k < b.ex_ptr[row + 1]; ++k) {
            const double g = b.ex_G[k];
            const double* c = ch + (size_t)b.ex_lam[k] * no;
            for (int i = 0; i < no && i < 64; ++i) acc[i] += g * c[i];
        }
    }
    for (int i = 0; i < no && i < 64; ++i) {
        const int f = i * b.n_sigma + sigma;
        const double Bv = on ? b.h2_12 * (factor * acc[i]) : 0.0;
        B[mu + (size_t)f * b.Np_max] = Bv;
        Bs[mu + (size_t)f * b.Np_max] = Bv * dinv_of(b, b.l_sigma[sigma], n);
    }
}

// B, Bs, D^-1 of every group's chunk: grid (rows, groups, SCHUR_CHUNK).
__global__ void k_build_B(BatchDev b) {
    dep_sync();
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    const GroupDev& g = b.grp[blockIdx.y];
    const int j = blockIdx.z;
    if (g.n0 < 0 || j >= g.C) return;
    const size_t sl = bslot(b);
    build_B_row(b, row, g.n0 + j, g.Bc + j * sl, g.Bsc + j * sl, g.Dinvc + (size_t)j * (b.Nf > 0 ? b.Nf : 1));
}

// B(n), Bs(n), D^-1(n) into given buffers (post stages).
__global__ void k_build_B_at(BatchDev b, int n, double* B, double* Bs, double* Dinv) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    build_B_row(b, row, n, B, Bs, Dinv);
}

__device__ __forceinline__ bool in_seg(const EnergyDev& d, int n) { return n >= d.seg_lo && n < d.seg_hi; }

// Sinv of step n at chunk position j: the segment store, the asymptotic
// window store, or the chunk slot j.
__device__ __forceinline__ double* sinv_at(const BatchDev& b, const EnergyDev& d, int n, int j) {
    const size_t np2 = (size_t)d.Np * d.Np;
    if (in_seg(d, n)) return d.segS + (size_t)(n - d.seg_lo) * np2;
    return (n >= b.n_s && d.tailS) ? d.tailS + (size_t)(n - b.n_s) * np2 : d.Sinv + (size_t)j * np2;
}

// Rinv(n): the segment store, the asymptotic window store, or the ping-pong pair.
__device__ __forceinline__ double* rinv_at(const BatchDev& b, const EnergyDev& d, int n) {
    const size_t nt2 = (size_t)d.Nt * d.Nt;
    if (in_seg(d, n)) return d.segR + (size_t)(n - d.seg_lo) * nt2;
    return (n >= b.n_s && d.tailR) ? d.tailR + (size_t)(n - b.n_s) * nt2 : ((n & 1) ? d.Rinv1 : d.Rinv0);
}

// G(n-1)^T, accumulated into H(n)^T during step n (K x N_t, ld K).
__device__ __forceinline__ double* gacc_at(const BatchDev& b, const EnergyDev& d, int n) {
    if (in_seg(d, n)) return d.segH + (size_t)(n - d.seg_lo) * b.Krows * d.Nt;
    return (n & 1) ? d.G1 : d.G0;
}

// Entry of a symmetric inverse of order n (ld n throughout), its status cleared.
// No rows are refined: over the 595 matrices R of a sweep (order 1046, 0.05
// bohr) the plain sweep's median error is 5.8e-16 (general inverse 6.8e-16), the
// rescue's rules take the outliers, and the dipoles at k = 1.5, which rounding of
// one S^-1 moves by 1e-7 to 3e-7, stay within the tolerance of the stored oracle
// results (1.1e-7; with refined rows 1.2e-7 to 3e-7).
__device__ __forceinline__ SymEntry sym_entry(double* A, double* W, double* panel, double* out, unsigned* stat,
                                              int* status, int n) {
    const size_t T = sym_tiles_of(n);
    status[0] = status[1] = 0;
    return SymEntry{A, W, panel, panel + T * SYM_TILE, panel + 2 * T * SYM_TILE, out, stat, status, n, n, INFINITY};
}

// Fills a chunk's GEMM and inverse entries, index j * count + e (pointer
// bookkeeping only; one launch for its SCHUR_CHUNK steps, which read nothing
// that the chunk changes).  Entries of steps outside a slot's chunk, and of
// stages a step does not take, are empty (M = 0, n = 0): the kernels skip them.
// An inverse has one of its two entries filled: with `symmetric` the sweep's
// where the slot's own N_t is above one tile, else the general inverse's.
__global__ void k_prepare(BatchDev b, bool symmetric) {
    dep_sync();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx <= SCHUR_CHUNK) b.barrier[idx] = 0;
    // the records of both inverses' entries
    const size_t words4 = 2 * (size_t)b.count * SCHUR_CHUNK * b.stat_stride / 4;
    for (size_t u = idx; u < words4; u += (size_t)gridDim.x * blockDim.x)
        reinterpret_cast<uint4*>(b.stat)[u] = make_uint4(0, 0, 0, 0);
    if (idx >= b.count * SCHUR_CHUNK) return;
    const int j = idx / b.count, e = idx % b.count;
    EnergyDev& d = b.ed[e];
    const int n = step_of(b, d, j);
    const int Np = d.Np, Nt = d.Nt, Nf = b.Nf, K = b.Krows;
    const size_t np2 = (size_t)Np * Np;
    double* S = d.S + j * np2;
    const GemmEntry none{nullptr, nullptr, nullptr, 0, 0, 0, 1, 1, 1, 0.0, 1.0};
    GemmEntry *gmG1 = b.gmG + 2 * (size_t)j * b.count + e, *gmG2 = gmG1 + b.count;
    if (n < 0) {
        b.gmS[idx] = b.gmT[idx] = b.gmF[idx] = *gmG1 = *gmG2 = b.gmG3[idx] = b.gmGA[idx] = none;
        b.gjS[idx] = GjEntry{S, S, S, d.sigS, d.ridS, d.stS + 4 * j, 0, 1, 1, d.PS, d.sgS};
        b.gjR[idx] = GjEntry{d.Ra, d.Rw, d.Ra, d.sigR, d.ridR, d.stR + 4 * j, 0, 1, 1, d.PR, d.sgR};
        b.syS[idx].n = b.syR[idx].n = 0;
        return;
    }
    const bool exch = n < b.n_tr && Nf > 0;
    const bool sweep = n <= b.N - 1;
    double* sinv = sinv_at(b, d, n, j);
    double* rinv = rinv_at(b, d, n);
    double* gcur = gacc_at(b, d, n);
    double* gnext = gacc_at(b, d, n + 1);
    const double* Bs = Bs_of(b, d, j);
    const double* Cn = (n < b.n_pts) ? b.Ctab + (size_t)n * K * b.Np_max : nullptr;
    // Bs B^T = B D^-1 B^T and A are symmetric: lower tiles only, mirrored
    b.gmS[idx] = exch ? GemmEntry{Bs, B_of(b, d, j), S, Np, Np, Nf, b.Np_max, b.Np_max, Np, -1.0, 1.0, 1} : none;
    const bool sym = symmetric && Nt > SYM_NB;
    b.gjS[idx] = GjEntry{S, d.Sw + j * b.sw_stride, sinv, d.sigS + (size_t)j * Np, d.ridS + (size_t)j * Np,
                         d.stS + 4 * j, sym ? 0 : Np, Np, Np, d.PS + j * b.ps_stride, d.sgS + (size_t)j * 4 * Np};
    if (sym) b.syS[idx] = sym_entry(S, d.Sw + j * b.sw_stride, d.PS + j * b.ps_stride, sinv,
                                     b.stat + ((size_t)b.count * SCHUR_CHUNK + idx) * b.stat_stride, d.stS + 4 * j, Np);
    else b.syS[idx].n = 0;
    b.gmT[idx] = exch ? GemmEntry{sinv, Bs, d.T, Np, Nf, Np, Np, b.Np_max, Np, 1.0, 0.0} : none;
    // F = Bs^T Sinv Bs is symmetric: lower tiles only, mirrored
    b.gmF[idx] = exch ? GemmEntry{Bs, d.T, d.F, Nf, Nf, Np, b.Np_max, Np, Nf, 1.0, 0.0, 1} : none;
    *gmG1 = (sweep && Cn) ? GemmEntry{Cn, sinv, gcur, K, Np, Np, K, Np, K, 1.0, 1.0} : none;
    *gmG2 = (sweep && Cn && exch) ? GemmEntry{Cn, d.T, gcur + (size_t)Np * K, K, Nf, Np, K, Np, K, -1.0, 1.0} : none;
    b.gmG3[idx] = sweep ? GemmEntry{gcur, rinv, gnext, K, Nt, Nt, K, Nt, K, 1.0, 0.0} : none;
    // the fit accumulation G_A(n)^T = H_A(n)^T Rinv(n) over n_s <= n <= N - 1
    b.gmGA[idx] = (d.GA0 && n >= b.n_s && sweep)
                      ? GemmEntry{(n & 1) ? d.GA1 : d.GA0, rinv, (n & 1) ? d.GA0 : d.GA1, 2 * Np, Nt, Nt, 2 * Np, Nt,
                                  2 * Np, 1.0, 0.0}
                      : none;
    const bool inv = n >= b.n_start;
    b.gjR[idx] = GjEntry{d.Ra, d.Rw, rinv, d.sigR, d.ridR, d.stR + 4 * j, inv && !sym ? Nt : 0, Nt, Nt, d.PR, d.sgR};
    if (inv) b.rargs[idx] = RArgs{sinv, d.T, d.F, Dinv_of(b, d, j), rinv_at(b, d, n - 1), Np, Nt, Nf, n < b.n_tr};
    if (inv && sym) b.syR[idx] = sym_entry(d.Ra, d.Rw, d.PR, rinv, b.stat + (size_t)idx * b.stat_stride,
                                             d.stR + 4 * j, Nt);
    else b.syR[idx].n = 0;
}

// A = (1 + h^2 E / 6) I - h^2/6 V(n) into Schur slot j (SchurInverter.cpp:253-261);
// grid (x, slots, SCHUR_CHUNK).
__global__ void k_init_S(BatchDev b) {
    dep_sync();
    const int e = blockIdx.y, j = blockIdx.z;
    const EnergyDev& d = b.ed[e];
    if (step_of(b, d, j) < 0) return;
    const int Np = d.Np;
    const long total = (long)Np * Np;
    double* S = d.S + (size_t)j * total;
    const double* V = V_of(b, d, j);
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
         idx += (long)gridDim.x * blockDim.x) {
        const int i = (int)(idx % Np), jc = (int)(idx / Np);
        const double diag = (i == jc) ? d.c : 0.0;
        S[idx] = diag - b.h2_6 * V[i + (size_t)jc * b.Np_max];
    }
}

__device__ double block_min(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_down_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = red[0];
        for (int i = 1; i < (int)(blockDim.x >> 5); ++i) m = fmin(m, red[i]);
        red[32] = m;
    }
    __syncthreads();
    return red[32];
}

// Johnson stability shift (SchurInverter.cpp:30-59): Gershgorin lower bound
// first; when inconclusive the exact smallest eigenvalue c + lambda_min(M),
// with lambda_min(M) precomputed per n (the matrix differs from M only by
// c I).  which = 0: A (also records delta_A), 1: S = A_shifted - Bs B^T
// (exchange steps only).  Grid (slots, SCHUR_CHUNK); steps n >= stab_n skip.
__global__ void k_stab(BatchDev b, int which) {
    dep_sync();
    const int e = blockIdx.x, slot = blockIdx.y;
    EnergyDev& d = b.ed[e];
    const int n = step_of(b, d, slot);
    if (n < 0 || n >= b.stab_n) return;
    if (which == 1 && !(n < b.n_tr && b.Nf > 0)) return;
    const int Np = d.Np;
    double* S = d.S + (size_t)slot * Np * Np;
    __shared__ double red[33];
    double g = INFINITY;
    for (int i = threadIdx.x; i < Np; i += blockDim.x) {
        double off = 0.0;
        for (int j = 0; j < Np; ++j)
            if (j != i) off += fabs(S[i + (size_t)j * Np]);
        g = fmin(g, S[i + (size_t)i * Np] - off);
    }
    const double gersh = block_min(g, red);
    if (threadIdx.x == 0) {
        double me;
        if (gersh > b.W_min + 0.05) me = gersh;
        else me = (which == 0) ? d.c + d.lmA[n] : (d.c + d.deltaAc[slot]) + d.lmS[n];
        double delta = 0.0;
        if (me < b.W_min) {
            delta = b.W_min - me + b.margin;
            // the chunk's steps run in parallel blocks of this slot: count atomically
            atomicAdd(which == 0 ? &d.shiftsA : &d.shiftsS, 1);
        }
        if (which == 0) d.deltaAc[slot] = delta;
        if (d.stabd) d.stabd[2 * n + which] = delta;
        red[0] = delta;
    }
    __syncthreads();
    const double delta = red[0];
    if (delta != 0.0)
        for (int i = threadIdx.x; i < Np; i += blockDim.x) S[i + (size_t)i * Np] += delta;
}

// Element (i, jc) of R = 12 W^-1 - 10 I - Rinv_prev, W^-1 = [[Sinv, -T],
// [-T^T, D^-1 + F]]; 0 where !in.  The sources are chosen by selects and read
// under predicates (no branch keeps one element's loads behind another's).
__device__ __forceinline__ double r_elem(const RArgs& a, int i, int jc, bool in) {
    const bool pi = i < a.Np, pj = jc < a.Np;
    const int fi = i - a.Np, fj = jc - a.Np;
    const double* src = pi && pj ? a.sinv + i + (size_t)jc * a.Np
                        : pi     ? a.T + i + (size_t)fj * a.Np
                        : pj     ? a.T + jc + (size_t)fi * a.Np
                                 : a.F + fi + (size_t)fj * a.Nf;
    const bool some = in && ((pi && pj) || a.exch);
    const bool diag = in && i == jc;
    double w = some ? *src : 0.0;
    const double d = diag && !pi ? a.Dinv[fi] : 0.0;
    const double prev = in ? a.prev[i + (size_t)jc * a.Nt] : 0.0;
    w = (pi != pj) ? -w : w;
    const double u = 12.0 * (d + w) - (diag ? 10.0 : 0.0);
    return u - prev;
}

// R(n) into Ra, column-major, of the slots whose general inverse takes it (see
// k_prepare); those whose step is inside the analytic start skip.
__global__ void k_assemble_R(BatchDev b, int j) {
    dep_sync();
    const int e = blockIdx.y;
    const EnergyDev& d = b.ed[e];
    const int n = step_of(b, d, j);
    if (n < b.n_start) return;                 // also n < 0
    if (b.gjR[(size_t)j * b.count + e].n == 0) return;
    const RArgs a = b.rargs[(size_t)j * b.count + e];
    const int Nt = d.Nt;
    const long total = (long)Nt * Nt;
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
         idx += (long)gridDim.x * blockDim.x)
        d.Ra[idx] = r_elem(a, (int)(idx % Nt), (int)(idx / Nt), true);
}

// The same for one entry of a rescue (sym_rescue_kernel).
struct RSource {
    BatchDev b;
    int j;
    __device__ __forceinline__ void operator()(int e, const SymEntry& s, int first, int stride) const {
        const RArgs a = b.rargs[(size_t)j * b.count + e];
        const long total = (long)s.n * s.n;
        for (long idx = first; idx < total; idx += stride)
            s.A[idx] = r_elem(a, (int)(idx % s.n), (int)(idx / s.n), true);
    }
};

// R(n) packed for the symmetric sweep; nt tiles of the largest slot.  Bound
// by HBM: it reads Sinv, T, F and Rinv(n - 1) once (the lower triangle's half
// of the symmetric ones) and writes the triangle's tiles.
__global__ void __launch_bounds__(SYM_THREADS, 3) k_assemble_R_tiles(BatchDev b, int j, int nt) {
    dep_sync();
    extern __shared__ double smem[];
    int ent, t;
    sym_pack_index(blockIdx.x, b.count, nt, ent, t);
    const SymEntry s = b.syR[(size_t)j * b.count + ent];
    const RArgs a = b.rargs[(size_t)j * b.count + ent];
    const int T = sym_tiles_of(s.n);
    if (t >= T * (T + 1) / 2) return;
    // the sources are symmetric: taken transposed, consecutive lanes read consecutive rows
    sym_pack_tile(s, t, *reinterpret_cast<SymDiagShared*>(smem),
                  [&a](int gi, int gj, bool in) { return r_elem(a, gj, gi, in); });
}

// Analytic diagonal Rinv for 1 <= n < n_start, 0 at n = 0
// (ForwardRPropagator.cpp:78-134): zero fill, then k_analytic_R_diag.
__global__ void k_analytic_R(BatchDev b, int j) {
    dep_sync();
    const int e = blockIdx.y;
    const EnergyDev& d = b.ed[e];
    const int n = step_of(b, d, j);
    if (n < 0 || n >= b.n_start) return;
    double* out = rinv_at(b, d, n);
    const long total = (long)d.Nt * d.Nt;
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
         idx += (long)gridDim.x * blockDim.x)
        out[idx] = 0.0;
}

__global__ void k_analytic_R_diag(BatchDev b, int j) {
    dep_sync();
    const int e = blockIdx.y;
    const EnergyDev& d = b.ed[e];
    const int n = step_of(b, d, j);
    if (n <= 0 || n >= b.n_start) return;
    const int Np = d.Np, Nt = d.Nt;
    double* out = rinv_at(b, d, n);
    const double* V = V_of(b, d, j);
    const double* vdiag1 = b.grp[d.grp].vdiag1;
    const double h = b.dr;
    const double rn = b.dr + n * h, rn1 = b.dr + (n + 1) * h;
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < Nt; m += gridDim.x * blockDim.x) {
        double val = 0.0;
        if (m < Np) {
            const int l = b.l_of_mu[m];
            const double Mn = 1.0 + b.h2_6 * (d.E - V[m + (size_t)m * b.Np_max]);
            const double Mn1 = 1.0 + b.h2_6 * (d.E - vdiag1[m]);
            const double yn = riccati_j(l, d.k * rn);
            const double yn1 = riccati_j(l, d.k * rn1);
            const double den = Mn1 * yn1;
            if (fabs(den) > 1e-300) val = (Mn * yn) / den;
        } else {
            const int f = m - Np;
            const int l = b.l_sigma[f % b.n_sigma];
            const double rn2 = rn * rn, rn12 = rn1 * rn1;
            const double cn = (rn2 > 1e-30) ? (double)(l * (l + 1)) / rn2 : 0.0;
            const double cn1 = (rn12 > 1e-30) ? (double)(l * (l + 1)) / rn12 : 0.0;
            double Mn = 1.0 - b.h2_12 * cn, Mn1 = 1.0 - b.h2_12 * cn1;
            if (Mn < b.W_min) Mn = b.W_min;
            if (Mn1 < b.W_min) Mn1 = b.W_min;
            const double yn = pow(rn, (double)(l + 1));
            const double yn1 = pow(rn1, (double)(l + 1));
            const double den = Mn1 * yn1;
            if (fabs(den) > 1e-300) val = (Mn * yn) / den;
        }
        out[m + (size_t)m * Nt] = val;
    }
}

// sticky per-slot error: the chunk's first failing inversion (step, code),
// Schur inverse before R^-1 at each step; runs at the end of the chunk.
__global__ void k_collect(BatchDev b) {
    dep_sync();
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= b.count) return;
    EnergyDev& d = b.ed[e];
    for (int j = 0; j < SCHUR_CHUNK && d.err_code == 0; ++j) {
        const int n = step_of(b, d, j);
        if (n < 0) break;
        int st = d.stS[4 * j];
        if (st == 0 && n >= b.n_start) st = d.stR[4 * j];
        if (st != 0) {
            d.err_code = (st == DEV_SINGULAR) ? SCATT_ERR_SINGULAR : SCATT_ERR_NONFINITE;
            d.err_step = n;
        }
    }
}

// ---- forward accumulation of the amplitude fit (no window store)
// The fit (AsymptoticAmplitudes.cpp:64-359) is linear in psi over the window
// [n_s, ne_fit]: per channel mu of angular momentum l,
//   A[mu, :] = sum_i (M00 j_l(i) + M01 y_l(i)) psi_i[mu, :],  B likewise with M10, M11,
// with M the inverse of the 2 x 2 normal matrix of (j_l, y_l) on the window.
// psi_i = E_psi W^-1(i) Z(i) and Z(i) = Rinv(i) ... Rinv(N-1) Z_N, so [A; B] =
// G_A(N-1)^T Z_N with G_A accumulated forward like the dipole rows.

// normal matrices per l (as k_aa_normal, same order of summation); grid (l, slots of the range)
__global__ void k_ab_normal(BatchDev b, int e0) {
    EnergyDev& d = b.ed[e0 + blockIdx.y];
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (!d.live || !d.Mab || l > d.l_cont) return;
    double m00 = 0.0, m01 = 0.0, m11 = 0.0;
    for (int i = 0; i < b.nfit; ++i) {
        const double r = b.dr + (b.n_s + i) * b.dr;
        const double jv = riccati_j(l, d.k * r), yv = riccati_y(l, d.k * r);
        m00 += jv * jv;
        m01 += jv * yv;
        m11 += yv * yv;
    }
    const double det = m00 * m11 - m01 * m01;
    const double mx = fmax(fabs(m00), fmax(fabs(m01), fabs(m11)));
    const bool singular = !(fabs(det) > 1e-20 * mx * mx);
    double* o = d.Mab + l * 8;
    o[4] = singular ? 1.0 : 0.0;
    o[5] = det;
    o[6] = mx;
    if (!singular) {
        o[0] = m11 / det; o[1] = -m01 / det; o[2] = -m01 / det; o[3] = m00 / det;
    } else {
        o[0] = 1.0; o[1] = 0.0; o[2] = 0.0; o[3] = 1.0;
    }
}

// fit weights wAB[i][a][mu]; grid (x, slots of the range)
__global__ void k_ab_weights(BatchDev b, int e0) {
    EnergyDev& d = b.ed[e0 + blockIdx.y];
    if (!d.live || !d.wAB) return;
    const int Np = d.Np;
    const long total = (long)b.nfit * Np;
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total; idx += (long)gridDim.x * blockDim.x) {
        const int i = (int)(idx / Np), mu = (int)(idx % Np);
        const int l = b.l_of_mu[mu];
        const double r = b.dr + (b.n_s + i) * b.dr;
        const double jv = riccati_j(l, d.k * r), yv = riccati_y(l, d.k * r);
        const double* m = d.Mab + l * 8;
        const bool closed = m[4] != 0.0;
        d.wAB[((size_t)i * 2 + 0) * Np + mu] = closed ? 0.0 : m[0] * jv + m[1] * yv;
        d.wAB[((size_t)i * 2 + 1) * Np + mu] = closed ? 0.0 : m[2] * jv + m[3] * yv;
    }
}

// H_A(n)^T = G_A(n-1)^T + D_AB(n) [Sinv, -T] on the fit window; grid (x, slots)
__global__ void k_acc_ab(BatchDev b, int j) {
    dep_sync();
    const EnergyDev& d = b.ed[blockIdx.y];
    const int n = step_of(b, d, j);
    if (n < b.n_s || n > b.ne_fit || !d.GA0) return;
    const int Np = d.Np, Nt = d.Nt, two = 2 * Np;
    const bool exch = n < b.n_tr && b.Nf > 0;
    const double* sinv = sinv_at(b, d, n, j);
    const double* w = d.wAB + (size_t)(n - b.n_s) * two;
    double* ga = (n & 1) ? d.GA1 : d.GA0;
    const long total = (long)two * Nt;
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total; idx += (long)gridDim.x * blockDim.x) {
        const int r = (int)(idx % two), c = (int)(idx / two);
        const int mu = r % Np;
        double v;
        if (c < Np) v = sinv[mu + (size_t)c * Np];
        else v = exch ? -d.T[mu + (size_t)(c - Np) * Np] : 0.0;
        ga[idx] += w[r] * v;
    }
}

// rows of closed channels: A = I, B = 0 (AsymptoticAmplitudes.cpp:177-212); grid (x, energies)
struct AbEntry {
    double* A;
    double* B;
    const double* Mab;
    int Np;
};
__global__ void k_ab_closed(const AbEntry* __restrict__ ents, const int* l_of_mu) {
    const AbEntry a = ents[blockIdx.y];
    const long total = (long)a.Np * a.Np;
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total; idx += (long)gridDim.x * blockDim.x) {
        const int mu = (int)(idx % a.Np), col = (int)(idx / a.Np);
        if (a.Mab[l_of_mu[mu] * 8 + 4] != 0.0) {
            a.A[idx] = (col == mu) ? 1.0 : 0.0;
            a.B[idx] = 0.0;
        }
    }
}

// End of a chunk: every running group moves on by its chunk's length; a
// group whose chunk reached the stop step stops (n0 = -1).
__global__ void k_advance(BatchDev b) {
    dep_sync();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= b.ngroups) return;
    GroupDev& G = b.grp[g];
    if (G.n0 < 0) return;
    const int n0 = G.n0 + G.C;
    if (n0 >= b.n_stop) { G.n0 = -1; G.C = 0; return; }
    G.n0 = n0;
    G.C = min(SCHUR_CHUNK, b.n_stop - n0);
}

// Start (n0 >= 0) or stop (n0 = -1) one group between chunks.
__global__ void k_set_group(BatchDev b, int g, int n0) {
    GroupDev& G = b.grp[g];
    G.n0 = n0;
    G.C = n0 < 0 ? 0 : min(SCHUR_CHUNK, b.n_stop - n0);
}


// ================================================================ post kernels

struct CopyEntry {
    const double* src;
    double* dst;
    int rows, cols, lds, ldd;
    double scale;
};

__global__ void k_copy(const CopyEntry* __restrict__ ents) {
    const CopyEntry c = ents[blockIdx.y];
    const long total = (long)c.rows * c.cols;
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
         idx += (long)gridDim.x * blockDim.x) {
        const int i = (int)(idx % c.rows), j = (int)(idx / c.rows);
        c.dst[i + (size_t)j * c.ldd] = c.scale * c.src[i + (size_t)j * c.lds];
    }
}

// Frobenius norms of R_psi_f and R_f_psi (KMatrixExtractor.cpp:108-121)
__global__ void k_block_norms(const double* const* R, const int* Np, const int* Nt, double* out) {
    const int e = blockIdx.x;
    const double* M = R[e];
    const int np = Np[e], nt = Nt[e];
    __shared__ double red[2][32];
    double a = 0.0, c = 0.0;
    for (long idx = threadIdx.x; idx < (long)np * (nt - np); idx += blockDim.x) {
        const int i = (int)(idx % np), j = np + (int)(idx / np);
        const double x = M[i + (size_t)j * nt];
        a += x * x;
        const double y = M[j + (size_t)i * nt];
        c += y * y;
    }
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        c += __shfl_down_sync(0xffffffffu, c, o);
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) { red[0][w] = a; red[1][w] = c; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double sa = 0.0, sc = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) { sa += red[0][i]; sc += red[1][i]; }
        out[2 * e] = sqrt(sa);
        out[2 * e + 1] = sqrt(sc);
    }
}

// Riccati tables of the matching radii: J/Y/W at r_in, r_out (KMatrixExtractor.cpp:131-153)
struct KmeEntry {
    const double* Ssch;   // Np x Np (ld Np)
    double* Amat;
    double* Bmat;
    double* tab;          // 6 x Np: Jin Jout Yin Yout Win Wout
    int Np;
    double k;
};

__global__ void k_kme_tab(const KmeEntry* __restrict__ ents, const int* l_of_mu, double dr, int Nr) {
    const KmeEntry en = ents[blockIdx.y];
    const int mu = blockIdx.x * blockDim.x + threadIdx.x;
    if (mu >= en.Np) return;
    const int l = l_of_mu[mu];
    const double h = dr;
    const double h2_12 = h * h / 12.0;
    const int n_match = Nr - 2;
    const double r_in = dr + n_match * h, r_out = dr + (n_match + 1) * h;
    const double k = en.k, k2 = k * k;
    const double ci = (double)(l * (l + 1)) / (r_in * r_in);
    const double co = (double)(l * (l + 1)) / (r_out * r_out);
    en.tab[0 * en.Np + mu] = riccati_j(l, k * r_in);
    en.tab[1 * en.Np + mu] = riccati_j(l, k * r_out);
    en.tab[2 * en.Np + mu] = riccati_y(l, k * r_in);
    en.tab[3 * en.Np + mu] = riccati_y(l, k * r_out);
    en.tab[4 * en.Np + mu] = 1.0 + h2_12 * (k2 - ci);
    en.tab[5 * en.Np + mu] = 1.0 + h2_12 * (k2 - co);
}

// A_mat = W_out J_out - sym(S) (W_in J_in),  B_mat = sym(S) (W_in Y_in) - W_out Y_out
__global__ void k_kme_mats(const KmeEntry* __restrict__ ents) {
    const KmeEntry en = ents[blockIdx.y];
    const int Np = en.Np;
    const long total = (long)Np * Np;
    const double* t = en.tab;
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
         idx += (long)gridDim.x * blockDim.x) {
        const int i = (int)(idx % Np), j = (int)(idx / Np);
        const double s = 0.5 * (en.Ssch[idx] + en.Ssch[j + (size_t)i * Np]);
        const double Jin = t[j], Yin = t[2 * Np + j], Win = t[4 * Np + j];
        const double dJ = (i == j) ? t[5 * Np + i] * t[1 * Np + i] : 0.0;
        const double dY = (i == j) ? t[5 * Np + i] * t[3 * Np + i] : 0.0;
        en.Amat[idx] = dJ - s * (Win * Jin);
        en.Bmat[idx] = s * (Win * Yin) - dY;
    }
}

// K <- sym(K_raw) (KMatrixExtractor.cpp:165);  psi_bc = J_N + Y_N K (:222-223)
__global__ void k_kme_final(const KmeEntry* __restrict__ ents, const double* const* Kraw,
                            double* const* Kout, double* const* psibc) {
    const KmeEntry en = ents[blockIdx.y];
    const int e = blockIdx.y;
    const int Np = en.Np;
    const long total = (long)Np * Np;
    const double* t = en.tab;
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
         idx += (long)gridDim.x * blockDim.x) {
        const int i = (int)(idx % Np), j = (int)(idx / Np);
        const double K = 0.5 * (Kraw[e][idx] + Kraw[e][j + (size_t)i * Np]);
        Kout[e][idx] = K;
        psibc[e][idx] = ((i == j) ? t[1 * Np + i] : 0.0) + t[3 * Np + i] * K;
    }
}

// Z_psi = psi + h^2/6 E psi - h^2/6 V_N psi + B_N f_N  (BackPropagator.cpp:176-181); Z_f = 0
struct ZEntry {
    const double* psi;    // Np x Np
    const double* Vpsi;   // h^2/6 V psi
    const double* Bf;     // B f  (or nullptr)
    double* Z;            // Nt x Np
    int Np, Nt;
    double hE;            // h^2/6 E
};

__global__ void k_build_Z(const ZEntry* __restrict__ ents) {
    const ZEntry z = ents[blockIdx.y];
    const long total = (long)z.Nt * z.Np;
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
         idx += (long)gridDim.x * blockDim.x) {
        const int i = (int)(idx % z.Nt), j = (int)(idx / z.Nt);
        double v = 0.0;
        if (i < z.Np) {
            const size_t q = i + (size_t)j * z.Np;
            const double p = z.psi[q];
            v = p + z.hE * p;
            v -= z.Vpsi[q];
            if (z.Bf) v += z.Bf[q];
        }
        z.Z[idx] = v;
    }
}

// ---- asymptotic amplitudes (AsymptoticAmplitudes.cpp:64-359)
struct AaEntry {
    const double* psiT;   // window psi, slot (n - n_s) * Np * Np
    double* tab;          // [2][lmax+1][nfit]  jhat, yhat
    double* M;            // [lmax+1][8]: Minv (4), closed flag, det, maxM, unused
    double* A;
    double* B;
    double* red;          // [Np*Np][2] per (mu, j): max |psi|, max residual
    int Np, lmax;
    double k;
};

__global__ void k_aa_tab(const AaEntry* __restrict__ ents, int ns, int nfit, double dr) {
    const AaEntry a = ents[blockIdx.y];
    const int total = (a.lmax + 1) * nfit;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
        const int l = idx / nfit, i = idx % nfit;
        const double r = dr + (ns + i) * dr;
        const double kr = a.k * r;
        a.tab[(0 * (a.lmax + 1) + l) * nfit + i] = riccati_j(l, kr);
        a.tab[(1 * (a.lmax + 1) + l) * nfit + i] = riccati_y(l, kr);
    }
}

__global__ void k_aa_normal(const AaEntry* __restrict__ ents, int nfit) {
    const AaEntry a = ents[blockIdx.y];
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l > a.lmax) return;
    const double* jv = a.tab + (0 * (a.lmax + 1) + l) * nfit;
    const double* yv = a.tab + (1 * (a.lmax + 1) + l) * nfit;
    double m00 = 0.0, m01 = 0.0, m11 = 0.0;
    for (int i = 0; i < nfit; ++i) {
        m00 += jv[i] * jv[i];
        m01 += jv[i] * yv[i];
        m11 += yv[i] * yv[i];
    }
    const double det = m00 * m11 - m01 * m01;
    const double mx = fmax(fabs(m00), fmax(fabs(m01), fabs(m11)));
    const bool singular = !(fabs(det) > 1e-20 * mx * mx);
    double* o = a.M + l * 8;
    o[4] = singular ? 1.0 : 0.0;
    o[5] = det;
    o[6] = mx;
    if (!singular) {
        o[0] = m11 / det;
        o[1] = -m01 / det;
        o[2] = -m01 / det;
        o[3] = m00 / det;
    } else {
        o[0] = 1.0; o[1] = 0.0; o[2] = 0.0; o[3] = 1.0;
    }
}

__global__ void k_aa_fit(const AaEntry* __restrict__ ents, const int* l_of_mu, int nfit) {
    const AaEntry a = ents[blockIdx.y];
    const int Np = a.Np;
    const long total = (long)Np * Np;
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
         idx += (long)gridDim.x * blockDim.x) {
        const int mu = (int)(idx % Np);
        const int l = l_of_mu[mu];
        const double* jv = a.tab + (0 * (a.lmax + 1) + l) * nfit;
        const double* yv = a.tab + (1 * (a.lmax + 1) + l) * nfit;
        double yj = 0.0, yy = 0.0, mxp = 0.0;
        for (int i = 0; i < nfit; ++i) {
            const double p = a.psiT[(size_t)i * Np * Np + idx];
            yj += jv[i] * p;
            yy += yv[i] * p;
            mxp = fmax(mxp, fabs(p));
        }
        const double* m = a.M + l * 8;
        double A, B;
        if (m[4] != 0.0) {
            A = ((int)(idx / Np) == mu) ? 1.0 : 0.0;
            B = 0.0;
        } else {
            A = m[0] * yj + m[1] * yy;
            B = m[2] * yj + m[3] * yy;
        }
        a.A[idx] = A;
        a.B[idx] = B;
        double res = 0.0;
        if (m[4] == 0.0) {
            for (int i = 0; i < nfit; ++i) {
                const double p = a.psiT[(size_t)i * Np * Np + idx];
                res = fmax(res, fabs((jv[i] * A + yv[i] * B) - p));
            }
        }
        a.red[2 * idx] = mxp;
        a.red[2 * idx + 1] = res;
    }
}

// max over a per-energy array of pairs -> out[2e], out[2e+1]
__global__ void k_max_pairs(const double* const* red, const int* count, double* out) {
    const int e = blockIdx.x;
    __shared__ double s0[32], s1[32];
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < count[e]; i += blockDim.x) {
        a = fmax(a, red[e][2 * i]);
        b = fmax(b, red[e][2 * i + 1]);
    }
    for (int o = 16; o > 0; o >>= 1) {
        a = fmax(a, __shfl_down_sync(0xffffffffu, a, o));
        b = fmax(b, __shfl_down_sync(0xffffffffu, b, o));
    }
    if ((threadIdx.x & 31) == 0) { s0[threadIdx.x >> 5] = a; s1[threadIdx.x >> 5] = b; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < (int)(blockDim.x >> 5); ++i) { a = fmax(a, s0[i]); b = fmax(b, s1[i]); }
        a = fmax(a, s0[0]); b = fmax(b, s1[0]);
        out[2 * e] = a;
        out[2 * e + 1] = b;
    }
}

// max |M - M^T| and max |M - I| of an Np x Np matrix
__global__ void k_sym_err(const double* const* M, const int* Np, double* out) {
    const int e = blockIdx.x;
    const int n = Np[e];
    const double* A = M[e];
    __shared__ double s0[32], s1[32];
    double a = 0.0, b = 0.0;
    for (long idx = threadIdx.x; idx < (long)n * n; idx += blockDim.x) {
        const int i = (int)(idx % n), j = (int)(idx / n);
        a = fmax(a, fabs(A[idx] - A[j + (size_t)i * n]));
        b = fmax(b, fabs(A[idx] - (i == j ? 1.0 : 0.0)));
    }
    for (int o = 16; o > 0; o >>= 1) {
        a = fmax(a, __shfl_down_sync(0xffffffffu, a, o));
        b = fmax(b, __shfl_down_sync(0xffffffffu, b, o));
    }
    if ((threadIdx.x & 31) == 0) { s0[threadIdx.x >> 5] = a; s1[threadIdx.x >> 5] = b; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) { a = fmax(a, s0[i]); b = fmax(b, s1[i]); }
        out[2 * e] = a;
        out[2 * e + 1] = b;
    }
}

// Q = [[A, B], [-B, A]]  (real form of A - iB; (A - iB)^-1 = X + iY with [X; Y] = Q^-1 [I; 0])
__global__ void k_embed(const double* const* A, const double* const* B, double* const* Q, const int* Np) {
    const int e = blockIdx.y;
    const int n = Np[e], n2 = 2 * n;
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < (long)n2 * n2;
         idx += (long)gridDim.x * blockDim.x) {
        const int i = (int)(idx % n2), j = (int)(idx / n2);
        const int bi = i / n, bj = j / n, ii = i % n, jj = j % n;
        const double a = A[e][ii + (size_t)jj * n], b = B[e][ii + (size_t)jj * n];
        double v;
        if (bi == bj) v = a;
        else if (bi == 0) v = b;
        else v = -b;
        Q[e][idx] = v;
    }
}

// Dipole finalisation (DipoleMatrixElement.cpp:920-947):
//   M = ((A - iB)^-1)^dagger = X^T - i Y^T, D_raw = M d_raw, o = M b,
//   D = D_raw - sum_alpha N_alpha o_alpha d_corr(alpha)
struct DmeEntry {
    const double* Qinv;   // 2Np x 2Np
    const double* dall;   // K x Np (ld K): rows 0..5 d_raw per slot, 6.. overlap rows
    const double* dcorr;  // [alpha][slot]
    const double* spin;   // n_occ
    double* Dre; double* Dim; double* Drre; double* Drim; double* ore; double* oim;
    int Np, K, n_occ;
};

__global__ void k_dme_o(const DmeEntry* __restrict__ ents) {
    const DmeEntry d = ents[blockIdx.y];
    const int n = d.Np, n2 = 2 * n;
    const int tot = n * (N_SLOTS + d.n_occ);
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < tot; idx += gridDim.x * blockDim.x) {
        const int mu = idx % n, row = idx / n;
        double re = 0.0, im = 0.0;
        for (int b = 0; b < n; ++b) {
            const double v = d.dall[row + (size_t)b * d.K];
            re += d.Qinv[b + (size_t)mu * n2] * v;          // X(b, mu)
            im -= d.Qinv[(n + b) + (size_t)mu * n2] * v;    // -Y(b, mu)
        }
        if (row < N_SLOTS) { d.Drre[row * n + mu] = re; d.Drim[row * n + mu] = im; }
        else { d.ore[(row - N_SLOTS) * n + mu] = re; d.oim[(row - N_SLOTS) * n + mu] = im; }
    }
}

__global__ void k_dme_D(const DmeEntry* __restrict__ ents, int orthogonalize) {
    const DmeEntry d = ents[blockIdx.y];
    const int n = d.Np;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n * N_SLOTS; idx += gridDim.x * blockDim.x) {
        const int mu = idx % n, s = idx / n;
        double sre = 0.0, sim = 0.0;
        if (orthogonalize) {
            for (int a = 0; a < d.n_occ; ++a) {
                const double w = d.spin[a] * d.dcorr[a * N_SLOTS + s];
                sre += d.ore[a * n + mu] * w;
                sim += d.oim[a * n + mu] * w;
            }
        }
        d.Dre[s * n + mu] = d.Drre[s * n + mu] - sre;
        d.Dim[s * n + mu] = d.Drim[s * n + mu] - sim;
    }
}

// ---- dipole rows C_n and d_correction (energy independent)
struct CtabArgs {
    int n_pts, Np, Kr, n_lambda, n_occ;
    double dr;
    const double* w;          // Simpson weights
    const double* chi_init;   // [n][nu]
    const double* dchi;       // [n][nu]
    const double* chi;        // [n][lambda][i] (n < n_tr)
    const int* l_of_nu;
    const int* dptr[3];
    const int* dnu[3];
    const double* da[3];
    const double* dc[3];
    double* C;                // [n][K x Np]
    double* part;             // [n][alpha][slot] for d_correction
};

__global__ void k_ctab(CtabArgs a) {
    const int n = blockIdx.x;
    if (n >= a.n_pts) return;
    const double r = a.dr + n * a.dr;                 // r_min + ir dr, r_min = dr
    const double inv_r = (r > 1e-30) ? 1.0 / r : 0.0;
    const double w = a.w[n];
    __shared__ double part[64 * N_SLOTS];
    for (int i = threadIdx.x; i < a.n_occ * N_SLOTS; i += blockDim.x) part[i] = 0.0;
    __syncthreads();
    double* Cn = a.C + (size_t)n * a.Kr * a.Np;
    const double* ci = a.chi_init + (size_t)n * a.n_lambda;
    const double* di = a.dchi + (size_t)n * a.n_lambda;
    for (int mu = threadIdx.x; mu < a.Np; mu += blockDim.x) {
        double xi[N_SLOTS];
        for (int q = 0; q < 3; ++q) {
            double sL = 0.0, sV = 0.0;
            for (int k = a.dptr[q][mu]; k < a.dptr[q][mu + 1]; ++k) {
                const int nu = a.dnu[q][k];
                const double av = a.da[q][k];
                const double c = a.dc[q][k];
                sL += av * ci[nu];
                sV += av * (di[nu] + c * inv_r * ci[nu]);
            }
            xi[q] = sL;
            xi[3 + q] = sV;
        }
        for (int s = 0; s < N_SLOTS; ++s) {
            const double rfac = (s < 3) ? r : 1.0;
            Cn[s + (size_t)mu * a.Kr] = w * (rfac * xi[s]);
        }
        for (int al = 0; al < a.n_occ; ++al) {
            // phi_alpha(n, mu) = chi(n, lambda = mu, alpha), mu < min(Np, n_lambda)
            const double phi = (mu < a.n_lambda) ? a.chi[((size_t)n * a.n_lambda + mu) * a.n_occ + al] : 0.0;
            Cn[(N_SLOTS + al) + (size_t)mu * a.Kr] = w * phi;
            for (int s = 0; s < N_SLOTS; ++s) atomicAdd(&part[al * N_SLOTS + s], phi * xi[s]);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < a.n_occ * N_SLOTS; i += blockDim.x) {
        const int s = i % N_SLOTS;
        const double rfac = (s < 3) ? r : 1.0;
        a.part[(size_t)n * a.n_occ * N_SLOTS + i] = w * (rfac * part[i]);
    }
}

// -M_A = h^2/6 V (n) sub-block, for the stability eigenvalues
__global__ void k_neg_hV(const double* V, int ldV, double h2_6, double* out, int Np) {
    const long total = (long)Np * Np;
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
         idx += (long)gridDim.x * blockDim.x) {
        const int i = (int)(idx % Np), j = (int)(idx / Np);
        out[idx] = -(h2_6 * V[i + (size_t)j * ldV]);
    }
}

}  // namespace

// ================================================================ host side

namespace {

template <class T>
int upload_vec(DevBuf<T>& d, const std::vector<T>& h, cudaStream_t s) {
    SCATT_TRY(d.alloc(h.size()));
    if (!h.empty()) SCATT_CUDA_TRY(cudaMemcpyAsync(d.p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, s));
    return SCATT_OK;
}

// batched GEMM / GJ helpers for the (non-hot) post stages: entries staged
// through a small device scratch array.  Nothing waits for the device: the
// entries are copied from pageable memory (staged before the call returns)
// and the scratch arrays are reused in stream order.
struct Launcher {
    cudaStream_t s;
    DevBuf<GemmEntry> ge;
    DevBuf<GjEntry> je;
    DevBuf<CopyEntry> ce;
    int gemm(const std::vector<GemmEntry>& v, int opA, int opB) {
        if (v.empty()) return SCATT_OK;
        int mM = 0, mN = 0;
        for (auto& e : v) { mM = std::max(mM, e.M); mN = std::max(mN, e.N); }
        if (ge.n < v.size()) SCATT_TRY(ge.alloc(v.size()));
        SCATT_CUDA_TRY(cudaMemcpyAsync(ge.p, v.data(), v.size() * sizeof(GemmEntry), cudaMemcpyHostToDevice, s));
        return gemm_batched(ge.p, (int)v.size(), mM, mN, opA, opB, s);
    }
    DevBuf<double> gp;   // panel windows of the two-level inverses
    DevBuf<int> gs;
    int gj(const std::vector<GjEntry>& v, bool sym) {
        if (v.empty()) return SCATT_OK;
        int mn = 0;
        for (auto& e : v) mn = std::max(mn, e.n);
        if (je.n < v.size()) SCATT_TRY(je.alloc(v.size()));
        // the two-level inverses by the automatic rule's order, 64-column windows, no look-ahead
        size_t pd = 0, si = 0;
        for (auto& e : v) { pd += 2 * (size_t)e.ld * 64; si += 2 * (size_t)e.n; }
        if (gp.n < pd) SCATT_TRY(gp.alloc(pd));
        if (gs.n < si) SCATT_TRY(gs.alloc(si));
        std::vector<GjEntry> w(v);
        pd = si = 0;
        for (auto& e : w) {
            e.P = gp.p + pd;
            e.sigt = gs.p + si;
            pd += 2 * (size_t)e.ld * 64;
            si += 2 * (size_t)e.n;
        }
        SCATT_CUDA_TRY(cudaMemcpyAsync(je.p, w.data(), w.size() * sizeof(GjEntry), cudaMemcpyHostToDevice, s));
        return mn > 512 ? gj_inverse_batched3(je.p, (int)w.size(), mn, sym, s, false, -1, 64)
                        : gj_inverse_batched2(je.p, (int)w.size(), mn, sym, s);
    }
    int copy(const std::vector<CopyEntry>& v) {
        if (v.empty()) return SCATT_OK;
        if (ce.n < v.size()) SCATT_TRY(ce.alloc(v.size()));
        SCATT_CUDA_TRY(cudaMemcpyAsync(ce.p, v.data(), v.size() * sizeof(CopyEntry), cudaMemcpyHostToDevice, s));
        k_copy<<<dim3(64, (unsigned)v.size()), TPB, 0, s>>>(ce.p);
        SCATT_COUNT_LAUNCH(1);
        return SCATT_CUDA_TRY_RET(cudaGetLastError());
    }
};

}  // namespace

// ---------------------------------------------------------------- static upload
int upload_static(Context& ctx, const scatt_scan_desc& D) {
    if (D.Nr < 8 || !(D.dr > 0.0) || D.l_cont_max < 0 || D.n_occ < 1 || D.n_orb < D.n_occ ||
        D.Nlm_store < 1 || D.Nr_store < 1 || D.Nr_store > D.Nr || !D.psi_lm || (D.n_H > 0 && !D.V_H) ||
        (D.n_atoms > 0 && !D.atoms)) {
        set_last_error("scatt_upload_static: invalid scan description");
        return SCATT_ERR_ARG;
    }
    if (D.n_occ > 64) {
        set_last_error("scatt_upload_static: n_occ > 64 is beyond the exchange kernel's register budget");
        return SCATT_ERR_SIZE;
    }
    SCATT_TRY(require_device());
    SCATT_CUDA_TRY(cudaSetDevice(ctx.device));
    cudaStream_t s = ctx.stream;
    auto T = std::make_unique<ScanTables>();
    ScanTables& t = *T;
    t.Nr = D.Nr;
    t.dr = D.dr;
    t.l_max = D.l_cont_max;
    t.l_x = std::min(D.l_cont_max, 10);
    t.n_sigma = (t.l_x + 1) * (t.l_x + 1);
    t.n_occ = D.n_occ;
    t.Np_max = (t.l_max + 1) * (t.l_max + 1);
    t.n_lambda = (t.l_max + t.l_x + 1) * (t.l_max + t.l_x + 1);
    t.Nf = t.n_occ * t.n_sigma;
    t.n_exp = (2 * t.l_max + 1) * (2 * t.l_max + 1);
    t.alpha_pol = D.alpha_pol;
    t.pol_form = D.pol_form;
    t.r_c = D.r_c > 0.0 ? D.r_c : 1.5;
    // ---- n_transition (WavefunctionSetup.cpp:278-324)
    if (D.n_transition > 0) {
        t.n_tr = std::min(D.n_transition, D.Nr);
    } else {
        const double cut = D.chi_cutoff > 0.0 ? D.chi_cutoff : 1e-15;
        const int nlam = std::min(t.n_lambda, D.Nlm_store);
        int last = 0;
        for (int ir = D.Nr_store - 1; ir >= 0 && last == 0; --ir) {
            double mx = 0.0;
            for (int j = 0; j < D.n_occ; ++j)
                for (int lam = 0; lam < nlam; ++lam)
                    mx = std::max(mx, std::abs(D.psi_lm[((size_t)j * D.Nlm_store + lam) * D.Nr_store + ir]));
            if (mx > cut) { last = ir; break; }
        }
        const int buffer = std::max(100, (int)(5.0 / D.dr));
        t.n_tr = std::min({D.Nr, D.Nr_store, last + 1 + buffer});
        if (t.n_tr < 1) t.n_tr = 1;
    }
    // ---- potential tables
    std::vector<double> vs = build_vsigma(D.Nr, D.dr, t.l_max, D.n_H, D.V_H, D.n_atoms, D.atoms);
    SCATT_TRY(upload_vec(t.vsig, vs, s));
    PairCSR P = build_gaunt_pairs(t.l_max);
    t.n_pairs = (int)P.row.size();
    SCATT_TRY(upload_vec(t.pair_row, P.row, s));
    SCATT_TRY(upload_vec(t.pair_col, P.col, s));
    SCATT_TRY(upload_vec(t.pair_ptr, P.ptr, s));
    SCATT_TRY(upload_vec(t.pair_sig, P.sig, s));
    SCATT_TRY(upload_vec(t.pair_G, P.G, s));
    // ---- exchange CSR (G_combined rows mu*n_sigma + sigma)
    ExchCSR X = build_exchange(t.Np_max, t.n_sigma, t.n_lambda);
    t.n_lambda_ex = X.n_lambda_max;
    SCATT_TRY(upload_vec(t.ex_ptr, X.ptr, s));
    SCATT_TRY(upload_vec(t.ex_lam, X.lam, s));
    SCATT_TRY(upload_vec(t.ex_G, X.G, s));
    // ---- chi[n][lambda][i] = (n dr) psi_lm (WavefunctionSetup.cpp:196-204)
    const int nl = std::min(t.n_lambda, D.Nlm_store);
    {
        std::vector<double> chi((size_t)t.n_tr * t.n_lambda * t.n_occ, 0.0);
        for (int n = 0; n < std::min(t.n_tr, D.Nr_store); ++n) {
            const double r = n * D.dr;
            for (int lam = 0; lam < nl; ++lam)
                for (int i = 0; i < t.n_occ; ++i)
                    chi[((size_t)n * t.n_lambda + lam) * t.n_occ + i] =
                        r * D.psi_lm[((size_t)i * D.Nlm_store + lam) * D.Nr_store + n];
        }
        SCATT_TRY(upload_vec(t.chi, chi, s));
    }
    // ---- initial state, its derivative, dipole rows (main.cpp:767-822, DipoleMatrixElement.cpp:49-233)
    const int init = D.init_state >= 0 ? D.init_state : D.n_occ - 1;
    if (init >= D.n_orb) {
        set_last_error("scatt_upload_static: init_state beyond the stored orbitals");
        return SCATT_ERR_ARG;
    }
    std::vector<double> chi_init((size_t)D.Nr * t.n_lambda, 0.0), dchi((size_t)D.Nr * t.n_lambda, 0.0);
    {
        const int ntake = std::min(t.n_tr, D.Nr_store);
        for (int n = 0; n < ntake; ++n) {
            const double r = n * D.dr;
            for (int lam = 0; lam < nl; ++lam)
                chi_init[(size_t)n * t.n_lambda + lam] = r * D.psi_lm[((size_t)init * D.Nlm_store + lam) * D.Nr_store + n];
        }
        std::vector<double> f(D.Nr), df(D.Nr);
        for (int lam = 0; lam < t.n_lambda; ++lam) {
            for (int n = 0; n < D.Nr; ++n) f[n] = chi_init[(size_t)n * t.n_lambda + lam];
            five_point_derivative(f.data(), D.Nr, D.dr, df.data());
            for (int n = 0; n < D.Nr; ++n) dchi[(size_t)n * t.n_lambda + lam] = df[n];
        }
    }
    const int n_keep_hi = std::min(D.Nr - 1, std::max(1, t.n_tr - 1));
    const int n_pts = std::min(D.Nr, n_keep_hi + 1);
    if (n_pts < 5) {
        set_last_error("DipoleMatrixElement: too few radial points for integration");
        return SCATT_ERR_ARG;
    }
    std::vector<double> w = simpson_weights(n_pts, D.dr);
    DipCSR Dt = build_dipole_tables(t.Np_max, t.n_lambda);
    t.Krows = N_SLOTS + t.n_occ;
    {
        DevBuf<double> dw, dci, ddc, dpart;
        DevBuf<int> dl, dptr[3], dnu[3];
        DevBuf<double> da[3], dc[3];
        SCATT_TRY(upload_vec(dw, w, s));
        SCATT_TRY(upload_vec(dci, chi_init, s));
        SCATT_TRY(upload_vec(ddc, dchi, s));
        CtabArgs a{};
        for (int q = 0; q < 3; ++q) {
            SCATT_TRY(upload_vec(dptr[q], Dt.ptr[q], s));
            SCATT_TRY(upload_vec(dnu[q], Dt.nu[q].empty() ? std::vector<int>{0} : Dt.nu[q], s));
            SCATT_TRY(upload_vec(da[q], Dt.a[q].empty() ? std::vector<double>{0.0} : Dt.a[q], s));
            SCATT_TRY(upload_vec(dc[q], Dt.c[q].empty() ? std::vector<double>{0.0} : Dt.c[q], s));
            a.dptr[q] = dptr[q].p; a.dnu[q] = dnu[q].p; a.da[q] = da[q].p; a.dc[q] = dc[q].p;
        }
        SCATT_TRY(t.Ctab.alloc((size_t)n_pts * t.Krows * t.Np_max));
        SCATT_TRY(dpart.alloc((size_t)n_pts * t.n_occ * N_SLOTS));
        a.n_pts = n_pts; a.Np = t.Np_max; a.Kr = t.Krows; a.n_lambda = t.n_lambda; a.n_occ = t.n_occ;
        a.dr = D.dr; a.w = dw.p; a.chi_init = dci.p; a.dchi = ddc.p; a.chi = t.chi.p;
        a.C = t.Ctab.p; a.part = dpart.p;
        k_ctab<<<n_pts, TPB, 0, s>>>(a);
        SCATT_COUNT_LAUNCH(1);
        SCATT_CUDA_TRY(cudaGetLastError());
        std::vector<double> part((size_t)n_pts * t.n_occ * N_SLOTS);
        SCATT_CUDA_TRY(cudaMemcpyAsync(part.data(), dpart.p, part.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
        SCATT_CUDA_TRY(cudaStreamSynchronize(s));
        t.d_corr.assign((size_t)t.n_occ * N_SLOTS, 0.0);
        for (int n = 0; n < n_pts; ++n)
            for (int i = 0; i < t.n_occ * N_SLOTS; ++i) t.d_corr[i] += part[(size_t)n * t.n_occ * N_SLOTS + i];
    }
    t.spin.assign(t.n_occ, 2.0);
    t.l_of_mu.resize(t.Np_max);
    for (int m = 0; m < t.Np_max; ++m) t.l_of_mu[m] = l_of(m);
    SCATT_TRY(upload_vec(t.d_l_of_mu, t.l_of_mu, s));
    std::vector<int> ls(t.n_sigma);
    for (int m = 0; m < t.n_sigma; ++m) ls[m] = l_of(m);
    SCATT_TRY(upload_vec(t.d_l_sigma, ls, s));
    SCATT_CUDA_TRY(cudaStreamSynchronize(s));
    t.ready = true;
    ctx.tab = std::move(T);
    return SCATT_OK;
}

namespace {

// ---------------------------------------------------------------- scan constants
// Grid rules shared by every energy of a scan (SolverParams, the fit window,
// n_start), with the static tables' device pointers.
int make_consts(const ScanTables& t, const scatt_solve_opts& o, BatchDev& b) {
    b.Nr = t.Nr;
    b.N = t.Nr - 1;
    b.n_stop = t.Nr;
    b.n_tr = t.n_tr;
    const int n_keep_hi = std::min(t.Nr - 1, std::max(1, t.n_tr - 1));
    b.n_pts = std::min(t.Nr, n_keep_hi + 1);
    {
        const int lmf = t.l_x;
        const double r_crit = t.dr * std::sqrt((double)(lmf * (lmf + 1)) / 12.0);
        int ns = std::max(1, (int)std::ceil(2.0 * r_crit / t.dr));
        b.n_start = std::min(ns, t.Nr - 1);
    }
    {
        const int Nr = t.Nr, N = Nr - 1;
        int nsf = std::max(Nr - 200, (int)(0.9 * Nr));
        int nef = Nr - 1 - 3;
        const int lo = N - std::max(0, o.n_asym) + 1;
        nsf = std::max(nsf, lo);
        nef = std::min(nef, N);
        if (nef - nsf + 1 < 10) {
            set_last_error("AsymptoticAmplitudes: fit window is too small (" + std::to_string(nef - nsf + 1) +
                           " points)");
            return SCATT_ERR_FIT_WINDOW;
        }
        b.n_s = nsf;
        b.ne_fit = nef;
        b.nfit = nef - nsf + 1;
    }
    b.stab_n = std::min(o.stab_n_max, t.Nr);
    b.Np_max = t.Np_max;
    b.Nf = t.Nf;
    b.n_sigma = t.n_sigma;
    b.n_occ = t.n_occ;
    b.Krows = t.Krows;
    b.n_lambda = t.n_lambda;
    b.n_lambda_ex = t.n_lambda_ex;
    b.dr = t.dr;
    b.h2_6 = t.dr * t.dr / 6.0;
    b.h2_12 = t.dr * t.dr / 12.0;
    b.W_min = o.W_min;
    b.margin = o.shift_margin;
    b.alpha_pol = t.alpha_pol;
    b.r_c = t.r_c;
    b.pol_form = t.pol_form;
    b.dV = t.dV;
    b.vsig = t.vsig.p;
    b.n_exp = t.n_exp;
    b.n_pairs = t.n_pairs;
    b.pair_row = t.pair_row.p; b.pair_col = t.pair_col.p; b.pair_ptr = t.pair_ptr.p;
    b.pair_sig = t.pair_sig.p; b.pair_G = t.pair_G.p;
    b.ex_ptr = t.ex_ptr.p; b.ex_lam = t.ex_lam.p; b.ex_G = t.ex_G.p;
    b.chi = t.chi.p;
    b.Ctab = t.Ctab.p;
    b.l_of_mu = t.d_l_of_mu.p;
    b.l_sigma = t.d_l_sigma.p;
    return SCATT_OK;
}

// V(n), B(n), Bs(n), D^-1(n) into one set of buffers (post stages, setup).
struct VBAt {
    DevBuf<double> V, B, Bs, Dinv;
    int alloc(const BatchDev& b) {
        SCATT_TRY(V.alloc((size_t)b.Np_max * b.Np_max));
        SCATT_TRY(B.alloc((size_t)b.Np_max * std::max(1, b.Nf)));
        SCATT_TRY(Bs.alloc((size_t)b.Np_max * std::max(1, b.Nf)));
        SCATT_TRY(Dinv.alloc(std::max(1, b.Nf)));
        return SCATT_OK;
    }
    void build(const BatchDev& b, int n, cudaStream_t s) {
        k_build_V_at<<<cdiv(b.n_pairs, TPB), TPB, 0, s>>>(b, n, V.p);
        SCATT_COUNT_LAUNCH(1);
        const int rows = std::max(b.Np_max * b.n_sigma, b.Nf);
        k_build_B_at<<<cdiv(rows, 128), 128, 0, s>>>(b, n, B.p, Bs.p, Dinv.p);
        SCATT_COUNT_LAUNCH(1);
    }
};

// lambda_min(-h^2/6 V(n)) and lambda_min(-h^2/6 V(n) - Bs B^T) for n < stab_n (per Np)
int ensure_stab(Context& ctx, const scatt_solve_opts& o, int l_cont, const double** lmA, const double** lmS,
                std::vector<DevBuf<double>>& keep) {
    ScanTables& t = *ctx.tab;
    cudaStream_t s = ctx.stream;
    for (auto& se : t.stab)
        if (se.l_cont == l_cont && (int)se.lmA.size() >= std::min(o.stab_n_max, t.Nr)) {
            keep.emplace_back();
            SCATT_TRY(upload_vec(keep.back(), se.lmA, s));
            *lmA = keep.back().p;
            keep.emplace_back();
            SCATT_TRY(upload_vec(keep.back(), se.lmS, s));
            *lmS = keep.back().p;
            return SCATT_OK;
        }
    BatchDev b{};
    SCATT_TRY(make_consts(t, o, b));
    const int Np = (l_cont + 1) * (l_cont + 1);
    const int ns = std::min(o.stab_n_max, t.Nr);
    std::vector<double> lA(std::max(ns, 1), 0.0), lS(std::max(ns, 1), 0.0);
    if (ns > 0) {
        VBAt vb;
        SCATT_TRY(vb.alloc(b));
        DevBuf<double> MA, MS, d, e, wk, outA, outS;
        SCATT_TRY(MA.alloc((size_t)ns * Np * Np));
        SCATT_TRY(MS.alloc((size_t)ns * Np * Np));
        SCATT_TRY(d.alloc((size_t)2 * ns * Np));
        SCATT_TRY(e.alloc((size_t)2 * ns * Np));
        SCATT_TRY(wk.alloc((size_t)4 * ns * Np));
        SCATT_TRY(outA.alloc(ns));
        SCATT_TRY(outS.alloc(ns));
        Launcher L{s};
        for (int n = 0; n < ns; ++n) {
            vb.build(b, n, s);
            k_neg_hV<<<64, TPB, 0, s>>>(vb.V.p, t.Np_max, b.h2_6, MA.p + (size_t)n * Np * Np, Np);
            SCATT_COUNT_LAUNCH(1);
            SCATT_CUDA_TRY(cudaMemcpyAsync(MS.p + (size_t)n * Np * Np, MA.p + (size_t)n * Np * Np,
                                           (size_t)Np * Np * sizeof(double), cudaMemcpyDeviceToDevice, s));
            if (n < t.n_tr && t.Nf > 0) {
                std::vector<GemmEntry> g{GemmEntry{vb.Bs.p, vb.B.p, MS.p + (size_t)n * Np * Np, Np, Np, t.Nf,
                                                   t.Np_max, t.Np_max, Np, -1.0, 1.0}};
                SCATT_TRY(L.gemm(g, 0, 1));
            }
        }
        std::vector<EigEntry> ee;
        for (int n = 0; n < ns; ++n) {
            ee.push_back(EigEntry{MA.p + (size_t)n * Np * Np, Np, Np, d.p + (size_t)(2 * n) * Np,
                                  e.p + (size_t)(2 * n) * Np, wk.p + (size_t)(4 * n) * Np, outA.p + n});
            ee.push_back(EigEntry{MS.p + (size_t)n * Np * Np, Np, Np, d.p + (size_t)(2 * n + 1) * Np,
                                  e.p + (size_t)(2 * n + 1) * Np, wk.p + (size_t)(4 * n + 2) * Np, outS.p + n});
        }
        DevBuf<EigEntry> de;
        SCATT_TRY(upload_vec(de, ee, s));
        SCATT_TRY(sym_eigvals_batched(de.p, (int)ee.size(), Np, 1, s));
        SCATT_CUDA_TRY(cudaMemcpyAsync(lA.data(), outA.p, ns * sizeof(double), cudaMemcpyDeviceToHost, s));
        SCATT_CUDA_TRY(cudaMemcpyAsync(lS.data(), outS.p, ns * sizeof(double), cudaMemcpyDeviceToHost, s));
        SCATT_CUDA_TRY(cudaStreamSynchronize(s));
    }
    t.stab.push_back(ScanTables::StabEig{l_cont, lA, lS});
    keep.emplace_back();
    SCATT_TRY(upload_vec(keep.back(), lA, s));
    *lmA = keep.back().p;
    keep.emplace_back();
    SCATT_TRY(upload_vec(keep.back(), lS, s));
    *lmS = keep.back().p;
    return SCATT_OK;
}

// Doubles of the panel buffers of one inverse of order n: the Gauss-Jordan
// windows (four, with the look-ahead) or the symmetric sweep's P, M and D.
// (in slots that may take it, N_t above one tile).
size_t panel_doubles(int n, int Nt) {
    return std::max((size_t)4 * GJ_WINDOW_MAX * n, Nt > SYM_NB ? sym_panel_doubles(n) : 0);
}
// Doubles of its work buffer: n x n for the Gauss-Jordan, or the sweep's tiles.
size_t work_doubles(int n, int Nt) { return std::max((size_t)n * n, Nt > SYM_NB ? sym_work_doubles(n) : 0); }

// Device doubles of one slot sized for (Np, Nt): the chunk's Schur slots,
// the W^-1 blocks, the R ping-pong buffers, the dipole rows, the asymptotic
// window store and the inverse's panel windows (every piece 256-byte aligned).
// Without the window store (keep_window = 0) the fit is accumulated
// forward instead: 2 x (2 Np x N_t) accumulators, the fit weights and the
// per-l normal matrices replace (N - n_s + 1) x (N_t^2 + 2 Np^2).
size_t slot_doubles(const BatchDev& b, int Np, int Nt, int l_cont, bool keep_window) {
    const int nslots = b.N - b.n_s + 1;
    auto al = [](size_t c) { return (c + 31) & ~size_t(31); };
    const size_t np2 = (size_t)Np * Np, nt2 = (size_t)Nt * Nt;
    const size_t base = 2 * al(SCHUR_CHUNK * np2) + al(SCHUR_CHUNK * al(work_doubles(Np, Nt))) +
                        al((size_t)Np * b.Nf) + al((size_t)b.Nf * b.Nf) + 3 * al(nt2) + al(work_doubles(Nt, Nt)) +
                        2 * al((size_t)b.Krows * Nt) + al(SCHUR_CHUNK * al(panel_doubles(Np, Nt))) +
                        al(panel_doubles(Nt, Nt));
    if (keep_window) return base + al((size_t)nslots * nt2) + 2 * al((size_t)nslots * np2);
    return base + 2 * al((size_t)2 * Np * Nt) + al((size_t)b.nfit * 2 * Np) + al((size_t)8 * (l_cont + 1));
}
size_t slot_ints(int Np, int Nt) { return SCHUR_CHUNK * (6 * (size_t)Np + 8) + 6 * (size_t)Nt; }
// Device doubles of one group's chunk arrays (V, B, Bs, D^-1 of SCHUR_CHUNK steps, V(n+1) diagonal).
size_t group_doubles(const BatchDev& b) {
    auto al = [](size_t c) { return (c + 31) & ~size_t(31); };
    const size_t sl = (size_t)b.Np_max * std::max(1, b.Nf);
    return al(SCHUR_CHUNK * (size_t)b.Np_max * b.Np_max) + 2 * al(SCHUR_CHUNK * sl) +
           al(SCHUR_CHUNK * (size_t)std::max(1, b.Nf)) + al(b.Np_max);
}
// Device doubles of one energy's post-stage buffers.
size_t post_doubles(const BatchDev& b, int Np, int Nt, int l_cont, int nfit, int n_occ) {
    const size_t np2 = (size_t)Np * Np;
    return 6 * Np + 14 * np2 + (size_t)b.Nf * Np + 2 * (size_t)Nt * Np + 12 * np2 +
           2 * (size_t)(l_cont + 1) * nfit + 8 * (size_t)(l_cont + 1) + 2 * np2 + (size_t)b.Krows * Np +
           24 * (size_t)Np + 2 * (size_t)n_occ * Np + 8 * (size_t)Np + 2 * np2 + 48 * 32;   // 48 >= the pieces, each rounded up
}
// ---------------------------------------------------------------- scan
struct PostBufs {        // per-energy post-processing buffers
    double *tab, *Amat, *Bmat, *Bw, *Binv, *Kraw, *K, *psibc, *VP, *Bf, *fN, *Z0, *Z1, *rhs;
    double *Q, *Qw, *Qinv, *aatab, *aaM, *aared, *Aaa, *Baa, *Aw, *Ainv, *Kc, *dall;
    double *Dre, *Dim, *Drre, *Drim, *ore, *oim, *ew_d, *ew_e, *ew_w, *eigK, *eigA;
    int *sig, *rid, *st;
};

struct Job {
    double E;
    int l_cont;
    long index;       // submission index
};

// CUDA events created once per scan and destroyed with it, so no early
// return leaks one.
struct EventPool {
    std::vector<cudaEvent_t> ev;
    size_t used = 0;
    ~EventPool() {
        for (auto e : ev) cudaEventDestroy(e);
    }
    int get(cudaEvent_t* out) {
        if (used == ev.size()) {
            cudaEvent_t e;
            SCATT_CUDA_TRY(cudaEventCreate(&e));
            ev.push_back(e);
        }
        *out = ev[used++];
        return SCATT_OK;
    }
    void reset() { used = 0; }
};

}  // namespace

// A scan: `slots` energies in flight in `ngroups` phase groups; energies
// wait in a queue and enter a group whenever the group is free.
struct Scan {
    Context* ctx = nullptr;
    scatt_solve_opts o{};
    BatchDev b{};
    int slots = 0, G = 1, gs = 1;
    int l_cap = 0, Np_cap = 0, Nt_cap = 0;
    int chunks_per_sweep = 0;
    bool general = false;               // S and R by the general inverse under the automatic scheme too
    std::vector<EnergyDev> ed;          // host copy of the slot state (pointers fixed at open)
    std::vector<GroupDev> grp;          // host mirror of the group state
    std::vector<long> job_of;           // submission index held by each slot (-1 empty)
    std::vector<long> start_chunk;      // first chunk at which each idle group may start
    std::deque<Job> queue;
    long chunk = 0;
    long submitted = 0;
    DevBuf<EnergyDev> d_ed;
    DevBuf<GroupDev> d_grp;
    DevBuf<double> arena, garena, parena;
    DevBuf<int> iarena, pia;
    DevBuf<GemmEntry> gm;
    DevBuf<GjEntry> gj;
    DevBuf<SymEntry> sy;
    DevBuf<unsigned> stat;
    DevBuf<unsigned> barrier;
    DevBuf<double> scratch;
    DevBuf<RArgs> rargs;
    VBAt vb;                            // V/B at one step for the post stages
    std::vector<PostBufs> P;            // gs energies
    std::vector<DevBuf<double>> keep;   // stability spectra per l_cont
    std::vector<std::pair<int, std::pair<const double*, const double*>>> stab_ptr;
    EventPool events;
    Launcher L{nullptr};
    int nfit = 0, ne_fit = 0;
    struct Graph {
        cudaGraphExec_t exec;
        unsigned long long launches;    // kernels per replay
    };
    std::map<std::pair<uint64_t, int>, Graph> graphs;   // (stage pattern, stop step) -> replay
    Scan() = default;
    Scan(const Scan&) = delete;
    Scan& operator=(const Scan&) = delete;
    ~Scan() {
        for (auto& g : graphs) cudaGraphExecDestroy(g.second.exec);
    }
};

namespace {

int gemm_slots(Scan& sc, GemmEntry* ents, int count, int which, int opA, int opB) {
    const int Np = sc.Np_cap, Nt = sc.Nt_cap, Nf = sc.b.Nf, K = sc.b.Krows;
    int M = 0, N = 0;
    switch (which) {
        case 0: M = Np; N = Np; break;       // S
        case 1: M = Np; N = Nf; break;       // T
        case 2: M = Nf; N = Nf; break;       // F
        case 3: M = K; N = std::max(Np, Nf); break;   // G1 and G2
        case 5: M = K; N = Nt; break;        // G3
        case 6: M = 2 * Np; N = Nt; break;   // GA (the fit accumulation)
    }
    return gemm_batched(ents, count, M, N, opA, opB, sc.ctx->stream);
}

int stab_for(Scan& sc, int l_cont, const double** lmA, const double** lmS) {
    for (auto& p : sc.stab_ptr)
        if (p.first == l_cont) {
            *lmA = p.second.first;
            *lmS = p.second.second;
            return SCATT_OK;
        }
    SCATT_TRY(ensure_stab(*sc.ctx, sc.o, l_cont, lmA, lmS, sc.keep));
    sc.stab_ptr.push_back({l_cont, {*lmA, *lmS}});
    return SCATT_OK;
}

int scan_open(Context& ctx, const scatt_solve_opts& o, int slots, int ngroups, int l_cap, Scan& sc) {
    ScanTables& t = *ctx.tab;
    cudaStream_t s = ctx.stream;
    if (slots < 1 || ngroups < 1 || ngroups > MAX_GROUPS || ngroups > slots || l_cap < 0 || l_cap > t.l_max) {
        set_last_error("scatt_scan_open: need 1 <= groups <= min(slots, " + std::to_string(MAX_GROUPS) +
                       ") and 0 <= l_cont_max <= the uploaded scan's");
        return SCATT_ERR_ARG;
    }
    sc.ctx = &ctx;
    sc.o = o;
    sc.L.s = s;
    BatchDev& b = sc.b;
    SCATT_TRY(make_consts(t, o, b));
    sc.slots = slots;
    sc.G = ngroups;
    sc.gs = (slots + ngroups - 1) / ngroups;
    sc.l_cap = l_cap;
    sc.Np_cap = (l_cap + 1) * (l_cap + 1);
    sc.Nt_cap = sc.Np_cap + b.Nf;
    sc.chunks_per_sweep = (b.N + 1 + SCHUR_CHUNK - 1) / SCHUR_CHUNK;
    sc.ne_fit = std::min(t.Nr - 1 - 3, b.N);
    sc.nfit = sc.ne_fit - b.n_s + 1;
    b.count = slots;
    b.ngroups = ngroups;
    b.sw_stride = (work_doubles(sc.Np_cap, sc.Nt_cap) + 31) & ~size_t(31);
    b.ps_stride = (panel_doubles(sc.Np_cap, sc.Nt_cap) + 31) & ~size_t(31);
    const int K = b.Krows, Nf = b.Nf;
    // ---- slot arena
    const bool keep = o.keep_window != 0;
    const size_t per = slot_doubles(b, sc.Np_cap, sc.Nt_cap, l_cap, keep);
    SCATT_TRY(sc.arena.alloc(per * slots));
    SCATT_TRY(sc.iarena.alloc(slot_ints(sc.Np_cap, sc.Nt_cap) * slots));
    SCATT_CUDA_TRY(cudaMemsetAsync(sc.iarena.p, 0, sc.iarena.n * sizeof(int), s));
    sc.ed.assign(slots, EnergyDev{});
    sc.job_of.assign(slots, -1);
    for (int e = 0; e < slots; ++e) {
        EnergyDev& d = sc.ed[e];
        std::memset(&d, 0, sizeof(d));
        const size_t np2 = (size_t)sc.Np_cap * sc.Np_cap, nt2 = (size_t)sc.Nt_cap * sc.Nt_cap;
        const int nslots = b.N - b.n_s + 1;
        double* p = sc.arena.p + per * e;
        // 256-byte aligned pieces (the inverse kernels copy 16-byte row pairs)
        auto take = [&p](size_t cnt) { double* r = p; p += (cnt + 31) & ~size_t(31); return r; };
        d.S = take(SCHUR_CHUNK * np2);
        d.Sw = take(SCHUR_CHUNK * b.sw_stride);
        d.Sinv = take(SCHUR_CHUNK * np2);
        d.T = take((size_t)sc.Np_cap * Nf);
        d.F = take((size_t)Nf * Nf);
        d.Ra = take(nt2);
        d.Rw = take(work_doubles(sc.Nt_cap, sc.Nt_cap));
        d.Rinv0 = take(nt2);
        d.Rinv1 = take(nt2);
        d.G0 = take((size_t)K * sc.Nt_cap);
        d.G1 = take((size_t)K * sc.Nt_cap);
        if (keep) {
            d.tailR = take((size_t)nslots * nt2);
            d.tailS = take((size_t)nslots * np2);
            d.psiT = take((size_t)nslots * np2);
        } else {
            d.GA0 = take((size_t)2 * sc.Np_cap * sc.Nt_cap);
            d.GA1 = take((size_t)2 * sc.Np_cap * sc.Nt_cap);
            d.wAB = take((size_t)b.nfit * 2 * sc.Np_cap);
            d.Mab = take((size_t)8 * (l_cap + 1));
        }
        d.PS = take(SCHUR_CHUNK * b.ps_stride);
        d.PR = take(panel_doubles(sc.Nt_cap, sc.Nt_cap));
        int* q = sc.iarena.p + slot_ints(sc.Np_cap, sc.Nt_cap) * e;
        const int Np = sc.Np_cap, Nt = sc.Nt_cap;
        d.sigS = q; q += SCHUR_CHUNK * Np;
        d.ridS = q; q += SCHUR_CHUNK * Np;
        d.sigR = q; q += Nt;
        d.ridR = q; q += Nt;
        d.stS = q; q += SCHUR_CHUNK * 4;
        d.stR = q; q += SCHUR_CHUNK * 4;
        d.sgS = q; q += SCHUR_CHUNK * 4 * Np;
        d.sgR = q; q += 4 * Nt;
        d.grp = e / sc.gs;
        d.live = 0;
    }
    SCATT_TRY(upload_vec(sc.d_ed, sc.ed, s));
    b.ed = sc.d_ed.p;
    // ---- group chunk arrays
    const size_t gper = group_doubles(b);
    SCATT_TRY(sc.garena.alloc(gper * ngroups));
    sc.grp.assign(ngroups, GroupDev{});
    for (int g = 0; g < ngroups; ++g) {
        GroupDev& G = sc.grp[g];
        double* p = sc.garena.p + gper * g;
        auto take = [&p](size_t cnt) { double* r = p; p += (cnt + 31) & ~size_t(31); return r; };
        const size_t sl = (size_t)b.Np_max * std::max(1, Nf);
        G.n0 = -1;
        G.C = 0;
        G.Vc = take(SCHUR_CHUNK * (size_t)b.Np_max * b.Np_max);
        G.Bc = take(SCHUR_CHUNK * sl);
        G.Bsc = take(SCHUR_CHUNK * sl);
        G.Dinvc = take(SCHUR_CHUNK * (size_t)std::max(1, Nf));
        G.vdiag1 = take(b.Np_max);
    }
    SCATT_TRY(upload_vec(sc.d_grp, sc.grp, s));
    b.grp = sc.d_grp.p;
    // staggered starts: group g first starts g / G of a sweep after group 0
    sc.start_chunk.assign(ngroups, 0);
    for (int g = 0; g < ngroups; ++g) sc.start_chunk[g] = (long)g * sc.chunks_per_sweep / ngroups;
    // ---- entry arrays
    const size_t all = SCHUR_CHUNK * (size_t)slots;
    SCATT_TRY(sc.gm.alloc(7 * all));
    SCATT_TRY(sc.gj.alloc(2 * all));
    SCATT_TRY(sc.sy.alloc(2 * all));
    b.stat_stride = sym_stat_words(sc.Nt_cap);
    SCATT_TRY(sc.stat.alloc(2 * all * b.stat_stride));
    SCATT_TRY(sc.barrier.alloc(SCHUR_CHUNK + 1));
    SCATT_TRY(sc.scratch.alloc(sym_scratch_doubles(sc.Nt_cap)));      // S and R are rescued one after the other
    b.gmS = sc.gm.p; b.gmT = sc.gm.p + all; b.gmF = sc.gm.p + 2 * all; b.gmG = sc.gm.p + 3 * all;
    b.gmG3 = sc.gm.p + 5 * all; b.gmGA = sc.gm.p + 6 * all;
    b.gjR = sc.gj.p; b.gjS = sc.gj.p + all;
    b.syR = sc.sy.p; b.syS = sc.sy.p + all;
    b.stat = sc.stat.p;
    b.barrier = sc.barrier.p;
    SCATT_TRY(sc.rargs.alloc(all));
    b.rargs = sc.rargs.p;
    // ---- post-stage buffers for one group
    SCATT_TRY(sc.vb.alloc(b));
    {
        const int Np = sc.Np_cap, Nt = sc.Nt_cap;
        const size_t pd = (post_doubles(b, Np, Nt, l_cap, sc.nfit, t.n_occ) + 31) & ~size_t(31);
        SCATT_TRY(sc.parena.alloc(pd * sc.gs));
        SCATT_TRY(sc.pia.alloc((4 * (size_t)Np + 8) * sc.gs));
        sc.P.assign(sc.gs, PostBufs{});
        const size_t np2 = (size_t)Np * Np;
        for (int i = 0; i < sc.gs; ++i) {
            double* p = sc.parena.p + pd * i;
            int* q = sc.pia.p + (4 * (size_t)Np + 8) * i;
            PostBufs& x = sc.P[i];
            // 256-byte aligned pieces, as the inverses need for even orders
            auto take = [&p](size_t cnt) { double* r = p; p += (cnt + 31) & ~size_t(31); return r; };
            x.tab = take(6 * Np);
            x.Amat = take(np2); x.Bmat = take(np2); x.Bw = take(np2); x.Binv = take(np2);
            x.Kraw = take(np2); x.K = take(np2); x.psibc = take(np2); x.VP = take(np2);
            x.Bf = take(np2); x.rhs = take(np2); x.Aaa = take(np2); x.Baa = take(np2);
            x.Aw = take(np2); x.Ainv = take(np2);
            x.fN = take((size_t)Nf * Np);
            x.Z0 = take((size_t)Nt * Np); x.Z1 = take((size_t)Nt * Np);
            x.Q = take(4 * np2); x.Qw = take(4 * np2); x.Qinv = take(4 * np2);
            x.aatab = take(2 * (size_t)(l_cap + 1) * sc.nfit);
            x.aaM = take(8 * (size_t)(l_cap + 1));
            x.aared = take(2 * np2);
            x.dall = take((size_t)K * Np);
            x.Dre = take(6 * (size_t)Np); x.Dim = take(6 * (size_t)Np);
            x.Drre = take(6 * (size_t)Np); x.Drim = take(6 * (size_t)Np);
            x.ore = take((size_t)t.n_occ * Np); x.oim = take((size_t)t.n_occ * Np);
            x.ew_d = take(2 * (size_t)Np); x.ew_e = take(2 * (size_t)Np); x.ew_w = take(2 * (size_t)Np);
            x.eigK = take((size_t)Np); x.eigA = take((size_t)Np);
            x.Kc = take(2 * np2);
            x.sig = q; q += 2 * Np; x.rid = q; q += 2 * Np; x.st = q; q += 8;
        }
    }
    SCATT_CUDA_TRY(cudaStreamSynchronize(s));
    return SCATT_OK;
}

// Moves queued energies into the free slots of group g and starts the group
// at n = 0 (no-op when the queue is empty).
int load_group(Scan& sc, int g) {
    if (sc.queue.empty()) return SCATT_OK;
    cudaStream_t s = sc.ctx->stream;
    const int e0 = g * sc.gs, e1 = std::min(sc.slots, e0 + sc.gs);
    const BatchDev& b = sc.b;
    for (int e = e0; e < e1; ++e) {
        EnergyDev& d = sc.ed[e];
        if (sc.queue.empty()) {
            d.live = 0;
            sc.job_of[e] = -1;
            continue;
        }
        const Job j = sc.queue.front();
        sc.queue.pop_front();
        d.E = j.E;
        d.c = 1.0 + b.h2_6 * j.E;
        d.k = std::sqrt(2.0 * j.E);
        d.l_cont = j.l_cont;
        d.Np = (j.l_cont + 1) * (j.l_cont + 1);
        d.Nt = d.Np + b.Nf;
        d.shiftsA = d.shiftsS = 0;
        d.deltaA = 0.0;
        for (double& x : d.deltaAc) x = 0.0;
        d.err_code = d.err_step = 0;
        d.live = 1;
        SCATT_TRY(stab_for(sc, j.l_cont, &d.lmA, &d.lmS));
        sc.job_of[e] = j.index;
        SCATT_CUDA_TRY(cudaMemsetAsync(d.G0, 0, (size_t)b.Krows * d.Nt * sizeof(double), s));
    }
    // a pageable copy: the host copy may change as soon as the call returns
    SCATT_CUDA_TRY(cudaMemcpyAsync(sc.d_ed.p + e0, sc.ed.data() + e0, (size_t)(e1 - e0) * sizeof(EnergyDev),
                                   cudaMemcpyHostToDevice, s));
    if (sc.o.keep_window == 0 && e1 > e0) {
        // the fit accumulation starts at zero; weights from this energy's k
        for (int e = e0; e < e1; ++e) {
            const EnergyDev& d = sc.ed[e];
            if (!d.live) continue;
            const size_t ga = (size_t)2 * d.Np * d.Nt * sizeof(double);
            SCATT_CUDA_TRY(cudaMemsetAsync(d.GA0, 0, ga, s));
            SCATT_CUDA_TRY(cudaMemsetAsync(d.GA1, 0, ga, s));
        }
        k_ab_normal<<<dim3(cdiv(sc.l_cap + 1, 32), e1 - e0), 32, 0, s>>>(sc.b, e0);
        SCATT_COUNT_LAUNCH(1);
        k_ab_weights<<<dim3(64, e1 - e0), TPB, 0, s>>>(sc.b, e0);
        SCATT_COUNT_LAUNCH(1);
    }
    k_set_group<<<1, 1, 0, s>>>(sc.b, g, 0);
    SCATT_COUNT_LAUNCH(1);
    sc.grp[g].n0 = 0;
    sc.grp[g].C = std::min(SCHUR_CHUNK, b.n_stop);
    return SCATT_OK;
}

struct ChunkTiming {
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> rinv;   // sampled R^-1 inversions
    double flops = 0.0;                                       // n^3 (general schemes: 2 n^3) over their matrices
};

// One chunk of SCHUR_CHUNK radial steps for every running group.  With
// opts.use_graphs the chunk's launches are replayed from a CUDA graph: every
// kernel reads its radial step from the device-resident group state and its
// entries from device-side preparation, so one captured graph serves every
// chunk whose running groups need the same stages at each chunk position.
int run_chunk(Scan& sc, ChunkTiming* tm) {
    BatchDev& b = sc.b;
    cudaStream_t s = sc.ctx->stream;
    const int count = sc.slots, G = sc.G, Nf = b.Nf;
    // what the running groups need at each chunk position (host mirror)
    bool step[SCHUR_CHUNK] = {}, exch[SCHUR_CHUNK] = {}, start[SCHUR_CHUNK] = {}, rinv[SCHUR_CHUNK] = {};
    bool sweep[SCHUR_CHUNK] = {}, pts[SCHUR_CHUNK] = {}, win[SCHUR_CHUNK] = {};
    bool stab = false, stab_x = false, any_exch = false;
    const bool acc = sc.o.keep_window == 0;
    // S and R are symmetric: the automatic scheme takes the symmetric sweep (half the flops, no
    // column of pivots); the forced schemes keep the general inverse
    const bool symmetric = !sc.general && g_inverse_scheme.load(std::memory_order_relaxed) == 0;
    // Slots whose R is one tile stay with the general inverse: the sweep would be one pivot chain, no
    // faster, and its eight-column panels leave a few times the rounding of the general inverse's
    // sixteen (an objective's noise at N_t 64: 1.0e-14 against 1.0e-15).  That is not so of S, near
    // the unit matrix (orders 16 and 49: errors within 5 % of each other), which goes with its R:
    // the general inverse of S of order 49 takes 60 us a chunk longer.
    bool gen = false, sweeps = false;                                    // what the running slots need
    for (int e = 0; e < count; ++e) {
        const EnergyDev& d = sc.ed[e];
        if (d.live && sc.grp[d.grp].n0 >= 0) (symmetric && d.Nt > SYM_NB ? sweeps : gen) = true;
    }
    const int gen_Np = symmetric ? std::min(sc.Np_cap, SYM_NB) : sc.Np_cap;
    const int gen_Nt = symmetric ? std::min(sc.Nt_cap, SYM_NB) : sc.Nt_cap;
    int live_rinv[SCHUR_CHUNK] = {};
    std::vector<int> live_in(G, 0);
    for (int e = 0; e < count; ++e) live_in[sc.ed[e].grp] += sc.ed[e].live;
    for (int g = 0; g < G; ++g) {
        const GroupDev& gr = sc.grp[g];
        if (gr.n0 < 0) continue;
        for (int j = 0; j < gr.C; ++j) {
            const int n = gr.n0 + j;
            step[j] = true;
            const bool x = n < b.n_tr && Nf > 0;
            exch[j] |= x;
            any_exch |= x;
            start[j] |= n < b.n_start;
            if (n >= b.n_start) { rinv[j] = true; live_rinv[j] += live_in[g]; }
            sweep[j] |= n <= b.N - 1;
            pts[j] |= n < b.n_pts && n <= b.N - 1;
            win[j] |= acc && n >= b.n_s && n <= b.N - 1;
            stab |= n < b.stab_n;
            stab_x |= n < b.stab_n && x;
        }
    }
    // one R^-1 call in two chunks is timed (one in 16 under graphs) while every slot takes part
    const bool sample_chunk = tm && rinv[0] && live_rinv[0] == count &&
                              (sc.chunk % (sc.o.use_graphs ? 16 : 2) == 0);
    auto issue = [&]() -> int {
        // ---- Schur complements of the chunk's steps: A(n), S(n) = A - Bs B^T, one batched inverse
        auto run = [&](auto kernel, dim3 grid, int threads, size_t smem, auto... args) -> int {
            SCATT_COUNT_LAUNCH(1);
            return cuda_status(launch_dep(kernel, grid, dim3(threads), smem, s, args...), "run_chunk");
        };
        SCATT_TRY(run(k_build_V, dim3(cdiv(b.n_pairs, TPB), G, SCHUR_CHUNK), TPB, 0, b));
        SCATT_TRY(run(k_build_B, dim3(cdiv(std::max(b.Np_max * b.n_sigma, b.Nf), 128), G, SCHUR_CHUNK), 128, 0, b));
        SCATT_TRY(run(k_init_S, dim3(64, count, SCHUR_CHUNK), TPB, 0, b));
        if (stab) SCATT_TRY(run(k_stab, dim3(count, SCHUR_CHUNK), TPB, 0, b, 0));
        SCATT_TRY(run(k_prepare, dim3(cdiv(count * SCHUR_CHUNK, 128)), 128, 0, b, symmetric));
        if (any_exch) SCATT_TRY(gemm_slots(sc, b.gmS, count * SCHUR_CHUNK, 0, 0, 1));
        if (stab_x) SCATT_TRY(run(k_stab, dim3(count, SCHUR_CHUNK), TPB, 0, b, 1));
        if (sweeps) {
            SCATT_TRY(sym_pack_batched(b.syS, count * SCHUR_CHUNK, sc.Np_cap, s));
            SCATT_TRY(sym_sweep_batched(b.syS, count * SCHUR_CHUNK, sc.Np_cap, s));
            SCATT_TRY(sym_rescue_batched(b.syS, count * SCHUR_CHUNK, b.barrier + SCHUR_CHUNK, sc.scratch.p, s));
        }
        if (gen) SCATT_TRY(gj_inverse_selected(b.gjS, count * SCHUR_CHUNK, gen_Np, true, s, true));
        // ---- the R-ratio recurrence over the chunk's steps
        const dim3 eg(64, count);
        for (int j = 0; j < SCHUR_CHUNK; ++j) {
            if (!step[j]) continue;
            const size_t at = (size_t)j * count;
            if (start[j]) SCATT_TRY(run(k_vdiag, dim3(cdiv(b.Np_max, 128), G), 128, 0, b, j));
            if (exch[j]) {
                SCATT_TRY(gemm_slots(sc, b.gmT + at, count, 1, 0, 0));
                SCATT_TRY(gemm_slots(sc, b.gmF + at, count, 2, 1, 0));
            }
            if (start[j]) {
                SCATT_TRY(run(k_analytic_R, eg, TPB, 0, b, j));
                SCATT_TRY(run(k_analytic_R_diag, dim3(4, count), TPB, 0, b, j));
            }
            if (rinv[j]) {
                if (sweeps) {
                    const int T = sym_tiles_of(sc.Nt_cap), nt = T * (T + 1) / 2;
                    static std::atomic<unsigned long long> done{0};
                    SCATT_TRY(allow_smem(k_assemble_R_tiles, sizeof(SymDiagShared), done));
                    SCATT_TRY(run(k_assemble_R_tiles, dim3(count * nt), SYM_THREADS, sizeof(SymDiagShared), b, j, nt));
                }
                if (gen) SCATT_TRY(run(k_assemble_R, eg, TPB, 0, b, j));
                const bool sample = sample_chunk && j == 0;
                cudaEvent_t a0 = nullptr, a1 = nullptr;
                if (sample) {
                    SCATT_TRY(sc.events.get(&a0));
                    SCATT_TRY(sc.events.get(&a1));
                    SCATT_CUDA_TRY(cudaEventRecord(a0, s));
                }
                if (sweeps) {
                    SCATT_TRY(sym_sweep_batched(b.syR + at, count, sc.Nt_cap, s));
                    SCATT_TRY(sym_rescue_launch(b.syR + at, count, b.barrier + j, sc.scratch.p, RSource{b, j}, s));
                }
                if (gen) SCATT_TRY(gj_inverse_selected(b.gjR + at, count, gen_Nt, true, s, true));
                if (sample) {
                    SCATT_CUDA_TRY(cudaEventRecord(a1, s));
                    tm->rinv.push_back({a0, a1});
                    // order N_t at every step: past n_transition the coupling
                    // carried by Rinv(n-1) keeps R from being block-diagonal
                    for (int e = 0; e < count; ++e) {
                        const double n = sc.ed[e].Nt;
                        tm->flops += (symmetric && sc.ed[e].Nt > SYM_NB ? 1.0 : 2.0) * n * n * n;
                    }
                }
            }
            if (sweep[j]) {
                // C_n Sinv and -C_n T go to different columns of G(n-1)^T: one batch
                if (pts[j]) SCATT_TRY(gemm_slots(sc, b.gmG + 2 * at, exch[j] ? 2 * count : count, 3, 0, 0));
                SCATT_TRY(gemm_slots(sc, b.gmG3 + at, count, 5, 0, 0));
            }
            if (win[j]) {
                SCATT_TRY(run(k_acc_ab, eg, TPB, 0, b, j));
                SCATT_TRY(gemm_slots(sc, b.gmGA + at, count, 6, 0, 0));
            }
        }
        SCATT_TRY(run(k_collect, dim3(cdiv(count, 128)), 128, 0, b));
        SCATT_TRY(run(k_advance, dim3(1), MAX_GROUPS, 0, b));
        return SCATT_CUDA_TRY_RET(cudaGetLastError());
    };
    uint64_t key = (stab ? 1u : 0u) | (stab_x ? 2u : 0u) | (any_exch ? 4u : 0u) | ((uint64_t)gen << 59) |
                   ((uint64_t)sweeps << 60) | ((uint64_t)symmetric << 61);
    for (int j = 0; j < SCHUR_CHUNK; ++j) {
        const uint64_t bits = (step[j] ? 1u : 0u) | (exch[j] ? 2u : 0u) | (start[j] ? 4u : 0u) |
                              (rinv[j] ? 8u : 0u) | (sweep[j] ? 16u : 0u) | (pts[j] ? 32u : 0u) |
                              (win[j] ? 64u : 0u);
        key |= bits << (3 + 7 * j);
    }
    if (sc.o.use_graphs && !sample_chunk && sc.chunk > 0) {
        const auto gk = std::make_pair(key, b.n_stop);
        auto it = sc.graphs.find(gk);
        if (it == sc.graphs.end()) {
            SCATT_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
            const unsigned long long l0 = launch_counter();
            const int st = issue();
            cudaGraph_t g = nullptr;
            const cudaError_t ce = cudaStreamEndCapture(s, &g);
            const unsigned long long nl = launch_counter() - l0;
            launch_counter().fetch_sub(nl);          // captured, not launched
            if (st != SCATT_OK) { if (g) cudaGraphDestroy(g); return st; }
            if (ce != cudaSuccess) { if (g) cudaGraphDestroy(g); return cuda_status(ce, "cudaStreamEndCapture"); }
            cudaGraphExec_t ex = nullptr;
            const cudaError_t ie = cudaGraphInstantiate(&ex, g, 0);
            cudaGraphDestroy(g);
            if (ie != cudaSuccess) return cuda_status(ie, "cudaGraphInstantiate");
            it = sc.graphs.emplace(gk, Scan::Graph{ex, nl}).first;
        }
        SCATT_CUDA_TRY(cudaGraphLaunch(it->second.exec, s));
        SCATT_COUNT_LAUNCH(it->second.launches);
    } else {
        SCATT_TRY(issue());
    }
    for (auto& gr : sc.grp) {
        if (gr.n0 < 0) continue;
        const int n0 = gr.n0 + gr.C;
        if (n0 >= b.n_stop) { gr.n0 = -2; gr.C = 0; }      // finished: post stages pending
        else { gr.n0 = n0; gr.C = std::min(SCHUR_CHUNK, b.n_stop - n0); }
    }
    ++sc.chunk;
    return SCATT_OK;
}

// Post stages of the slots `sel` of one group, whose sweep has reached N:
// K extraction, the outer boundary value, the backward sweep over the
// asymptotic window, the amplitude fit and the dipoles.  Outputs go to rows
// `rows` of `out`.  A failed energy (singular pivot, closed channel) leaves
// its status in out->status and the first one in *first_status / *first_msg.
int post_slots(Scan& sc, const std::vector<int>& sel, const std::vector<long>& rows, const scatt_outputs* out,
               int* first_status, std::string* first_msg) {
    ScanTables& t = *sc.ctx->tab;
    const scatt_solve_opts& o = sc.o;
    cudaStream_t s = sc.ctx->stream;
    BatchDev& b = sc.b;
    const int cnt = (int)sel.size();
    if (cnt == 0) return SCATT_OK;
    const int N = b.N, K = b.Krows, Nf = b.Nf;
    const int ne_fit = sc.ne_fit, nfit = sc.nfit;
    auto ED = [&](int i) -> const EnergyDev& { return sc.ed[sel[i]]; };
    std::vector<PostBufs>& P = sc.P;
    Launcher& L = sc.L;
    int maxNp = 0;
    for (int e = 0; e < cnt; ++e) maxNp = std::max(maxNp, ED(e).Np);
    // the slots' device counters: stability shifts and the first failing step
    std::vector<EnergyDev> edh(cnt);
    SCATT_CUDA_TRY(cudaStreamSynchronize(s));
    for (int e = 0; e < cnt; ++e)
        SCATT_CUDA_TRY(cudaMemcpy(&edh[e], sc.d_ed.p + sel[e], sizeof(EnergyDev), cudaMemcpyDeviceToHost));
    std::vector<int> status(cnt, SCATT_OK);
    for (int e = 0; e < cnt; ++e)
        if (edh[e].err_code) status[e] = edh[e].err_code;

    // ---- KMatrixExtractor (KMatrixExtractor.cpp:75-198), n_match = Nr - 2
    {
        std::vector<CopyEntry> cp;
        std::vector<GjEntry> gj;
        for (int e = 0; e < cnt; ++e) {
            const EnergyDev& d = ED(e);
            const double* rin = d.tailR ? d.tailR + (size_t)(N - 1 - b.n_s) * d.Nt * d.Nt
                                        : (((N - 1) & 1) ? d.Rinv1 : d.Rinv0);
            cp.push_back(CopyEntry{rin, d.Ra, d.Nt, d.Nt, d.Nt, d.Nt, 1.0});
            gj.push_back(GjEntry{d.Ra, d.Rw, d.Rinv0, d.sigR, d.ridR, d.stR, d.Nt, d.Nt, d.Nt});
        }
        SCATT_TRY(L.copy(cp));
        SCATT_TRY(L.gj(gj, false));
        // coupling norms
        std::vector<const double*> Rp(cnt);
        std::vector<int> np(cnt), nt(cnt);
        for (int e = 0; e < cnt; ++e) { Rp[e] = ED(e).Rinv0; np[e] = ED(e).Np; nt[e] = ED(e).Nt; }
        DevBuf<const double*> dRp;
        DevBuf<int> dnp, dnt;
        DevBuf<double> dnorm;
        SCATT_TRY(upload_vec(dRp, Rp, s));
        SCATT_TRY(upload_vec(dnp, np, s));
        SCATT_TRY(upload_vec(dnt, nt, s));
        SCATT_TRY(dnorm.alloc(2 * (size_t)cnt));
        k_block_norms<<<cnt, 1024, 0, s>>>(dRp.p, dnp.p, dnt.p, dnorm.p);
        SCATT_COUNT_LAUNCH(1);
        std::vector<double> norms(2 * cnt);
        SCATT_CUDA_TRY(cudaMemcpyAsync(norms.data(), dnorm.p, norms.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
        SCATT_CUDA_TRY(cudaStreamSynchronize(s));
        std::vector<CopyEntry> c2, c3;
        std::vector<GjEntry> g2;
        std::vector<GemmEntry> m1, m2;
        std::vector<int> coupled(cnt, 0);
        for (int e = 0; e < cnt; ++e) {
            const EnergyDev& d = ED(e);
            const int Np = d.Np, Nt = d.Nt;
            // S_schur starts as R_psi_psi
            c2.push_back(CopyEntry{d.Rinv0, d.Sw, Np, Np, Nt, Np, 1.0});
            coupled[e] = (Nf > 0) && !(norms[2 * e] < 1e-14 && norms[2 * e + 1] < 1e-14);
            if (coupled[e]) {
                c3.push_back(CopyEntry{d.Rinv0 + (size_t)Np * Nt + Np, d.Ra, Nf, Nf, Nt, Nf, 1.0});
                g2.push_back(GjEntry{d.Ra, d.Rw, d.Rinv1, d.sigR, d.ridR, d.stR, Nf, Nf, Nf});
                // Y = R_psi_f R_ff^-1 (into T), S_schur -= Y R_f_psi
                m1.push_back(GemmEntry{d.Rinv0 + (size_t)Np * Nt, d.Rinv1, d.T, Np, Nf, Nf, Nt, Nf, Np, 1.0, 0.0});
                m2.push_back(GemmEntry{d.T, d.Rinv0 + Np, d.Sw, Np, Np, Nf, Np, Nt, Np, -1.0, 1.0});
            }
        }
        SCATT_TRY(L.copy(c2));
        SCATT_TRY(L.copy(c3));
        SCATT_TRY(L.gj(g2, false));
        SCATT_TRY(L.gemm(m1, 0, 0));
        SCATT_TRY(L.gemm(m2, 0, 0));
        std::vector<KmeEntry> ke;
        for (int e = 0; e < cnt; ++e) {
            const EnergyDev& d = ED(e);
            ke.push_back(KmeEntry{d.Sw, P[e].Amat, P[e].Bmat, P[e].tab, d.Np, d.k});
        }
        DevBuf<KmeEntry> dke;
        SCATT_TRY(upload_vec(dke, ke, s));
        k_kme_tab<<<dim3(cdiv(maxNp, 128), cnt), 128, 0, s>>>(dke.p, t.d_l_of_mu.p, t.dr, t.Nr);
        SCATT_COUNT_LAUNCH(1);
        k_kme_mats<<<dim3(64, cnt), TPB, 0, s>>>(dke.p);
        SCATT_COUNT_LAUNCH(1);
        SCATT_CUDA_TRY(cudaGetLastError());
        // K = B_mat^-1 A_mat (the reference solves with partial-pivot LU)
        std::vector<CopyEntry> c4;
        std::vector<GjEntry> g4;
        std::vector<GemmEntry> m4;
        for (int e = 0; e < cnt; ++e) {
            const int Np = ED(e).Np;
            c4.push_back(CopyEntry{P[e].Bmat, P[e].Bw, Np, Np, Np, Np, 1.0});
            g4.push_back(GjEntry{P[e].Bw, P[e].Kc, P[e].Binv, P[e].sig, P[e].rid, P[e].st, Np, Np, Np});
            m4.push_back(GemmEntry{P[e].Binv, P[e].Amat, P[e].Kraw, Np, Np, Np, Np, Np, Np, 1.0, 0.0});
        }
        SCATT_TRY(L.copy(c4));
        SCATT_TRY(L.gj(g4, false));
        SCATT_TRY(L.gemm(m4, 0, 0));
        std::vector<const double*> kr(cnt);
        std::vector<double*> ko(cnt), pb(cnt);
        for (int e = 0; e < cnt; ++e) { kr[e] = P[e].Kraw; ko[e] = P[e].K; pb[e] = P[e].psibc; }
        DevBuf<const double*> dkr;
        DevBuf<double*> dko, dpb;
        SCATT_TRY(upload_vec(dkr, kr, s));
        SCATT_TRY(upload_vec(dko, ko, s));
        SCATT_TRY(upload_vec(dpb, pb, s));
        k_kme_final<<<dim3(64, cnt), TPB, 0, s>>>(dke.p, dkr.p, dko.p, dpb.p);
        SCATT_COUNT_LAUNCH(1);
        SCATT_CUDA_TRY(cudaGetLastError());
        SCATT_CUDA_TRY(cudaStreamSynchronize(s));
        for (int e = 0; e < cnt; ++e) edh[e].deltaA = coupled[e] ? 0.0 : 1.0;
    }

    // ---- outer boundary Z_N (BackPropagator.cpp:127-197) and the dipole contraction
    sc.vb.build(b, N, s);
    {
        std::vector<GemmEntry> mv, mf, mb;
        for (int e = 0; e < cnt; ++e) {
            const EnergyDev& d = ED(e);
            const int Np = d.Np;
            mv.push_back(GemmEntry{sc.vb.V.p, P[e].psibc, P[e].VP, Np, Np, Np, b.Np_max, Np, Np, b.h2_6, 0.0});
            if (N < b.n_tr && Nf > 0) {
                mf.push_back(GemmEntry{sc.vb.B.p, P[e].psibc, P[e].fN, Nf, Np, Np, b.Np_max, Np, Nf, 1.0, 0.0});
            }
        }
        SCATT_TRY(L.gemm(mv, 0, 0));
        if (!mf.empty()) {
            SCATT_TRY(L.gemm(mf, 1, 0));
            // f_N = -D^-1 (B^T psi): scale rows by -Dinv through a copy-with-scale per f row is
            // not expressible as one CopyEntry; do it with a tiny GEMM-free kernel via Bs^T:
            // B_N f_N = B_N (-(D^-1 B^T psi)) = -(Bs_N)(B_N^T psi) with Bs = B D^-1.
            for (int e = 0; e < cnt; ++e) {
                const int Np = ED(e).Np;
                mb.push_back(GemmEntry{sc.vb.Bs.p, P[e].fN, P[e].Bf, Np, Np, Nf, b.Np_max, Nf, Np, -1.0, 0.0});
            }
            SCATT_TRY(L.gemm(mb, 0, 0));
        }
        std::vector<ZEntry> ze;
        for (int e = 0; e < cnt; ++e) {
            const EnergyDev& d = ED(e);
            ze.push_back(ZEntry{P[e].psibc, P[e].VP, mb.empty() ? nullptr : P[e].Bf, P[e].Z0, d.Np, d.Nt,
                                b.h2_6 * d.E});
        }
        DevBuf<ZEntry> dze;
        SCATT_TRY(upload_vec(dze, ze, s));
        k_build_Z<<<dim3(64, cnt), TPB, 0, s>>>(dze.p);
        SCATT_COUNT_LAUNCH(1);
        SCATT_CUDA_TRY(cudaGetLastError());
        // d_all = G_{N-1} Z_N (+ C_N psi_N when N is inside the dipole window)
        std::vector<GemmEntry> md, mc;
        for (int e = 0; e < cnt; ++e) {
            const EnergyDev& d = ED(e);
            const double* Gf = (N & 1) ? d.G1 : d.G0;
            md.push_back(GemmEntry{Gf, P[e].Z0, P[e].dall, K, d.Np, d.Nt, K, d.Nt, K, 1.0, 0.0});
            if (N < b.n_pts)
                mc.push_back(GemmEntry{t.Ctab.p + (size_t)N * K * b.Np_max, P[e].psibc, P[e].dall, K, d.Np, d.Np,
                                       K, d.Np, K, 1.0, 1.0});
        }
        SCATT_TRY(L.gemm(md, 0, 0));
        SCATT_TRY(L.gemm(mc, 0, 0));
    }

    // ---- backward sweep over the asymptotic window (BackPropagator.cpp:603-703),
    // when the window is kept; otherwise the fit was accumulated forward
    const bool keep = o.keep_window != 0;
    if (keep) {
        std::vector<CopyEntry> c0;
        for (int e = 0; e < cnt; ++e) {
            const EnergyDev& d = ED(e);
            c0.push_back(CopyEntry{P[e].psibc, d.psiT + (size_t)(N - b.n_s) * d.Np * d.Np, d.Np, d.Np, d.Np, d.Np, 1.0});
        }
        SCATT_TRY(L.copy(c0));
        std::vector<double*> zc(cnt), zn(cnt);
        for (int e = 0; e < cnt; ++e) { zc[e] = P[e].Z0; zn[e] = P[e].Z1; }
        for (int n = N - 1; n >= b.n_s; --n) {
            const bool exch = n < b.n_tr && Nf > 0;
            if (exch) sc.vb.build(b, n, s);
            std::vector<GemmEntry> mz, mr, mp;
            std::vector<CopyEntry> cr;
            for (int e = 0; e < cnt; ++e) {
                const EnergyDev& d = ED(e);
                const int Np = d.Np, Nt = d.Nt;
                const size_t slot = (size_t)(n - b.n_s);
                mz.push_back(GemmEntry{d.tailR + slot * Nt * Nt, zc[e], zn[e], Nt, Np, Nt, Nt, Nt, Nt, 1.0, 0.0});
                const double* sinv = d.tailS + slot * Np * Np;
                if (exch) {
                    cr.push_back(CopyEntry{zn[e], P[e].rhs, Np, Np, Nt, Np, 1.0});
                    mr.push_back(GemmEntry{sc.vb.Bs.p, zn[e] + Np, P[e].rhs, Np, Np, Nf, b.Np_max, Nt, Np, -1.0, 1.0});
                    mp.push_back(GemmEntry{sinv, P[e].rhs, d.psiT + slot * Np * Np, Np, Np, Np, Np, Np, Np, 1.0, 0.0});
                } else {
                    mp.push_back(GemmEntry{sinv, zn[e], d.psiT + slot * Np * Np, Np, Np, Np, Np, Nt, Np, 1.0, 0.0});
                }
            }
            SCATT_TRY(L.gemm(mz, 0, 0));
            SCATT_TRY(L.copy(cr));
            SCATT_TRY(L.gemm(mr, 0, 0));
            SCATT_TRY(L.gemm(mp, 0, 0));
            std::swap(zc, zn);
        }
    }

    // ---- AsymptoticAmplitudes (AsymptoticAmplitudes.cpp:64-359)
    std::vector<double> aared(2 * cnt), aasym(2 * cnt);
    std::vector<int> nclosed(cnt, 0);
    if (!keep) {
        // [A; B] = G_A(N-1)^T Z_N, then the closed channels' rows
        std::vector<GemmEntry> ma;
        std::vector<AbEntry> ab;
        for (int e = 0; e < cnt; ++e) {
            const EnergyDev& d = ED(e);
            const double* GA = (N & 1) ? d.GA1 : d.GA0;
            const int Np = d.Np, Nt = d.Nt;
            ma.push_back(GemmEntry{GA, P[e].Z0, P[e].Aaa, Np, Np, Nt, 2 * Np, Nt, Np, 1.0, 0.0});
            ma.push_back(GemmEntry{GA + Np, P[e].Z0, P[e].Baa, Np, Np, Nt, 2 * Np, Nt, Np, 1.0, 0.0});
            ab.push_back(AbEntry{P[e].Aaa, P[e].Baa, d.Mab, Np});
        }
        SCATT_TRY(L.gemm(ma, 0, 0));
        DevBuf<AbEntry> dab;
        SCATT_TRY(upload_vec(dab, ab, s));
        k_ab_closed<<<dim3(64, cnt), TPB, 0, s>>>(dab.p, t.d_l_of_mu.p);
        SCATT_COUNT_LAUNCH(1);
        SCATT_CUDA_TRY(cudaGetLastError());
        SCATT_CUDA_TRY(cudaStreamSynchronize(s));
        for (int e = 0; e < cnt; ++e) {
            aared[2 * e] = 1.0;                 // the fit residual needs psi at every window point: not kept
            aared[2 * e + 1] = NAN;
            std::vector<double> M(8 * (size_t)(ED(e).l_cont + 1));
            SCATT_CUDA_TRY(cudaMemcpy(M.data(), ED(e).Mab, M.size() * sizeof(double), cudaMemcpyDeviceToHost));
            for (int l = 0; l <= ED(e).l_cont; ++l)
                if (M[8 * l + 4] != 0.0) ++nclosed[e];
            if (nclosed[e] > 0 && !o.allow_closed_channels && status[e] == SCATT_OK) status[e] = SCATT_ERR_CLOSED_CHANNEL;
        }
    }
    {
      if (keep) {
        std::vector<AaEntry> ae;
        int maxl = 0;
        for (int e = 0; e < cnt; ++e) {
            const EnergyDev& d = ED(e);
            ae.push_back(AaEntry{d.psiT, P[e].aatab, P[e].aaM, P[e].Aaa, P[e].Baa, P[e].aared, d.Np, d.l_cont, d.k});
            maxl = std::max(maxl, d.l_cont);
        }
        DevBuf<AaEntry> dae;
        SCATT_TRY(upload_vec(dae, ae, s));
        k_aa_tab<<<dim3(64, cnt), TPB, 0, s>>>(dae.p, b.n_s, nfit, t.dr);
        SCATT_COUNT_LAUNCH(1);
        k_aa_normal<<<dim3(cdiv(maxl + 1, 64), cnt), 64, 0, s>>>(dae.p, nfit);
        SCATT_COUNT_LAUNCH(1);
        k_aa_fit<<<dim3(64, cnt), TPB, 0, s>>>(dae.p, t.d_l_of_mu.p, nfit);
        SCATT_COUNT_LAUNCH(1);
        SCATT_CUDA_TRY(cudaGetLastError());
        std::vector<const double*> rp(cnt);
        std::vector<int> rc(cnt);
        for (int e = 0; e < cnt; ++e) { rp[e] = P[e].aared; rc[e] = ED(e).Np * ED(e).Np; }
        DevBuf<const double*> drp;
        DevBuf<int> drc;
        DevBuf<double> dout;
        SCATT_TRY(upload_vec(drp, rp, s));
        SCATT_TRY(upload_vec(drc, rc, s));
        SCATT_TRY(dout.alloc(2 * (size_t)cnt));
        k_max_pairs<<<cnt, 1024, 0, s>>>(drp.p, drc.p, dout.p);
        SCATT_COUNT_LAUNCH(1);
        SCATT_CUDA_TRY(cudaMemcpyAsync(aared.data(), dout.p, 2 * cnt * sizeof(double), cudaMemcpyDeviceToHost, s));
        SCATT_CUDA_TRY(cudaStreamSynchronize(s));
        for (int e = 0; e < cnt; ++e) {
            std::vector<double> M(8 * (size_t)(ED(e).l_cont + 1));
            SCATT_CUDA_TRY(cudaMemcpy(M.data(), P[e].aaM, M.size() * sizeof(double), cudaMemcpyDeviceToHost));
            for (int l = 0; l <= ED(e).l_cont; ++l)
                if (M[8 * l + 4] != 0.0) ++nclosed[e];
            if (nclosed[e] > 0 && !o.allow_closed_channels && status[e] == SCATT_OK) status[e] = SCATT_ERR_CLOSED_CHANNEL;
        }
      }
        // K = B A^-1
        std::vector<CopyEntry> ca;
        std::vector<GjEntry> ga;
        std::vector<GemmEntry> mk;
        for (int e = 0; e < cnt; ++e) {
            const int Np = ED(e).Np;
            ca.push_back(CopyEntry{P[e].Aaa, P[e].Aw, Np, Np, Np, Np, 1.0});
            ga.push_back(GjEntry{P[e].Aw, P[e].Kc, P[e].Ainv, P[e].sig, P[e].rid, P[e].st, Np, Np, Np});
            mk.push_back(GemmEntry{P[e].Baa, P[e].Ainv, P[e].Kc + (size_t)Np * Np, Np, Np, Np, Np, Np, Np, 1.0, 0.0});
        }
        SCATT_TRY(L.copy(ca));
        SCATT_TRY(L.gj(ga, false));
        SCATT_TRY(L.gemm(mk, 0, 0));
        std::vector<const double*> kp(cnt), ap(cnt);
        std::vector<int> npv(cnt);
        for (int e = 0; e < cnt; ++e) {
            kp[e] = P[e].Kc + (size_t)ED(e).Np * ED(e).Np;
            ap[e] = P[e].Aaa;
            npv[e] = ED(e).Np;
        }
        DevBuf<const double*> dkp, dap;
        DevBuf<int> dnpv;
        DevBuf<double> dsk, dsa;
        SCATT_TRY(upload_vec(dkp, kp, s));
        SCATT_TRY(upload_vec(dap, ap, s));
        SCATT_TRY(upload_vec(dnpv, npv, s));
        SCATT_TRY(dsk.alloc(2 * (size_t)cnt));
        SCATT_TRY(dsa.alloc(2 * (size_t)cnt));
        k_sym_err<<<cnt, 1024, 0, s>>>(dkp.p, dnpv.p, dsk.p);
        SCATT_COUNT_LAUNCH(1);
        k_sym_err<<<cnt, 1024, 0, s>>>(dap.p, dnpv.p, dsa.p);
        SCATT_COUNT_LAUNCH(1);
        std::vector<double> sk(2 * cnt), sa(2 * cnt);
        SCATT_CUDA_TRY(cudaMemcpyAsync(sk.data(), dsk.p, sk.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
        SCATT_CUDA_TRY(cudaMemcpyAsync(sa.data(), dsa.p, sa.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
        SCATT_CUDA_TRY(cudaStreamSynchronize(s));
        for (int e = 0; e < cnt; ++e) { aasym[2 * e] = sk[2 * e]; aasym[2 * e + 1] = sa[2 * e + 1]; }
    }

    // ---- DipoleMatrixElement finalisation (DipoleMatrixElement.cpp:673-947)
    {
        std::vector<const double*> ap(cnt), bp;
        std::vector<double*> qp(cnt);
        std::vector<int> npv(cnt);
        bp.resize(cnt);
        for (int e = 0; e < cnt; ++e) {
            ap[e] = P[e].Aaa; bp[e] = P[e].Baa; qp[e] = P[e].Q; npv[e] = ED(e).Np;
        }
        DevBuf<const double*> dap, dbp;
        DevBuf<double*> dqp;
        DevBuf<int> dnp;
        SCATT_TRY(upload_vec(dap, ap, s));
        SCATT_TRY(upload_vec(dbp, bp, s));
        SCATT_TRY(upload_vec(dqp, qp, s));
        SCATT_TRY(upload_vec(dnp, npv, s));
        k_embed<<<dim3(64, cnt), TPB, 0, s>>>(dap.p, dbp.p, dqp.p, dnp.p);
        SCATT_COUNT_LAUNCH(1);
        SCATT_CUDA_TRY(cudaGetLastError());
        std::vector<GjEntry> gq;
        for (int e = 0; e < cnt; ++e) {
            const int n2 = 2 * ED(e).Np;
            gq.push_back(GjEntry{P[e].Q, P[e].Qw, P[e].Qinv, P[e].sig, P[e].rid, P[e].st, n2, n2, n2});
        }
        SCATT_TRY(L.gj(gq, false));
        DevBuf<double> ddc, dsp;
        SCATT_TRY(upload_vec(ddc, t.d_corr, s));
        SCATT_TRY(upload_vec(dsp, t.spin, s));
        std::vector<DmeEntry> de;
        for (int e = 0; e < cnt; ++e)
            de.push_back(DmeEntry{P[e].Qinv, P[e].dall, ddc.p, dsp.p, P[e].Dre, P[e].Dim, P[e].Drre, P[e].Drim,
                                  P[e].ore, P[e].oim, ED(e).Np, K, t.n_occ});
        DevBuf<DmeEntry> dde;
        SCATT_TRY(upload_vec(dde, de, s));
        k_dme_o<<<dim3(64, cnt), TPB, 0, s>>>(dde.p);
        SCATT_COUNT_LAUNCH(1);
        k_dme_D<<<dim3(16, cnt), TPB, 0, s>>>(dde.p, o.orthogonalize);
        SCATT_COUNT_LAUNCH(1);
        SCATT_CUDA_TRY(cudaGetLastError());
        SCATT_CUDA_TRY(cudaStreamSynchronize(s));
    }

    // ---- eigenphases (diagnostics)
    std::vector<std::vector<double>> eigk(cnt), eiga(cnt);
    if (o.diagnostics) {
        std::vector<CopyEntry> cc;
        std::vector<EigEntry> ee;
        for (int e = 0; e < cnt; ++e) {
            const int Np = ED(e).Np;
            cc.push_back(CopyEntry{P[e].K, P[e].Amat, Np, Np, Np, Np, 1.0});
            cc.push_back(CopyEntry{P[e].Kc + (size_t)Np * Np, P[e].Bmat, Np, Np, Np, Np, 1.0});
            ee.push_back(EigEntry{P[e].Amat, Np, Np, P[e].ew_d, P[e].ew_e, P[e].ew_w, P[e].eigK});
            ee.push_back(EigEntry{P[e].Bmat, Np, Np, P[e].ew_d + Np, P[e].ew_e + Np, P[e].Bw, P[e].eigA});
        }
        SCATT_TRY(L.copy(cc));
        DevBuf<EigEntry> dee;
        SCATT_TRY(upload_vec(dee, ee, s));
        SCATT_TRY(sym_eigvals_batched(dee.p, (int)ee.size(), maxNp, 0, s));
        SCATT_CUDA_TRY(cudaStreamSynchronize(s));
        for (int e = 0; e < cnt; ++e) {
            const int Np = ED(e).Np;
            eigk[e].resize(Np);
            eiga[e].resize(Np);
            SCATT_CUDA_TRY(cudaMemcpy(eigk[e].data(), P[e].eigK, Np * sizeof(double), cudaMemcpyDeviceToHost));
            SCATT_CUDA_TRY(cudaMemcpy(eiga[e].data(), P[e].eigA, Np * sizeof(double), cudaMemcpyDeviceToHost));
        }
    }

    // ================================================================ outputs
    const int Npm = t.Np_max;
    for (int e = 0; e < cnt; ++e) {
        const EnergyDev& d = ED(e);
        const int Np = d.Np, ge = rows[e];
        auto mat = [&](double* host, const double* dev) -> int {
            if (!host) return SCATT_OK;
            double* h = host + (size_t)ge * Npm * Npm;
            if (Np < Npm) std::fill(h, h + (size_t)Npm * Npm, 0.0);      // else all of it is copied over
            return cuda_status(cudaMemcpy2D(h, Npm * sizeof(double), dev, Np * sizeof(double), Np * sizeof(double),
                                            Np, cudaMemcpyDeviceToHost), "download");
        };
        SCATT_TRY(mat(out->K_kme, P[e].K));
        SCATT_TRY(mat(out->A, P[e].Aaa));
        SCATT_TRY(mat(out->B, P[e].Baa));
        SCATT_TRY(mat(out->K_aa, P[e].Kc + (size_t)Np * Np));
        std::vector<double> dall((size_t)K * Np), Dre(6 * Np), Dim(6 * Np), Drre(6 * Np), Drim(6 * Np);
        SCATT_CUDA_TRY(cudaMemcpy(dall.data(), P[e].dall, dall.size() * sizeof(double), cudaMemcpyDeviceToHost));
        SCATT_CUDA_TRY(cudaMemcpy(Dre.data(), P[e].Dre, Dre.size() * sizeof(double), cudaMemcpyDeviceToHost));
        SCATT_CUDA_TRY(cudaMemcpy(Dim.data(), P[e].Dim, Dim.size() * sizeof(double), cudaMemcpyDeviceToHost));
        SCATT_CUDA_TRY(cudaMemcpy(Drre.data(), P[e].Drre, Drre.size() * sizeof(double), cudaMemcpyDeviceToHost));
        SCATT_CUDA_TRY(cudaMemcpy(Drim.data(), P[e].Drim, Drim.size() * sizeof(double), cudaMemcpyDeviceToHost));
        if (out->b_overlap) {
            double* h = out->b_overlap + (size_t)ge * Npm * t.n_occ;
            std::fill(h, h + (size_t)Npm * t.n_occ, 0.0);
            for (int a = 0; a < t.n_occ; ++a)
                for (int be = 0; be < Np; ++be) h[be + (size_t)a * Npm] = o.orthogonalize ? dall[(N_SLOTS + a) + (size_t)be * K] : 0.0;
        }
        for (int sl = 0; sl < N_SLOTS; ++sl) {
            double ps = 0.0;
            for (int mu = 0; mu < Np; ++mu) {
                const double re = o.orthogonalize ? Dre[sl * Np + mu] : Drre[sl * Np + mu];
                const double im = o.orthogonalize ? Dim[sl * Np + mu] : Drim[sl * Np + mu];
                ps += re * re + im * im;
            }
            auto put = [&](double* host, const std::vector<double>& v, bool raw_d) {
                if (!host) return;
                double* h = host + ((size_t)ge * N_SLOTS + sl) * Npm;
                std::fill(h, h + Npm, 0.0);
                for (int mu = 0; mu < Np; ++mu) h[mu] = raw_d ? dall[sl + (size_t)mu * K] : v[sl * Np + mu];
            };
            put(out->D_re, o.orthogonalize ? Dre : Drre, false);
            put(out->D_im, o.orthogonalize ? Dim : Drim, false);
            put(out->Draw_re, Drre, false);
            put(out->Draw_im, Drim, false);
            put(out->d_raw, Dre, true);
            if (out->d_corr)
                for (int a = 0; a < t.n_occ; ++a)
                    out->d_corr[((size_t)ge * N_SLOTS + sl) * t.n_occ + a] = o.orthogonalize ? t.d_corr[a * N_SLOTS + sl] : 0.0;
            if (out->partial_sigma) out->partial_sigma[(size_t)ge * N_SLOTS + sl] = ps;
        }
        if (out->eig_kme) {
            double* h = out->eig_kme + (size_t)ge * Npm;
            std::fill(h, h + Npm, 0.0);
            for (int i = 0; i < (int)eigk[e].size(); ++i) h[i] = std::atan(eigk[e][i]);
        }
        if (out->eig_aa) {
            double* h = out->eig_aa + (size_t)ge * Npm;
            std::fill(h, h + Npm, 0.0);
            for (int i = 0; i < (int)eiga[e].size(); ++i) h[i] = std::atan(eiga[e][i]);
        }
        if (out->diag) {
            double* g = out->diag + (size_t)ge * SCATT_NDIAG;
            std::fill(g, g + SCATT_NDIAG, 0.0);
            g[SCATT_DIAG_FIT_RESIDUAL_MAX] = aared[2 * e + 1];
            g[SCATT_DIAG_FIT_RESIDUAL_REL] = aared[2 * e + 1] / std::max(aared[2 * e], 1e-30);
            g[SCATT_DIAG_A_MINUS_I_MAX] = aasym[2 * e + 1];
            g[SCATT_DIAG_K_SYMMETRY_ERR_AA] = aasym[2 * e];
            g[SCATT_DIAG_S_UNITARITY_ERR_AA] = NAN;
            g[SCATT_DIAG_K_SYMMETRY_ERR_KME] = 0.0;
            g[SCATT_DIAG_UNITARITY_ERR_KME] = NAN;
            g[SCATT_DIAG_N_FIT_START] = b.n_s;
            g[SCATT_DIAG_N_FIT_END] = ne_fit;
            g[SCATT_DIAG_N_TRANSITION] = t.n_tr;
            g[SCATT_DIAG_SHIFTS_A] = edh[e].shiftsA;
            g[SCATT_DIAG_SHIFTS_S] = edh[e].shiftsS;
            g[SCATT_DIAG_N_CLOSED_L] = nclosed[e];
            g[SCATT_DIAG_SCHUR_COUPLING_0] = edh[e].deltaA;
        }
        if (out->status) out->status[ge] = status[e];
    }
    for (int e = 0; e < cnt; ++e)
        if (status[e] != SCATT_OK && *first_status == SCATT_OK) {
            *first_status = status[e];
            if (status[e] == SCATT_ERR_CLOSED_CHANNEL)
                *first_msg = "AsymptoticAmplitudes: singular normal matrix (closed channel) at energy " +
                             std::to_string(rows[e]) + "; set allow_closed_channels";
            else
                *first_msg = "singular or non-finite pivot at energy " + std::to_string(rows[e]) + ", radial step " +
                             std::to_string(edh[e].err_step);
        }
    return SCATT_OK;
}

// Runs chunks until at least one group has finished its sweep, then its
// post stages.  out_row(slot, i) gives the output row of the i-th finished
// energy (held by `slot`).  *n_done receives the number of finished energies
// (0: nothing was in flight and the queue is empty); done_jobs lists their
// submission indices.
template <class RowOf>
int scan_advance(Scan& sc, const scatt_outputs* out, RowOf out_row, int* n_done, std::vector<long>* done_jobs,
                 int* first_status, std::string* first_msg) {
    cudaStream_t s = sc.ctx->stream;
    *n_done = 0;
    SolveStats& stats = sc.ctx->stats;
    const unsigned long long launches0 = launch_counter();
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, evp = nullptr;
    ChunkTiming tm;
    sc.events.reset();
    if (sc.o.timing) {
        SCATT_TRY(sc.events.get(&ev0));
        SCATT_TRY(sc.events.get(&ev1));
        SCATT_TRY(sc.events.get(&evp));
        SCATT_CUDA_TRY(cudaEventRecord(ev0, s));
    }
    std::vector<int> finished;
    for (;;) {
        // idle groups whose turn has come take queued energies
        for (int g = 0; g < sc.G; ++g)
            if (sc.grp[g].n0 == -1 && sc.chunk >= sc.start_chunk[g] && !sc.queue.empty())
                SCATT_TRY(load_group(sc, g));
        bool running = false, waiting = false;
        for (int g = 0; g < sc.G; ++g) {
            running |= sc.grp[g].n0 >= 0;
            waiting |= sc.grp[g].n0 == -1 && sc.chunk < sc.start_chunk[g];
        }
        if (!running) {
            if (sc.queue.empty() || !waiting) break;
            // nothing runs until the next staggered start: start it now
            long next = -1;
            for (int g = 0; g < sc.G; ++g)
                if (sc.grp[g].n0 == -1 && (next < 0 || sc.start_chunk[g] < next)) next = sc.start_chunk[g];
            sc.chunk = std::max(sc.chunk, next);
            continue;
        }
        SCATT_TRY(run_chunk(sc, sc.o.timing ? &tm : nullptr));
        for (int g = 0; g < sc.G; ++g)
            if (sc.grp[g].n0 == -2) finished.push_back(g);
        if (!finished.empty()) break;
    }
    if (sc.o.timing) SCATT_CUDA_TRY(cudaEventRecord(evp, s));
    for (int g : finished) {
        std::vector<int> sel;
        std::vector<long> rows;
        for (int e = g * sc.gs; e < std::min(sc.slots, (g + 1) * sc.gs); ++e)
            if (sc.ed[e].live) {
                sel.push_back(e);
                rows.push_back(out_row(e, *n_done + (int)sel.size() - 1));
            }
        SCATT_TRY(post_slots(sc, sel, rows, out, first_status, first_msg));
        for (int e : sel) {
            if (done_jobs) done_jobs->push_back(sc.job_of[e]);
            sc.ed[e].live = 0;
            sc.job_of[e] = -1;
        }
        *n_done += (int)sel.size();
        sc.grp[g].n0 = -1;                    // k_advance already stopped it on the device
        sc.start_chunk[g] = sc.chunk;         // refill at once: the group keeps its phase
    }
    if (sc.o.timing) {
        SCATT_CUDA_TRY(cudaEventRecord(ev1, s));
        SCATT_CUDA_TRY(cudaEventSynchronize(ev1));
        float ms_all = 0.f, ms_sweep = 0.f;
        SCATT_CUDA_TRY(cudaEventElapsedTime(&ms_all, ev0, ev1));
        SCATT_CUDA_TRY(cudaEventElapsedTime(&ms_sweep, ev0, evp));
        double rs = 0.0;
        for (auto& pr : tm.rinv) {
            float ms = 0.f;
            SCATT_CUDA_TRY(cudaEventElapsedTime(&ms, pr.first, pr.second));
            rs += ms * 1e-3;
        }
        stats.device_s += ms_all * 1e-3;
        stats.sweep_s += ms_sweep * 1e-3;
        stats.post_s += (ms_all - ms_sweep) * 1e-3;
        stats.rinv_s += rs;
        stats.rinv_calls += (double)tm.rinv.size();
        stats.rinv_flops += tm.flops;
    }
    stats.launches += launch_counter() - launches0;
    return SCATT_OK;
}

int check_energies(const ScanTables& t, int n, const double* E, const int* lc, const char* who) {
    for (int e = 0; e < n; ++e) {
        if (!(E[e] > 0.0)) {
            set_last_error("KMatrixExtractor: energy must be > 0 for scattering");
            return SCATT_ERR_ARG;
        }
        const int l = lc ? lc[e] : t.l_max;
        if (l < 0 || l > t.l_max || std::min(l, 10) != t.l_x) {
            set_last_error(std::string(who) + ": l_cont " + std::to_string(l) +
                           " is outside the uploaded scan or changes the exchange cutoff min(l_cont, 10)");
            return SCATT_ERR_ARG;
        }
    }
    return SCATT_OK;
}

// Slots that fit in 85% of the free device memory at continuum cutoff l_cap
// with `groups` phase groups (at least 1).
int slots_that_fit(Context& ctx, const scatt_solve_opts& o, int l_cap, int groups, int* out) {
    const ScanTables& t = *ctx.tab;
    BatchDev b{};
    SCATT_TRY(make_consts(t, o, b));
    size_t freeb = 0, totb = 0;
    SCATT_CUDA_TRY(cudaMemGetInfo(&freeb, &totb));
    const int Np = (l_cap + 1) * (l_cap + 1), Nt = Np + t.Nf;
    const int nfit = std::min(t.Nr - 1 - 3, b.N) - b.n_s + 1;
    const size_t per = 8 * (slot_doubles(b, Np, Nt, l_cap, o.keep_window != 0) +
                            post_doubles(b, Np, Nt, l_cap, nfit, t.n_occ)) +
                       4 * slot_ints(Np, Nt);
    const size_t fixed = 8 * (group_doubles(b) * (size_t)groups + sym_scratch_doubles(Nt)) + (64u << 20);
    const size_t avail = (size_t)(0.85 * freeb) > fixed ? (size_t)(0.85 * freeb) - fixed : 0;
    *out = (int)std::max<size_t>(1, avail / std::max<size_t>(per, 1));
    return SCATT_OK;
}

}  // namespace

int solve_batch(Context& ctx, const scatt_solve_opts& o, int n_energy, const double* E, const int* lc,
                const scatt_outputs* out) {
    const ScanTables& t = *ctx.tab;
    SCATT_TRY(check_energies(t, n_energy, E, lc, "scatt_solve_batch"));
    if (n_energy == 0) return SCATT_OK;
    int l_cap = 0;
    for (int e = 0; e < n_energy; ++e) l_cap = std::max(l_cap, lc ? lc[e] : t.l_max);
    int fit = 1;
    SCATT_TRY(slots_that_fit(ctx, o, l_cap, 1, &fit));
    int slots = std::min(n_energy, o.max_batch > 0 ? o.max_batch : n_energy);
    slots = std::max(1, std::min(slots, fit));
    // lock-step batches: one phase group, refilled when the whole batch is done
    Scan sc;
    SCATT_TRY(scan_open(ctx, o, slots, 1, l_cap, sc));
    for (int e = 0; e < n_energy; ++e) sc.queue.push_back(Job{E[e], lc ? lc[e] : t.l_max, e});
    sc.submitted = n_energy;
    ctx.stats = SolveStats{};
    int first = SCATT_OK;
    std::string msg;
    for (;;) {
        int done = 0;
        SCATT_TRY(scan_advance(sc, out, [&](int slot, int) { return sc.job_of[slot]; }, &done, nullptr, &first, &msg));
        if (done == 0) break;
    }
    if (first != SCATT_OK) set_last_error(msg);
    return first;
}

// ================================================================ adjoint
// Reverse pass of the forward recurrence and the dipole sweep for a batch of
// energies solved as one phase group, with R-ratios checkpointed every
// `segment` steps and each segment recomputed before it is walked backward.
// The reference has no adjoint; the arithmetic is the one of the oracle's
// DipoleAdjoint (oracle/adjoint_recurrence.py):
//   Rbar(n)  = chain + H(n) Gbar(n)^T [+ dJ/dRinv(n) of the small stages]
//   Hbar(n)  = Rinv(n) Gbar(n),  Gbar(n-1) = Hbar(n)
//   chain    = X sym(Rbar) X  (the next step's Rbar start), X = Rinv(n)
//   Wbar(n)  = -12 chain + E_psi L(n) Hbar(n)^T
//   Sinvbar  = Wbar_pp + U Bs^T - Bs Wbar_fp,  U = Bs Wbar_ff - Wbar_pf  [+ small stages]
//   Sbar     = -Y sym(Sinvbar) Y,  Y = Sinv(n)
//   through the stability shifts (n < stab_n): Mbar -= tr(Mbar) P with P the
//   projector on the eigenvectors of lambda_min (averaged over a degenerate
//   cluster); dJ/dV(n) = -h^2/6 Abar, plus the analytic start's diagonal terms.
// The small stages (K extraction, psi_N, the fit window, dipoles) are
// differentiated by the caller (the Python binding runs them in torch on
// views of the window store) and enter as dJ/dRinv, dJ/dSinv over the
// window and dJ/dG(N-1).
namespace {

struct AdjSlot {
    double *ckR, *ckG;             // per segment a: Rinv(a-1) (Nt x Nt), G(a-1)^T (K x Nt)
    double *RB, *T1, *T2, *WB;     // Nt x Nt
    double *GB0, *GB1;             // K x Nt: Gbar^T ping-pong (parity of n)
    double *U;                     // Np x Nf
    double *SBi, *SBs, *SB, *SB2;  // Np x Np
    double *RBw, *SBw;             // window cotangents: (N - n_s) x Nt^2, (N - n_s) x Np^2
    double *ab;                    // 2 Np: analytic-start terms of diag dJ/dV(n), dJ/dV(n+1)
    double *vtr;                   // Nr: tr dJ/dV(n)
    const double *PA, *PS;         // stab_n x Np x Np shift projectors
    int Np, Nt;
};

enum { G_HG, G_HB, G_X1, G_X2, G_CH, G_U, G_S1, G_S2, G_Y1, G_Y2, G_NUM };

struct AdjArgs {
    AdjSlot* s;
    EnergyDev* ed;
    GemmEntry* gm;                 // G_NUM x count
    const double* Ctab;
    const double* Bs;              // Bs(n), Np_max x Nf
    const double* Vn;              // V(n), Np_max x Np_max
    const double* Vn1;             // V(n + 1)
    const int* l_of_mu;
    double* vfull;                 // optional [Nr][Np_max][Np_max] sum over slots
    int count, K, Nf, Np_max, n_start, n_tr, n_pts, n_s, N, stab_n, seg_lo;
    double dr, h2_6;
};

__global__ void k_prep_rev(AdjArgs a, int n) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.count) return;
    const AdjSlot& S = a.s[e];
    const EnergyDev& d = a.ed[e];
    const GemmEntry none{nullptr, nullptr, nullptr, 0, 0, 0, 1, 1, 1, 0.0, 1.0};
    GemmEntry* g = a.gm;
    const int c = a.count;
    if (!d.live) {
        for (int k = 0; k < G_NUM; ++k) g[k * c + e] = none;
        return;
    }
    const int Np = S.Np, Nt = S.Nt, K = a.K, Nf = a.Nf;
    const size_t i = (size_t)(n - a.seg_lo);
    double* Rn = d.segR + i * Nt * Nt;
    double* Yn = d.segS + i * Np * Np;
    double* Ht = d.segH + i * K * Nt;
    double* GBt = (n & 1) ? S.GB1 : S.GB0;
    double* HBt = (n & 1) ? S.GB0 : S.GB1;
    const bool exch = n < a.n_tr && Nf > 0;
    const bool chain = n >= a.n_start;
    g[G_HG * c + e] = GemmEntry{Ht, GBt, S.RB, Nt, Nt, K, K, K, Nt, 1.0, 1.0};
    g[G_HB * c + e] = GemmEntry{GBt, Rn, HBt, K, Nt, Nt, K, Nt, K, 1.0, 0.0};
    g[G_X1 * c + e] = chain ? GemmEntry{Rn, S.T1, S.T2, Nt, Nt, Nt, Nt, Nt, Nt, 1.0, 0.0} : none;
    g[G_X2 * c + e] = chain ? GemmEntry{S.T2, Rn, S.RB, Nt, Nt, Nt, Nt, Nt, Nt, 1.0, 0.0, 1} : none;
    g[G_CH * c + e] = (n < a.n_pts) ? GemmEntry{a.Ctab + (size_t)n * K * a.Np_max, HBt, S.WB, Np, Nt, K, K, K, Nt,
                                                1.0, 1.0}
                                    : none;
    g[G_U * c + e] = exch ? GemmEntry{a.Bs, S.WB + Np + (size_t)Np * Nt, S.U, Np, Nf, Nf, a.Np_max, Nt, Np, 1.0, 1.0}
                          : none;
    g[G_S1 * c + e] = exch ? GemmEntry{S.U, a.Bs, S.SBi, Np, Np, Nf, Np, a.Np_max, Np, 1.0, 1.0} : none;
    g[G_S2 * c + e] = exch ? GemmEntry{a.Bs, S.WB + Np, S.SBi, Np, Np, Nf, a.Np_max, Nt, Np, -1.0, 1.0} : none;
    g[G_Y1 * c + e] = GemmEntry{Yn, S.SBs, S.SB, Np, Np, Np, Np, Np, Np, 1.0, 0.0};
    g[G_Y2 * c + e] = GemmEntry{S.SB, Yn, S.SB2, Np, Np, Np, Np, Np, Np, -1.0, 0.0, 1};
}

// RB += dJ/dRinv(n) of the small stages (window steps); grid (x, slots)
__global__ void k_rev_window(AdjArgs a, int n) {
    const AdjSlot& S = a.s[blockIdx.y];
    if (!a.ed[blockIdx.y].live) return;
    const size_t nt2 = (size_t)S.Nt * S.Nt;
    const double* w = S.RBw + (size_t)(n - a.n_s) * nt2;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < nt2; idx += (size_t)gridDim.x * blockDim.x)
        S.RB[idx] += w[idx];
}

// which = 0: T1 = sym(RB);  1: SBs = sym(SBi)
__global__ void k_rev_sym(AdjArgs a, int which) {
    const AdjSlot& S = a.s[blockIdx.y];
    if (!a.ed[blockIdx.y].live) return;
    const int n = which ? S.Np : S.Nt;
    const double* in = which ? S.SBi : S.RB;
    double* out = which ? S.SBs : S.T1;
    const size_t tot = (size_t)n * n;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < tot; idx += (size_t)gridDim.x * blockDim.x) {
        const size_t r = idx % n, c = idx / n;
        out[idx] = 0.5 * (in[idx] + in[c + r * n]);
    }
}

// after the chain: WB = -12 RB (RB holds X sym(Rbar) X);  in the analytic
// start (chain = 0): RB = 0, WB = 0
__global__ void k_rev_wb(AdjArgs a, int chain) {
    const AdjSlot& S = a.s[blockIdx.y];
    if (!a.ed[blockIdx.y].live) return;
    const size_t tot = (size_t)S.Nt * S.Nt;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < tot; idx += (size_t)gridDim.x * blockDim.x) {
        if (chain) {
            S.WB[idx] = -12.0 * S.RB[idx];
        } else {
            S.WB[idx] = 0.0;
            S.RB[idx] = 0.0;
        }
    }
}

// d R_mumu / d V(n)_mumu and d R_mumu / d V(n+1)_mumu of the analytic start
// (ForwardRPropagator.cpp:78-134) times Rbar_mumu; grid (channels, slots)
__global__ void k_rev_analytic(AdjArgs a, int n) {
    const int e = blockIdx.y;
    const AdjSlot& S = a.s[e];
    const EnergyDev& d = a.ed[e];
    const int mu = blockIdx.x * blockDim.x + threadIdx.x;
    if (!d.live || mu >= S.Np) return;
    double gn = 0.0, gn1 = 0.0;
    if (n >= 1) {
        const int l = a.l_of_mu[mu];
        const double h = a.dr;
        const double rn = a.dr + n * h, rn1 = a.dr + (n + 1) * h;
        const double Mn = 1.0 + a.h2_6 * (d.E - a.Vn[mu + (size_t)mu * a.Np_max]);
        const double Mn1 = 1.0 + a.h2_6 * (d.E - a.Vn1[mu + (size_t)mu * a.Np_max]);
        const double yn = riccati_j(l, d.k * rn), yn1 = riccati_j(l, d.k * rn1);
        const double den = Mn1 * yn1;
        if (fabs(den) > 1e-300) {
            const double rb = S.RB[mu + (size_t)mu * S.Nt];
            gn = rb * (-a.h2_6 * yn / den);
            gn1 = rb * (a.h2_6 * Mn * yn / (Mn1 * den));
        }
    }
    S.ab[mu] = gn;
    S.ab[S.Np + mu] = gn1;
}

// SBi = Wbar_pp [+ window dJ/dSinv(n)];  exchange steps: U = -Wbar_pf
__global__ void k_rev_sbi(AdjArgs a, int n, int exch, int win) {
    const AdjSlot& S = a.s[blockIdx.y];
    if (!a.ed[blockIdx.y].live) return;
    const int Np = S.Np, Nt = S.Nt;
    const size_t np2 = (size_t)Np * Np;
    const double* w = win ? S.SBw + (size_t)(n - a.n_s) * np2 : nullptr;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < np2; idx += (size_t)gridDim.x * blockDim.x) {
        const size_t r = idx % Np, c = idx / Np;
        double v = S.WB[r + c * Nt];
        if (w) v += w[idx];
        S.SBi[idx] = v;
    }
    if (exch) {
        const size_t tot = (size_t)Np * a.Nf;
        for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < tot;
             idx += (size_t)gridDim.x * blockDim.x) {
            const size_t r = idx % Np, c = idx / Np;
            S.U[idx] = -S.WB[r + (Np + c) * Nt];
        }
    }
}

__device__ double block_sum(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += red[i];
        red[32] = s;
    }
    __syncthreads();
    return red[32];
}

// Sbar (in SB2) through the stability shifts of step n (in place: SB2 <- Abar)
// and tr dJ/dV(n) = -h^2/6 tr Abar (+ the analytic start's terms); one block per slot
__global__ void k_rev_vbar(AdjArgs a, int n) {
    const int e = blockIdx.x;
    const AdjSlot& S = a.s[e];
    const EnergyDev& d = a.ed[e];
    if (!d.live) return;
    const int Np = S.Np;
    const size_t np2 = (size_t)Np * Np;
    __shared__ double red[33];
    double t = 0.0;
    for (int i = threadIdx.x; i < Np; i += blockDim.x) t += S.SB2[i + (size_t)i * Np];
    double trS = block_sum(t, red);
    double cS = 0.0, cA = 0.0;
    if (n < a.stab_n) {
        const bool shS = d.stabd[2 * n + 1] != 0.0, shA = d.stabd[2 * n] != 0.0;
        cS = shS ? trS : 0.0;                  // Sbar -= tr(Sbar) P_S
        cA = shA ? trS - cS : 0.0;             // Abar -= tr(Abar) P_A, tr(Abar) = tr(Sbar) - cS
        if (cS != 0.0 || cA != 0.0) {
            const double* PS = S.PS + (size_t)n * np2;
            const double* PA = S.PA + (size_t)n * np2;
            for (size_t idx = threadIdx.x; idx < np2; idx += blockDim.x)
                S.SB2[idx] -= cS * PS[idx] + cA * PA[idx];
        }
    }
    if (threadIdx.x == 0) {
        S.vtr[n] += -a.h2_6 * (trS - cS - cA);
        if (n < a.n_start && n >= 1) {
            double s0 = 0.0, s1 = 0.0;
            for (int mu = 0; mu < Np; ++mu) { s0 += S.ab[mu]; s1 += S.ab[Np + mu]; }
            S.vtr[n] += s0;
            S.vtr[n + 1] += s1;
        }
    }
}

// vfull[n] += sum over slots of dJ/dV(n) (and the analytic start's diagonal
// terms at n and n + 1); slots in order, so the sum is deterministic
__global__ void k_rev_vfull(AdjArgs a, int n) {
    const size_t np2 = (size_t)a.Np_max * a.Np_max;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < np2; idx += (size_t)gridDim.x * blockDim.x) {
        const int r = (int)(idx % a.Np_max), c = (int)(idx / a.Np_max);
        double v = 0.0, v1 = 0.0;
        for (int e = 0; e < a.count; ++e) {
            const AdjSlot& S = a.s[e];
            if (!a.ed[e].live || r >= S.Np || c >= S.Np) continue;
            v += -a.h2_6 * S.SB2[r + (size_t)c * S.Np];
            if (r == c && n >= 1 && n < a.n_start) {
                v += S.ab[r];
                v1 += S.ab[S.Np + r];
            }
        }
        a.vfull[(size_t)n * np2 + idx] += v;
        if (v1 != 0.0) a.vfull[(size_t)(n + 1) * np2 + idx] += v1;
    }
}

// cyclic Jacobi eigen-decomposition of a symmetric n x n matrix (column-major,
// destroyed): eigenvalues w (ascending) and eigenvectors in the columns of Z
void jacobi_eig(std::vector<double>& A, int n, std::vector<double>& w, std::vector<double>& Z) {
    Z.assign((size_t)n * n, 0.0);
    for (int i = 0; i < n; ++i) Z[i + (size_t)i * n] = 1.0;
    auto at = [&](int i, int j) -> double& { return A[i + (size_t)j * n]; };
    double scale = 0.0;
    for (double x : A) scale = std::max(scale, std::fabs(x));
    for (int sweep = 0; sweep < 100; ++sweep) {
        double off = 0.0;
        for (int j = 0; j < n; ++j)
            for (int i = 0; i < j; ++i) off = std::max(off, std::fabs(at(i, j)));
        if (off <= 1e-17 * std::max(scale, 1e-300)) break;
        for (int p = 0; p < n - 1; ++p)
            for (int q = p + 1; q < n; ++q) {
                const double apq = at(p, q);
                if (std::fabs(apq) <= 1e-300) continue;
                const double theta = (at(q, q) - at(p, p)) / (2.0 * apq);
                const double tt = (theta >= 0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
                const double cs = 1.0 / std::sqrt(tt * tt + 1.0), sn = tt * cs;
                for (int k = 0; k < n; ++k) {           // columns p, q
                    const double akp = at(k, p), akq = at(k, q);
                    at(k, p) = cs * akp - sn * akq;
                    at(k, q) = sn * akp + cs * akq;
                }
                for (int k = 0; k < n; ++k) {           // rows p, q
                    const double apk = at(p, k), aqk = at(q, k);
                    at(p, k) = cs * apk - sn * aqk;
                    at(q, k) = sn * apk + cs * aqk;
                }
                for (int k = 0; k < n; ++k) {
                    const double zkp = Z[k + (size_t)p * n], zkq = Z[k + (size_t)q * n];
                    Z[k + (size_t)p * n] = cs * zkp - sn * zkq;
                    Z[k + (size_t)q * n] = sn * zkp + cs * zkq;
                }
            }
    }
    w.resize(n);
    for (int i = 0; i < n; ++i) w[i] = at(i, i);
}

// projector on the eigenvectors of the smallest eigenvalue of M (n x n,
// column-major), averaged over the eigenvalues within a relative 1e-9 of it
std::vector<double> min_eig_projector(std::vector<double> M, int n) {
    std::vector<double> w, Z;
    jacobi_eig(M, n, w, Z);
    const int i0 = (int)(std::min_element(w.begin(), w.end()) - w.begin());
    const double tol = 1e-9 * std::max(1.0, std::fabs(w[i0]));
    std::vector<int> cl;
    for (int i = 0; i < n; ++i)
        if (w[i] - w[i0] <= tol) cl.push_back(i);
    std::vector<double> P((size_t)n * n, 0.0);
    for (int k : cl)
        for (int c = 0; c < n; ++c)
            for (int r = 0; r < n; ++r) P[r + (size_t)c * n] += Z[r + (size_t)k * n] * Z[c + (size_t)k * n];
    for (double& x : P) x /= (double)cl.size();
    return P;
}

}  // namespace

// One adjoint batch: the forward scan (one phase group) with its checkpoints
// and window cotangents, ready for the reverse pass.
struct Adjoint {
    Scan sc;
    int segment = 256, nseg = 0, nwin = 0;
    std::vector<AdjSlot> slot;           // host copies (device pointers)
    DevBuf<AdjSlot> d_slot;
    DevBuf<double> arena;                // checkpoints, segment stores, work, cotangents
    DevBuf<double> stabd;                // 2 stab_n per slot
    std::vector<DevBuf<double>> proj;    // shift projectors PA, PS per distinct Np (pairs)
    std::vector<int> proj_Np;
    DevBuf<GemmEntry> gm;
    VBAt vb[2];                          // V/B at n (parity) for the reverse
    VBAt vbN;                            // V(N), B(N), Bs(N) for the small stages
    DevBuf<double> bswin;                // Bs(m) of the window steps inside the exchange region
    int n_energy = 0;
    std::vector<int> slot_of;            // submission order -> slot
    bool reversed = false;
};

namespace {

// device location of Rinv(n) outside any segment (rinv_at with in_seg false)
double* rinv_home(const BatchDev& b, const EnergyDev& d, int n) {
    const size_t nt2 = (size_t)d.Nt * d.Nt;
    return n >= b.n_s ? d.tailR + (size_t)(n - b.n_s) * nt2 : ((n & 1) ? d.Rinv1 : d.Rinv0);
}

int adj_projectors(Adjoint& A, int Np, const double** out_PA, const double** out_PS) {
    Scan& sc = A.sc;
    const BatchDev& b = sc.b;
    cudaStream_t s = sc.ctx->stream;
    for (size_t i = 0; i < A.proj_Np.size(); ++i)
        if (A.proj_Np[i] == Np) {
            *out_PA = A.proj[2 * i].p;
            *out_PS = A.proj[2 * i + 1].p;
            return SCATT_OK;
        }
    const size_t np2 = (size_t)Np * Np;
    const int ns = b.stab_n;
    std::vector<double> PA(std::max<size_t>(1, ns * np2), 0.0), PS(std::max<size_t>(1, ns * np2), 0.0);
    VBAt vb;
    SCATT_TRY(vb.alloc(b));
    const int Npm = b.Np_max, Nf = b.Nf;
    std::vector<double> V((size_t)Npm * Npm), B((size_t)Npm * std::max(1, Nf)), Bs((size_t)Npm * std::max(1, Nf));
    for (int n = 0; n < ns; ++n) {
        vb.build(b, n, s);
        SCATT_CUDA_TRY(cudaMemcpyAsync(V.data(), vb.V.p, V.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
        SCATT_CUDA_TRY(cudaMemcpyAsync(B.data(), vb.B.p, B.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
        SCATT_CUDA_TRY(cudaMemcpyAsync(Bs.data(), vb.Bs.p, Bs.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
        SCATT_CUDA_TRY(cudaStreamSynchronize(s));
        // the shifts compare c + lambda_min(-h^2/6 V) and c + dA + lambda_min(-h^2/6 V - Bs B^T):
        // the identity terms move no eigenvector
        std::vector<double> M(np2);
        for (int c = 0; c < Np; ++c)
            for (int r = 0; r < Np; ++r) M[r + (size_t)c * Np] = -b.h2_6 * V[r + (size_t)c * Npm];
        const auto pa = min_eig_projector(M, Np);
        std::copy(pa.begin(), pa.end(), PA.begin() + n * np2);
        if (n < b.n_tr && Nf > 0) {
            for (int c = 0; c < Np; ++c)
                for (int r = 0; r < Np; ++r) {
                    double acc = 0.0;
                    for (int f = 0; f < Nf; ++f) acc += Bs[r + (size_t)f * Npm] * B[c + (size_t)f * Npm];
                    M[r + (size_t)c * Np] = -b.h2_6 * V[r + (size_t)c * Npm] - acc;
                }
            // the device forms Bs B^T symmetric (lower tiles mirrored)
            for (int c = 0; c < Np; ++c)
                for (int r = 0; r < c; ++r) M[r + (size_t)c * Np] = M[c + (size_t)r * Np];
            const auto ps = min_eig_projector(M, Np);
            std::copy(ps.begin(), ps.end(), PS.begin() + n * np2);
        }
    }
    A.proj_Np.push_back(Np);
    A.proj.emplace_back();
    SCATT_TRY(upload_vec(A.proj.back(), PA, s));
    A.proj.emplace_back();
    SCATT_TRY(upload_vec(A.proj.back(), PS, s));
    SCATT_CUDA_TRY(cudaStreamSynchronize(s));
    *out_PA = A.proj[A.proj.size() - 2].p;
    *out_PS = A.proj.back().p;
    return SCATT_OK;
}

AdjArgs adj_args(Adjoint& A) {
    const BatchDev& b = A.sc.b;
    const ScanTables& t = *A.sc.ctx->tab;
    AdjArgs a{};
    a.s = A.d_slot.p;
    a.ed = A.sc.d_ed.p;
    a.gm = A.gm.p;
    a.Ctab = t.Ctab.p;
    a.l_of_mu = t.d_l_of_mu.p;
    a.count = A.sc.slots;
    a.K = b.Krows;
    a.Nf = b.Nf;
    a.Np_max = b.Np_max;
    a.n_start = b.n_start;
    a.n_tr = b.n_tr;
    a.n_pts = b.n_pts;
    a.n_s = b.n_s;
    a.N = b.N;
    a.stab_n = b.stab_n;
    a.dr = b.dr;
    a.h2_6 = b.h2_6;
    return a;
}

}  // namespace

// Forward scan of n energies (one group, every slot live) keeping the
// checkpoints; post stages as scatt_solve_batch (results into `out`, rows in
// submission order).
int adj_forward(Context& ctx, const scatt_solve_opts& o_in, int n, const double* E, const int* lc, int segment,
                const scatt_outputs* out, Adjoint& A) {
    ScanTables& t = *ctx.tab;
    cudaStream_t s = ctx.stream;
    if (n < 1 || segment < SCHUR_CHUNK || segment % SCHUR_CHUNK) {
        set_last_error("scatt_adjoint_forward: need n_energy >= 1 and a segment that is a positive multiple of " +
                       std::to_string(SCHUR_CHUNK));
        return SCATT_ERR_ARG;
    }
    int l_cap = 0;
    for (int e = 0; e < n; ++e) l_cap = std::max(l_cap, lc ? lc[e] : t.l_max);
    scatt_solve_opts o = o_in;
    o.use_graphs = 0;
    o.keep_window = 1;                 // the small stages read the window store
    Scan& sc = A.sc;
    SCATT_TRY(scan_open(ctx, o, n, 1, l_cap, sc));
    // The gradients keep the general inverse.  d sigma / d alpha is a sum with much cancellation of
    // its terms, which shows any change of rounding: from the general inverse to the sweep it moved, over
    // 40 sets of energies at N_t 196, by 2e-11 of itself in the median and by more than 1e-9 in three (two
    // blockings of the general inverse differ as much), and gradients are compared with earlier ones.  The
    // forward's K, A, B and D are therefore those of a solve under the general inverse, bit for bit, and of the
    // default solve bit for bit up to order 64 and to rounding above.
    sc.general = true;
    const BatchDev& b = sc.b;
    const int K = b.Krows, Nf = b.Nf, N = b.N;
    A.segment = segment;
    A.nseg = (N + segment - 1) / segment;            // segments [a, min(a + segment, N)), a < N
    A.nwin = N - b.n_s;                              // window steps n_s .. N - 1
    A.n_energy = n;
    for (int e = 0; e < n; ++e) sc.queue.push_back(Job{E[e], lc ? lc[e] : t.l_max, e});
    sc.submitted = n;
    SCATT_TRY(load_group(sc, 0));
    A.slot_of.assign(n, -1);
    for (int e = 0; e < n; ++e) A.slot_of[sc.job_of[e]] = e;
    // ---- arena: per slot checkpoints, segment stores, work and cotangents
    auto al = [](size_t c) { return (c + 31) & ~size_t(31); };
    std::vector<size_t> per(n);
    size_t total = 0;
    for (int e = 0; e < n; ++e) {
        const size_t Np = sc.ed[e].Np, Nt = sc.ed[e].Nt, np2 = Np * Np, nt2 = Nt * Nt, seg = segment;
        per[e] = A.nseg * (al(nt2) + al(K * Nt)) + al(seg * nt2) + al(seg * np2) + al(seg * K * Nt) + 4 * al(nt2) +
                 2 * al(K * Nt) + al(Np * std::max(1, Nf)) + 4 * al(np2) + al((size_t)A.nwin * nt2) +
                 al((size_t)A.nwin * np2) + al(2 * Np) + al(t.Nr + 1);
        total += per[e];
    }
    SCATT_TRY(A.arena.alloc(total));
    SCATT_CUDA_TRY(cudaMemsetAsync(A.arena.p, 0, total * sizeof(double), s));
    SCATT_TRY(A.stabd.alloc((size_t)n * 2 * std::max(1, b.stab_n)));
    SCATT_CUDA_TRY(cudaMemsetAsync(A.stabd.p, 0, A.stabd.n * sizeof(double), s));
    A.slot.assign(n, AdjSlot{});
    double* p = A.arena.p;
    auto take = [&p, &al](size_t c) { double* r = p; p += al(c); return r; };
    for (int e = 0; e < n; ++e) {
        EnergyDev& d = sc.ed[e];
        AdjSlot& S = A.slot[e];
        const size_t Np = d.Np, Nt = d.Nt, np2 = Np * Np, nt2 = Nt * Nt, seg = segment;
        S.Np = d.Np;
        S.Nt = d.Nt;
        S.ckR = take(A.nseg * al(nt2));
        S.ckG = take(A.nseg * al(K * Nt));
        d.segR = take(seg * nt2);
        d.segS = take(seg * np2);
        d.segH = take(seg * K * Nt);
        S.RB = take(nt2); S.T1 = take(nt2); S.T2 = take(nt2); S.WB = take(nt2);
        S.GB0 = take(K * Nt); S.GB1 = take(K * Nt);
        S.U = take(Np * std::max(1, Nf));
        S.SBi = take(np2); S.SBs = take(np2); S.SB = take(np2); S.SB2 = take(np2);
        S.RBw = take((size_t)A.nwin * nt2);
        S.SBw = take((size_t)A.nwin * np2);
        S.ab = take(2 * Np);
        S.vtr = take(t.Nr + 1);
        d.seg_lo = d.seg_hi = 0;
        d.stabd = A.stabd.p + (size_t)e * 2 * std::max(1, b.stab_n);
        SCATT_TRY(adj_projectors(A, d.Np, &S.PA, &S.PS));
    }
    SCATT_CUDA_TRY(cudaMemcpyAsync(sc.d_ed.p, sc.ed.data(), n * sizeof(EnergyDev), cudaMemcpyHostToDevice, s));
    SCATT_TRY(upload_vec(A.d_slot, A.slot, s));
    SCATT_TRY(A.gm.alloc((size_t)G_NUM * n));
    // ---- the sweep, with a checkpoint at every segment start a: Rinv(a-1), G(a-1)^T
    while (sc.grp[0].n0 >= 0) {
        const int next = sc.grp[0].n0 + sc.grp[0].C;
        SCATT_TRY(run_chunk(sc, nullptr));
        if (next % segment == 0 && next < N) {
            const int si = next / segment;
            for (int e = 0; e < n; ++e) {
                const EnergyDev& d = sc.ed[e];
                const size_t nt2 = (size_t)d.Nt * d.Nt;
                SCATT_CUDA_TRY(cudaMemcpyAsync(A.slot[e].ckR + si * al(nt2), rinv_home(b, d, next - 1),
                                               nt2 * sizeof(double), cudaMemcpyDeviceToDevice, s));
                SCATT_CUDA_TRY(cudaMemcpyAsync(A.slot[e].ckG + si * al((size_t)K * d.Nt), (next & 1) ? d.G1 : d.G0,
                                               (size_t)K * d.Nt * sizeof(double), cudaMemcpyDeviceToDevice, s));
            }
        }
    }
    // ---- post stages (slots keep their energies for the reverse pass)
    std::vector<int> sel(n);
    std::vector<long> rows(n);
    for (int e = 0; e < n; ++e) { sel[e] = e; rows[e] = sc.job_of[e]; }
    int first = SCATT_OK;
    std::string msg;
    SCATT_TRY(post_slots(sc, sel, rows, out, &first, &msg));
    sc.grp[0].n0 = -1;
    // ---- what the small stages read besides the window store: V(N), B(N), Bs(N); Bs of window steps
    SCATT_TRY(A.vbN.alloc(b));
    A.vbN.build(b, N, s);
    int nwx = 0;
    for (int m = b.n_s; m < N; ++m) nwx += (m < b.n_tr && Nf > 0) ? 1 : 0;
    SCATT_TRY(A.vb[0].alloc(b));
    SCATT_TRY(A.vb[1].alloc(b));
    if (nwx > 0) {
        const size_t sl = (size_t)b.Np_max * Nf;
        SCATT_TRY(A.bswin.alloc((size_t)A.nwin * sl));
        SCATT_CUDA_TRY(cudaMemsetAsync(A.bswin.p, 0, A.bswin.n * sizeof(double), s));
        for (int m = b.n_s; m < N; ++m)
            if (m < b.n_tr) {
                A.vb[0].build(b, m, s);
                SCATT_CUDA_TRY(cudaMemcpyAsync(A.bswin.p + (size_t)(m - b.n_s) * sl, A.vb[0].Bs.p, sl * sizeof(double),
                                               cudaMemcpyDeviceToDevice, s));
            }
    }
    SCATT_CUDA_TRY(cudaStreamSynchronize(s));
    if (first != SCATT_OK) set_last_error(msg);
    return first;
}

// The reverse pass: per segment, last to first, recompute it from its
// checkpoint, then walk its steps backward.  vtr_host: n_energy x (Nr)
// tr dJ/dV(n) in submission order; vfull (device, may be null):
// [Nr][Np_max][Np_max] += dJ/dV(n) summed over the energies.
int adj_reverse(Adjoint& A, double* vtr_host, double* vfull) {
    Scan& sc = A.sc;
    BatchDev& b = sc.b;
    cudaStream_t s = sc.ctx->stream;
    const int n = sc.slots, N = b.N, K = b.Krows, seg = A.segment;
    auto al = [](size_t c) { return (c + 31) & ~size_t(31); };
    if (A.reversed) {
        set_last_error("scatt_adjoint_reverse: the pass has run; run the forward again");
        return SCATT_ERR_STATE;
    }
    A.reversed = true;
    AdjArgs args = adj_args(A);
    args.vfull = vfull;
    // RB(N-1) starts at zero; Gbar(N-1)^T is the caller's dJ/dG(N-1)^T (buffer of parity N-1)
    for (int e = 0; e < n; ++e)
        SCATT_CUDA_TRY(cudaMemsetAsync(A.slot[e].RB, 0, (size_t)A.slot[e].Nt * A.slot[e].Nt * sizeof(double), s));
    A.vb[N & 1].build(b, N, s);                       // V(n + 1) for the first step n = N - 1
    const int Ntc = sc.Nt_cap, Npc = sc.Np_cap, Nf = b.Nf;
    auto gemm = [&](int which, int M, int Nn, int opA, int opB) {
        return gemm_batched(A.gm.p + (size_t)which * n, n, M, Nn, opA, opB, s);
    };
    const dim3 eg(64, n);
    for (int si = A.nseg - 1; si >= 0; --si) {
        const int a = si * seg, bnd = std::min(a + seg, N);
        // ---- recompute [a, bnd) from the checkpoint into the segment stores
        for (int e = 0; e < n; ++e) {
            EnergyDev& d = sc.ed[e];
            const size_t nt2 = (size_t)d.Nt * d.Nt, kn = (size_t)K * d.Nt;
            if (a >= 1) {
                SCATT_CUDA_TRY(cudaMemcpyAsync(rinv_home(b, d, a - 1), A.slot[e].ckR + si * al(nt2),
                                               nt2 * sizeof(double), cudaMemcpyDeviceToDevice, s));
                SCATT_CUDA_TRY(cudaMemcpyAsync(d.segH, A.slot[e].ckG + si * al(kn), kn * sizeof(double),
                                               cudaMemcpyDeviceToDevice, s));
            } else {
                SCATT_CUDA_TRY(cudaMemsetAsync(d.segH, 0, kn * sizeof(double), s));
            }
            d.seg_lo = a;
            d.seg_hi = bnd;
        }
        SCATT_CUDA_TRY(cudaMemcpyAsync(sc.d_ed.p, sc.ed.data(), n * sizeof(EnergyDev), cudaMemcpyHostToDevice, s));
        b.n_stop = bnd;
        k_set_group<<<1, 1, 0, s>>>(b, 0, a);
        SCATT_COUNT_LAUNCH(1);
        sc.grp[0].n0 = a;
        sc.grp[0].C = std::min(SCHUR_CHUNK, bnd - a);
        while (sc.grp[0].n0 >= 0) SCATT_TRY(run_chunk(sc, nullptr));
        sc.grp[0].n0 = -1;
        // ---- the steps of the segment, backward
        args.seg_lo = a;
        for (int m = bnd - 1; m >= a; --m) {
            VBAt& vc = A.vb[m & 1];
            vc.build(b, m, s);
            args.Bs = vc.Bs.p;
            args.Vn = vc.V.p;
            args.Vn1 = A.vb[(m + 1) & 1].V.p;
            const bool exch = m < b.n_tr && Nf > 0;
            const bool win = m >= b.n_s && m <= N - 1;
            k_prep_rev<<<cdiv(n, 64), 64, 0, s>>>(args, m);
            SCATT_COUNT_LAUNCH(1);
            if (win) { k_rev_window<<<eg, TPB, 0, s>>>(args, m); SCATT_COUNT_LAUNCH(1); }
            SCATT_TRY(gemm(G_HG, Ntc, Ntc, 1, 0));
            SCATT_TRY(gemm(G_HB, K, Ntc, 0, 0));
            if (m >= b.n_start) {
                k_rev_sym<<<eg, TPB, 0, s>>>(args, 0);
                SCATT_COUNT_LAUNCH(1);
                SCATT_TRY(gemm(G_X1, Ntc, Ntc, 0, 0));
                SCATT_TRY(gemm(G_X2, Ntc, Ntc, 0, 0));
                k_rev_wb<<<eg, TPB, 0, s>>>(args, 1);
                SCATT_COUNT_LAUNCH(1);
            } else {
                k_rev_analytic<<<dim3(cdiv(Npc, 128), n), 128, 0, s>>>(args, m);
                SCATT_COUNT_LAUNCH(1);
                k_rev_wb<<<eg, TPB, 0, s>>>(args, 0);
                SCATT_COUNT_LAUNCH(1);
            }
            if (m < b.n_pts) SCATT_TRY(gemm(G_CH, Npc, Ntc, 1, 0));
            k_rev_sbi<<<eg, TPB, 0, s>>>(args, m, exch ? 1 : 0, win ? 1 : 0);
            SCATT_COUNT_LAUNCH(1);
            if (exch) {
                SCATT_TRY(gemm(G_U, Npc, Nf, 0, 0));
                SCATT_TRY(gemm(G_S1, Npc, Npc, 0, 1));
                SCATT_TRY(gemm(G_S2, Npc, Npc, 0, 0));
            }
            k_rev_sym<<<eg, TPB, 0, s>>>(args, 1);
            SCATT_COUNT_LAUNCH(1);
            SCATT_TRY(gemm(G_Y1, Npc, Npc, 0, 0));
            SCATT_TRY(gemm(G_Y2, Npc, Npc, 0, 0));
            k_rev_vbar<<<n, TPB, 0, s>>>(args, m);
            SCATT_COUNT_LAUNCH(1);
            if (vfull) {
                k_rev_vfull<<<cdiv((long)b.Np_max * b.Np_max, TPB), TPB, 0, s>>>(args, m);
                SCATT_COUNT_LAUNCH(1);
            }
            SCATT_CUDA_TRY(cudaGetLastError());
        }
    }
    // segment mode off again
    for (int e = 0; e < n; ++e) sc.ed[e].seg_lo = sc.ed[e].seg_hi = 0;
    SCATT_CUDA_TRY(cudaMemcpyAsync(sc.d_ed.p, sc.ed.data(), n * sizeof(EnergyDev), cudaMemcpyHostToDevice, s));
    b.n_stop = b.Nr;
    if (vtr_host) {
        for (int i = 0; i < A.n_energy; ++i) {
            const int e = A.slot_of[i];
            SCATT_CUDA_TRY(cudaMemcpyAsync(vtr_host + (size_t)i * b.Nr, A.slot[e].vtr, b.Nr * sizeof(double),
                                           cudaMemcpyDeviceToHost, s));
        }
    }
    SCATT_CUDA_TRY(cudaStreamSynchronize(s));
    return SCATT_OK;
}

// ---------------------------------------------------------------- psi sweep
// BackPropagator::run (BackPropagator.cpp:533-703) with get_psi (:760-802)
// over any range [n_lo, n_hi) of the grid, for a lock-step batch of
// energies.  The forward sweep keeps R^-1(a - 1) at every segment start a;
// the post stages leave Z_N (the outer boundary, BackPropagator.cpp:127-197)
// in the post buffers.  The sweep then walks back from N - 1: each
// segment's Sinv(n) and R^-1(n) are recomputed from its checkpoint into the
// segment stores, and Z_n = R^-1(n) Z_{n+1}, psi(n) = (W^-1(n) Z_n)_psi
// (WInverseOperator.cpp:75-200: rhs = Z_psi - Bs(n) Z_f and psi = Sinv(n) rhs
// inside the exchange region, Sinv(n) Z_psi past it) -- the arithmetic of
// the post stages' window sweep.  A segment's psi goes to one of two device
// staging slabs (Np_max^2 per point, zero outside the energy's block) and
// from there to the caller's host buffer on a copy stream, so with
// page-locked host memory the copies of one segment overlap the
// recomputation of the next.
namespace {

struct StreamGuard {
    cudaStream_t s = nullptr;
    ~StreamGuard() { if (s) cudaStreamDestroy(s); }
};
struct EventGuard {
    cudaEvent_t e = nullptr;
    ~EventGuard() { if (e) cudaEventDestroy(e); }
};

}  // namespace

int psi_sweep(Context& ctx, const scatt_solve_opts& o_in, int n, const double* E, const int* lc, int segment,
              int n_lo, int n_hi, const scatt_outputs* out, double* psi_host) {
    ScanTables& t = *ctx.tab;
    cudaStream_t s = ctx.stream;
    if (n < 1 || segment < SCHUR_CHUNK || segment % SCHUR_CHUNK || n_lo < 0 || n_hi > t.Nr || n_lo >= n_hi ||
        !psi_host || !out) {
        set_last_error("scatt_psi_sweep: need n_energy >= 1, a segment that is a positive multiple of " +
                       std::to_string(SCHUR_CHUNK) + ", 0 <= n_lo < n_hi <= Nr and the output buffers");
        return SCATT_ERR_ARG;
    }
    int l_cap = 0;
    for (int e = 0; e < n; ++e) l_cap = std::max(l_cap, lc ? lc[e] : t.l_max);
    scatt_solve_opts o = o_in;
    o.use_graphs = 0;
    o.keep_window = 0;                   // the fit accumulates forward: no window store
    Scan sc;
    SCATT_TRY(scan_open(ctx, o, n, 1, l_cap, sc));
    BatchDev& b = sc.b;
    const int K = b.Krows, Nf = b.Nf, N = b.N, Npm = b.Np_max;
    const size_t npm2 = (size_t)Npm * Npm;
    const int nseg = (N + segment - 1) / segment;          // segments [a, min(a + segment, N)), a < N
    const size_t R = (size_t)(n_hi - n_lo);
    for (int e = 0; e < n; ++e) sc.queue.push_back(Job{E[e], lc ? lc[e] : t.l_max, e});
    sc.submitted = n;
    SCATT_TRY(load_group(sc, 0));
    std::vector<int> slot_of(n, -1);
    for (int e = 0; e < n; ++e) slot_of[sc.job_of[e]] = e;
    // ---- per slot: checkpoints, segment stores, the second Z buffer, rhs, staging
    struct PsiSlot {
        double *ck, *Z1, *rhs, *stg[2], *top;
    };
    std::vector<PsiSlot> ps(n);
    auto al = [](size_t c) { return (c + 31) & ~size_t(31); };
    const size_t seg = segment;
    size_t total = 0;
    for (int e = 0; e < n; ++e) {
        const size_t Np = sc.ed[e].Np, Nt = sc.ed[e].Nt;
        total += nseg * al(Nt * Nt) + al(seg * Nt * Nt) + al(seg * Np * Np) + al(seg * K * Nt) + al(Nt * Np) +
                 al(Np * Np) + 2 * al(seg * npm2) + al(npm2);
    }
    DevBuf<double> arena;
    SCATT_TRY(arena.alloc(total));
    SCATT_CUDA_TRY(cudaMemsetAsync(arena.p, 0, total * sizeof(double), s));
    double* p = arena.p;
    auto take = [&p, &al](size_t c) { double* r = p; p += al(c); return r; };
    for (int e = 0; e < n; ++e) {
        EnergyDev& d = sc.ed[e];
        const size_t Np = d.Np, Nt = d.Nt;
        ps[e].ck = take(nseg * al(Nt * Nt));
        d.segR = take(seg * Nt * Nt);
        d.segS = take(seg * Np * Np);
        d.segH = take(seg * K * Nt);
        ps[e].Z1 = take(Nt * Np);
        ps[e].rhs = take(Np * Np);
        ps[e].stg[0] = take(seg * npm2);
        ps[e].stg[1] = take(seg * npm2);
        ps[e].top = take(npm2);
        d.seg_lo = d.seg_hi = 0;
    }
    SCATT_CUDA_TRY(cudaMemcpyAsync(sc.d_ed.p, sc.ed.data(), n * sizeof(EnergyDev), cudaMemcpyHostToDevice, s));
    // ---- the forward sweep, with R^-1(a - 1) kept at every segment start a (ping-pong buffer of a - 1:
    // the window store is off)
    while (sc.grp[0].n0 >= 0) {
        const int next = sc.grp[0].n0 + sc.grp[0].C;
        SCATT_TRY(run_chunk(sc, nullptr));
        if (next % segment == 0 && next < N) {
            const int si = next / segment;
            for (int e = 0; e < n; ++e) {
                const EnergyDev& d = sc.ed[e];
                const size_t nt2 = (size_t)d.Nt * d.Nt;
                SCATT_CUDA_TRY(cudaMemcpyAsync(ps[e].ck + si * al(nt2), ((next - 1) & 1) ? d.Rinv1 : d.Rinv0,
                                               nt2 * sizeof(double), cudaMemcpyDeviceToDevice, s));
            }
        }
    }
    // ---- post stages: K, the fit, the dipoles into `out`; Z_N stays in P[e].Z0, psi(N) in P[e].psibc
    std::vector<int> sel(n);
    std::vector<long> rows(n);
    for (int e = 0; e < n; ++e) { sel[e] = e; rows[e] = sc.job_of[e]; }
    int first = SCATT_OK;
    std::string msg;
    SCATT_TRY(post_slots(sc, sel, rows, out, &first, &msg));
    sc.grp[0].n0 = -1;
    StreamGuard cs;                       // device-to-host copies of the staging slabs
    SCATT_CUDA_TRY(cudaStreamCreateWithFlags(&cs.s, cudaStreamNonBlocking));
    EventGuard ev_done[2], ev_copied[2];
    for (int i = 0; i < 2; ++i) {
        SCATT_CUDA_TRY(cudaEventCreateWithFlags(&ev_done[i].e, cudaEventDisableTiming));
        SCATT_CUDA_TRY(cudaEventCreateWithFlags(&ev_copied[i].e, cudaEventDisableTiming));
    }
    bool pending[2] = {false, false};
    if (n_lo <= N && N < n_hi) {          // psi(N) = the boundary value
        std::vector<CopyEntry> ct(n);
        for (int e = 0; e < n; ++e) {
            const int Np = sc.ed[e].Np;
            ct[e] = CopyEntry{sc.P[e].psibc, ps[e].top, Np, Np, Np, Npm, 1.0};
        }
        SCATT_TRY(sc.L.copy(ct));
        for (int i = 0; i < n; ++i)
            SCATT_CUDA_TRY(cudaMemcpyAsync(psi_host + ((size_t)i * R + (size_t)(N - n_lo)) * npm2, ps[slot_of[i]].top,
                                           npm2 * sizeof(double), cudaMemcpyDeviceToHost, s));
    }
    // ---- the backward sweep, segment by segment, last to first, down to n_lo
    const int Ntc = sc.Nt_cap, Npc = sc.Np_cap;
    std::vector<double*> zc(n), zn(n);
    for (int e = 0; e < n; ++e) { zc[e] = sc.P[e].Z0; zn[e] = ps[e].Z1; }
    const size_t ne = seg * (size_t)n;
    DevBuf<GemmEntry> dmz, dmr, dmp;
    DevBuf<CopyEntry> dcr;
    SCATT_TRY(dmz.alloc(ne));
    SCATT_TRY(dmr.alloc(ne));
    SCATT_TRY(dmp.alloc(ne));
    SCATT_TRY(dcr.alloc(ne));
    std::vector<GemmEntry> hmz(ne), hmr(ne), hmp(ne);
    std::vector<CopyEntry> hcr(ne, CopyEntry{nullptr, nullptr, 0, 0, 1, 1, 0.0});
    for (int si = nseg - 1; si >= 0; --si) {
        const int a = si * segment, bnd = std::min(a + segment, N);
        if (bnd <= n_lo) break;
        // recompute Sinv(n), R^-1(n) of [a, bnd) from the checkpoint into the segment stores
        for (int e = 0; e < n; ++e) {
            EnergyDev& d = sc.ed[e];
            const size_t nt2 = (size_t)d.Nt * d.Nt;
            if (a >= 1)
                SCATT_CUDA_TRY(cudaMemcpyAsync(((a - 1) & 1) ? d.Rinv1 : d.Rinv0, ps[e].ck + si * al(nt2),
                                               nt2 * sizeof(double), cudaMemcpyDeviceToDevice, s));
            d.seg_lo = a;
            d.seg_hi = bnd;
        }
        SCATT_CUDA_TRY(cudaMemcpyAsync(sc.d_ed.p, sc.ed.data(), n * sizeof(EnergyDev), cudaMemcpyHostToDevice, s));
        b.n_stop = bnd;
        k_set_group<<<1, 1, 0, s>>>(b, 0, a);
        SCATT_COUNT_LAUNCH(1);
        sc.grp[0].n0 = a;
        sc.grp[0].C = std::min(SCHUR_CHUNK, bnd - a);
        while (sc.grp[0].n0 >= 0) SCATT_TRY(run_chunk(sc, nullptr));
        sc.grp[0].n0 = -1;
        // this segment's staging slab is free once its previous copies are done
        const int par = si & 1;
        if (pending[par]) {
            SCATT_CUDA_TRY(cudaStreamWaitEvent(s, ev_copied[par].e, 0));
            pending[par] = false;
        }
        // the entries of the segment's steps n = bnd - 1 .. max(a, n_lo), in launch order
        const int m_lo = std::max(a, n_lo);
        const int steps = bnd - m_lo;
        for (int k = 0; k < steps; ++k) {
            const int m = bnd - 1 - k;
            const bool exch = m < b.n_tr && Nf > 0;
            for (int e = 0; e < n; ++e) {
                const EnergyDev& d = sc.ed[e];
                const int Np = d.Np, Nt = d.Nt;
                const size_t i = (size_t)k * n + e;
                hmz[i] = GemmEntry{d.segR + (size_t)(m - a) * Nt * Nt, zc[e], zn[e], Nt, Np, Nt, Nt, Nt, Nt, 1.0, 0.0};
                const double* sinv = d.segS + (size_t)(m - a) * Np * Np;
                double* dst = ps[e].stg[par] + (size_t)(m - a) * npm2;
                if (exch) {
                    hcr[i] = CopyEntry{zn[e], ps[e].rhs, Np, Np, Nt, Np, 1.0};
                    hmr[i] = GemmEntry{sc.vb.Bs.p, zn[e] + Np, ps[e].rhs, Np, Np, Nf, Npm, Nt, Np, -1.0, 1.0};
                    hmp[i] = GemmEntry{sinv, ps[e].rhs, dst, Np, Np, Np, Np, Np, Npm, 1.0, 0.0};
                } else {
                    hmp[i] = GemmEntry{sinv, zn[e], dst, Np, Np, Np, Np, Nt, Npm, 1.0, 0.0};
                }
            }
            std::swap(zc, zn);
        }
        if (steps > 0) {
            const size_t cnt = (size_t)steps * n;
            SCATT_CUDA_TRY(cudaMemcpyAsync(dmz.p, hmz.data(), cnt * sizeof(GemmEntry), cudaMemcpyHostToDevice, s));
            SCATT_CUDA_TRY(cudaMemcpyAsync(dmr.p, hmr.data(), cnt * sizeof(GemmEntry), cudaMemcpyHostToDevice, s));
            SCATT_CUDA_TRY(cudaMemcpyAsync(dmp.p, hmp.data(), cnt * sizeof(GemmEntry), cudaMemcpyHostToDevice, s));
            SCATT_CUDA_TRY(cudaMemcpyAsync(dcr.p, hcr.data(), cnt * sizeof(CopyEntry), cudaMemcpyHostToDevice, s));
        }
        for (int k = 0; k < steps; ++k) {
            const int m = bnd - 1 - k;
            const bool exch = m < b.n_tr && Nf > 0;
            SCATT_TRY(gemm_batched(dmz.p + (size_t)k * n, n, Ntc, Npc, 0, 0, s));       // Z_m = R^-1(m) Z_{m+1}
            if (m >= n_hi) continue;
            if (exch) {
                sc.vb.build(b, m, s);                                                     // Bs(m)
                k_copy<<<dim3(64, n), TPB, 0, s>>>(dcr.p + (size_t)k * n);                // rhs = Z_psi
                SCATT_COUNT_LAUNCH(1);
                SCATT_TRY(gemm_batched(dmr.p + (size_t)k * n, n, Npc, Npc, 0, 0, s));   // rhs -= Bs(m) Z_f
            }
            SCATT_TRY(gemm_batched(dmp.p + (size_t)k * n, n, Npc, Npc, 0, 0, s));       // psi(m) = Sinv(m) rhs
        }
        SCATT_CUDA_TRY(cudaGetLastError());
        // rows [r0, r1) of the staging slab go to the host on the copy stream
        const int r0 = m_lo, r1 = std::min(bnd, n_hi);
        if (r1 > r0) {
            SCATT_CUDA_TRY(cudaEventRecord(ev_done[par].e, s));
            SCATT_CUDA_TRY(cudaStreamWaitEvent(cs.s, ev_done[par].e, 0));
            for (int i = 0; i < n; ++i)
                SCATT_CUDA_TRY(cudaMemcpyAsync(psi_host + ((size_t)i * R + (size_t)(r0 - n_lo)) * npm2,
                                               ps[slot_of[i]].stg[par] + (size_t)(r0 - a) * npm2,
                                               (size_t)(r1 - r0) * npm2 * sizeof(double), cudaMemcpyDeviceToHost,
                                               cs.s));
            SCATT_CUDA_TRY(cudaEventRecord(ev_copied[par].e, cs.s));
            pending[par] = true;
        }
    }
    for (int e = 0; e < n; ++e) sc.ed[e].seg_lo = sc.ed[e].seg_hi = 0;
    b.n_stop = b.Nr;
    SCATT_CUDA_TRY(cudaStreamSynchronize(s));
    SCATT_CUDA_TRY(cudaStreamSynchronize(cs.s));
    if (first != SCATT_OK) set_last_error(msg);
    return first;
}

}  // namespace scatt

// ================================================================ C ABI
using namespace scatt;

struct scatt_ctx {
    Context c;
};

struct scatt_scan {
    scatt_ctx* ctx = nullptr;
    Scan s;
};

extern "C" {

void scatt_default_opts(scatt_solve_opts* o) {
    if (!o) return;
    o->W_min = 0.001;
    o->stab_n_max = 60;
    o->shift_margin = 0.01;
    o->n_asym = 300;
    o->allow_closed_channels = 0;
    o->orthogonalize = 1;
    o->max_batch = 0;
    o->use_graphs = 0;
    o->diagnostics = 1;
    o->timing = 0;
    o->keep_window = 1;
}

int scatt_last_stats(scatt_ctx* ctx, double* out7) {
    if (!ctx || !out7) return SCATT_ERR_ARG;
    const SolveStats& st = ctx->c.stats;
    out7[0] = st.device_s;
    out7[1] = st.rinv_s;
    out7[2] = st.rinv_calls;
    out7[3] = (double)st.launches;
    out7[4] = st.sweep_s;
    out7[5] = st.post_s;
    out7[6] = st.rinv_flops;
    return SCATT_OK;
}

int scatt_ctx_create(int device, scatt_ctx** out) {
    if (!out) return SCATT_ERR_ARG;
    *out = nullptr;
    SCATT_TRY(require_device());
    SCATT_CUDA_TRY(cudaSetDevice(device));
    auto* c = new scatt_ctx();
    c->c.device = device;
    cudaError_t e = cudaStreamCreateWithFlags(&c->c.stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        delete c;
        set_last_error(std::string("cudaStreamCreate: ") + cudaGetErrorString(e));
        return SCATT_ERR_CUDA;
    }
    *out = c;
    return SCATT_OK;
}

int scatt_ctx_destroy(scatt_ctx* ctx) {
    if (!ctx) return SCATT_OK;
    cudaSetDevice(ctx->c.device);
    ctx->c.tab.reset();
    if (ctx->c.stream) cudaStreamDestroy(ctx->c.stream);
    delete ctx;
    return SCATT_OK;
}

int scatt_upload_static(scatt_ctx* ctx, const scatt_scan_desc* desc) {
    if (!ctx || !desc) return SCATT_ERR_ARG;
    return upload_static(ctx->c, *desc);
}

int scatt_scan_info(scatt_ctx* ctx, int* out5) {
    if (!ctx || !out5) return SCATT_ERR_ARG;
    if (!ctx->c.tab || !ctx->c.tab->ready) {
        set_last_error("scatt_scan_info: no scan uploaded");
        return SCATT_ERR_STATE;
    }
    const ScanTables& t = *ctx->c.tab;
    out5[0] = t.n_tr;
    out5[1] = t.Np_max;
    out5[2] = t.Nf;
    out5[3] = t.n_lambda;
    out5[4] = t.n_sigma;
    return SCATT_OK;
}

int scatt_solve_batch(scatt_ctx* ctx, int n_energy, const double* energies, const int* l_cont,
                      const scatt_solve_opts* opts, const scatt_outputs* outputs) {
    if (!ctx || n_energy < 0 || (n_energy > 0 && !energies) || !outputs) return SCATT_ERR_ARG;
    if (!ctx->c.tab || !ctx->c.tab->ready) {
        set_last_error("scatt_solve_batch: call scatt_upload_static first");
        return SCATT_ERR_STATE;
    }
    SCATT_CUDA_TRY(cudaSetDevice(ctx->c.device));
    scatt_solve_opts o;
    if (opts) o = *opts; else scatt_default_opts(&o);
    return solve_batch(ctx->c, o, n_energy, energies, l_cont, outputs);
}

int scatt_scan_open(scatt_ctx* ctx, const scatt_solve_opts* opts, int slots, int groups, int l_cont_max,
                    scatt_scan** out) {
    if (!ctx || !out) return SCATT_ERR_ARG;
    *out = nullptr;
    if (!ctx->c.tab || !ctx->c.tab->ready) {
        set_last_error("scatt_scan_open: call scatt_upload_static first");
        return SCATT_ERR_STATE;
    }
    SCATT_CUDA_TRY(cudaSetDevice(ctx->c.device));
    scatt_solve_opts o;
    if (opts) o = *opts; else scatt_default_opts(&o);
    const ScanTables& t = *ctx->c.tab;
    const int l_cap = l_cont_max < 0 ? t.l_max : l_cont_max;
    if (l_cap > t.l_max || std::min(l_cap, 10) != t.l_x) {
        set_last_error("scatt_scan_open: l_cont_max is outside the uploaded scan");
        return SCATT_ERR_ARG;
    }
    if (groups < 1 || groups > MAX_GROUPS) {
        set_last_error("scatt_scan_open: groups must be in [1, " + std::to_string(MAX_GROUPS) + "]");
        return SCATT_ERR_ARG;
    }
    if (slots <= 0) SCATT_TRY(slots_that_fit(ctx->c, o, l_cap, groups, &slots));
    if (groups > slots) groups = slots;
    auto* h = new scatt_scan();
    h->ctx = ctx;
    const int st = scan_open(ctx->c, o, slots, groups, l_cap, h->s);
    if (st != SCATT_OK) {
        delete h;
        return st;
    }
    ctx->c.stats = SolveStats{};
    *out = h;
    return SCATT_OK;
}

int scatt_scan_submit(scatt_scan* sc, int n, const double* energies, const int* l_cont) {
    if (!sc || n < 0 || (n > 0 && !energies)) return SCATT_ERR_ARG;
    const ScanTables& t = *sc->ctx->c.tab;
    SCATT_TRY(check_energies(t, n, energies, l_cont, "scatt_scan_submit"));
    for (int e = 0; e < n; ++e)
        if ((l_cont ? l_cont[e] : sc->s.l_cap) > sc->s.l_cap) {
            set_last_error("scatt_scan_submit: l_cont above the scan's l_cont_max");
            return SCATT_ERR_ARG;
        }
    for (int e = 0; e < n; ++e)
        sc->s.queue.push_back(Job{energies[e], l_cont ? l_cont[e] : sc->s.l_cap, sc->s.submitted++});
    return SCATT_OK;
}

int scatt_scan_step(scatt_scan* sc, const scatt_outputs* outputs, int capacity, int* n_done,
                    long long* index_out) {
    if (!sc || !outputs || !n_done) return SCATT_ERR_ARG;
    *n_done = 0;
    if (capacity < sc->s.slots) {
        set_last_error("scatt_scan_step: output capacity below the scan's slot count");
        return SCATT_ERR_ARG;
    }
    SCATT_CUDA_TRY(cudaSetDevice(sc->ctx->c.device));
    int first = SCATT_OK;
    std::string msg;
    std::vector<long> jobs;
    SCATT_TRY(scan_advance(sc->s, outputs, [](int, int i) { return (long)i; }, n_done, &jobs, &first, &msg));
    if (index_out)
        for (size_t i = 0; i < jobs.size(); ++i) index_out[i] = jobs[i];
    if (first != SCATT_OK) set_last_error(msg);
    return first;
}

int scatt_scan_pending(scatt_scan* sc, int* queued, int* in_flight) {
    if (!sc) return SCATT_ERR_ARG;
    if (queued) *queued = (int)sc->s.queue.size();
    if (in_flight) {
        int f = 0;
        for (auto& d : sc->s.ed) f += d.live;
        *in_flight = f;
    }
    return SCATT_OK;
}

int scatt_scan_shape(scatt_scan* sc, int* slots, int* groups) {
    if (!sc) return SCATT_ERR_ARG;
    if (slots) *slots = sc->s.slots;
    if (groups) *groups = sc->s.G;
    return SCATT_OK;
}

int scatt_scan_close(scatt_scan* sc) {
    if (!sc) return SCATT_OK;
    cudaSetDevice(sc->ctx->c.device);
    cudaStreamSynchronize(sc->ctx->c.stream);
    delete sc;
    return SCATT_OK;
}

// ---------------------------------------------------------------- adjoint
struct scatt_adjoint {
    scatt_ctx* ctx = nullptr;
    Adjoint a;
};

int scatt_set_polarization(scatt_ctx* ctx, double alpha, double r_c, int pol_form) {
    if (!ctx || !ctx->c.tab || !ctx->c.tab->ready) return SCATT_ERR_STATE;
    if (!(r_c > 0.0) || (pol_form != 0 && pol_form != 1) || !std::isfinite(alpha)) return SCATT_ERR_ARG;
    ScanTables& t = *ctx->c.tab;
    t.alpha_pol = alpha;
    t.r_c = r_c;
    t.pol_form = pol_form;
    t.stab.clear();            // the stability spectra follow V
    return SCATT_OK;
}

int scatt_set_potential_delta(scatt_ctx* ctx, const double* dV) {
    if (!ctx || !ctx->c.tab || !ctx->c.tab->ready) return SCATT_ERR_STATE;
    ctx->c.tab->dV = dV;
    ctx->c.tab->stab.clear();
    return SCATT_OK;
}

int scatt_adjoint_forward(scatt_ctx* ctx, const scatt_solve_opts* opts, int n_energy, const double* energies,
                          const int* l_cont, int segment, const scatt_outputs* outputs, scatt_adjoint** out) {
    if (!ctx || !energies || !out || n_energy < 1) return SCATT_ERR_ARG;
    if (!ctx->c.tab || !ctx->c.tab->ready) {
        set_last_error("scatt_adjoint_forward: upload the static inputs first");
        return SCATT_ERR_STATE;
    }
    SCATT_TRY(require_device());
    SCATT_CUDA_TRY(cudaSetDevice(ctx->c.device));
    SCATT_TRY(check_energies(*ctx->c.tab, n_energy, energies, l_cont, "scatt_adjoint_forward"));
    scatt_solve_opts o;
    if (opts) o = *opts;
    else scatt_default_opts(&o);
    auto* h = new scatt_adjoint();
    h->ctx = ctx;
    const int st = adj_forward(ctx->c, o, n_energy, energies, l_cont, segment, outputs, h->a);
    if (st != SCATT_OK && h->a.slot.empty()) {
        delete h;
        return st;
    }
    *out = h;
    return st;
}

int scatt_adjoint_view_of(scatt_adjoint* h, int i, scatt_adjoint_view* v) {
    if (!h || !v || i < 0 || i >= h->a.n_energy) return SCATT_ERR_ARG;
    const Adjoint& A = h->a;
    const BatchDev& b = A.sc.b;
    const ScanTables& t = *A.sc.ctx->tab;
    const int e = A.slot_of[i];
    const EnergyDev& d = A.sc.ed[e];
    const AdjSlot& S = A.slot[e];
    std::memset(v, 0, sizeof(*v));
    v->N = b.N;
    v->n_s = b.n_s;
    v->n_window = A.nwin;
    v->n_tr = b.n_tr;
    v->n_pts = b.n_pts;
    v->n_start = b.n_start;
    v->ne_fit = A.sc.ne_fit;
    v->Np = d.Np;
    v->Nt = d.Nt;
    v->Nf = b.Nf;
    v->Krows = b.Krows;
    v->Np_max = b.Np_max;
    v->l_cont = d.l_cont;
    v->E = d.E;
    v->Rwin = d.tailR;
    v->Swin = d.tailS;
    v->G_last = (b.N & 1) ? d.G1 : d.G0;
    v->RBwin = S.RBw;
    v->SBwin = S.SBw;
    v->GB_last = ((b.N - 1) & 1) ? S.GB1 : S.GB0;
    v->V_N = A.vbN.V.p;
    v->B_N = A.vbN.B.p;
    v->Bs_N = A.vbN.Bs.p;
    v->C_N = (b.N < b.n_pts) ? t.Ctab.p + (size_t)b.N * b.Krows * b.Np_max : nullptr;
    v->Bs_win = A.bswin.p;
    return SCATT_OK;
}

int scatt_adjoint_reverse(scatt_adjoint* h, double* vtr, double* vfull_device) {
    if (!h) return SCATT_ERR_ARG;
    SCATT_CUDA_TRY(cudaSetDevice(h->ctx->c.device));
    return adj_reverse(h->a, vtr, vfull_device);
}

int scatt_adjoint_close(scatt_adjoint* h) {
    if (!h) return SCATT_OK;
    cudaSetDevice(h->ctx->c.device);
    delete h;
    return SCATT_OK;
}

// ---------------------------------------------------------------- psi sweep
int scatt_psi_sweep(scatt_ctx* ctx, const scatt_solve_opts* opts, int n_energy, const double* energies,
                    const int* l_cont, int segment, int n_lo, int n_hi, const scatt_outputs* outputs,
                    double* psi_out) {
    if (!ctx || !energies || !outputs || !psi_out || n_energy < 1) {
        set_last_error("scatt_psi_sweep: null argument or no energies");
        return SCATT_ERR_ARG;
    }
    if (!ctx->c.tab || !ctx->c.tab->ready) {
        set_last_error("scatt_psi_sweep: upload the static inputs first");
        return SCATT_ERR_STATE;
    }
    SCATT_TRY(require_device());
    SCATT_CUDA_TRY(cudaSetDevice(ctx->c.device));
    SCATT_TRY(check_energies(*ctx->c.tab, n_energy, energies, l_cont, "scatt_psi_sweep"));
    scatt_solve_opts o;
    if (opts) o = *opts;
    else scatt_default_opts(&o);
    return psi_sweep(ctx->c, o, n_energy, energies, l_cont, segment, n_lo, n_hi, outputs, psi_out);
}

}  // extern "C"
