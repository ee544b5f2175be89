// FP64 (plain form) translation and evaluation kernels of the 2D Laurent FMM
// (reference src/FMM/fmm2D.cpp). Expansions are complex: multipole
//   a_k = sum_j q_j (z_j - z_c)^k                      (P2M, fmm2D.cpp:237-284)
// and local coefficients b_p, with the field at z taken as
//   E_x = Re F, E_y = -Im F,  F = sum of q/(z - z_j) terms.
//
// Stage map:
//   fmm2d_upward_direct  moments of every cell of at most 1024 particles
//                 straight from its particles (upward_direct2d), then M2M of
//                 the larger cells level by level in one cooperative launch
//                 (m2m_big_levels_coop, shift2d.cu), with an optional event
//                 between the two; fmm2D.cpp:237-284, 309-379.
//   fmm2d_upward  P2M of every active leaf, then M2M over all levels (p2m2d,
//                 m2m_levels_coop), for orders the direct form does not cover.
//   fmm2d_m2l_only  lists 2 and 4 of every cell at level >= 2 in FP64 with the
//                 49 precomputed list-2 operators (m2l2d_op, fmm2D.cpp:396-556),
//                 in small trees and at high orders; the list-2 M2L per parent
//                 is in m2l_f64.cu (plain form) and m2l_tc.cu (mixed forms).
//   fmm2d_l2l     the L2L level loop (fmm2D.cpp:587-651), where the leaves' local
//                 expansions straight from their ancestors' M2L parts
//                 (fmm2d_l2l_leaves, shift2d.cu) do not apply.
//   fmm2d_eval, fmm2d_m2p, fmm2d_eval_combine  M2P over list 3
//                 (fmm2D.cpp:1040-1066) and L2P (fmm2D.cpp:1076-1093), warp per
//                 leaf; the combine pass adds the near field and writes the
//                 output in the caller's order.
//   fmm2d_p2p_f64, fmm2d_p2p_f32, fmm2d_p2p_potential  near field over list 1, j != i
//                 (fmm2D.cpp:135-179): FP64 (near2d_f64) for the plain form
//                 and the potential, packed FP32 tiles for the mixed forms.
#include "fmm2d.cuh"

#include <complex>
#include <vector>

namespace vpm {

namespace {

constexpr int W = kMaxP + 1;

int64_t binom_host(int n, int k, bool exact) {
    if (k > n) return 0;
    if (exact) {
        int64_t c = 1;
        for (int i = 1; i <= k; ++i) c = c * (n - k + i) / i;
        return c;
    }
    // The reference's binComb: n!/max(k,n-k)! in 32-bit int (wrapping), then
    // truncating divisions by min(k,n-k)!.
    int inv = n - k;
    int mx = inv > k ? inv : k, mn = inv > k ? k : inv;
    int32_t c = 1;
    for (int i = n; i > mx; --i) c = (int32_t)((uint32_t)c * (uint32_t)i);
    for (int i = mn; i > 1; --i) c /= i;
    return c;
}

// 1 / a for the FP64 near field: the hardware seed (about 23 correct bits)
// refined by one third-order step, y (1 + e + e^2) with e = 1 - a y, which
// leaves a relative error of order e^3 (below the double's own rounding), in
// three FMAs where two Newton steps take four.
__device__ __forceinline__ double rcp_nr(double a) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-a, y, 1.0);
    return fma(y, fma(e, e, e), y);
}


// ---- upward pass -----------------------------------------------------------

constexpr int kP2MWarps = 2;
constexpr int kAccPad = 33;  // padded lane stride of the P2M accumulators

// P2M, one warp per leaf: lane j takes particles j, j+32, ... and adds
// q (z - z_c)^k into its own shared-memory accumulator column k; the columns
// are then summed in a fixed order (deterministic).
__global__ void __launch_bounds__(32 * kP2MWarps)
p2m2d(Tree2D t, double2* __restrict__ a, int P, unsigned* err) {
    extern __shared__ double2 acc_sm[];
    if (fatal(err)) return;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    double2* acc = acc_sm + (size_t)wib * (P + 1) * kAccPad;
    const int nl = t.info->n_leaves;
    const int warps = gridDim.x * kP2MWarps;
    for (int li = blockIdx.x * kP2MWarps + wib; li < nl; li += warps) {
        const int c = t.leaf_cells[li];
        if (!(t.c_flags[c] & CELL_ACTIVE)) continue;
        for (int k = 0; k <= P; ++k) acc[k * kAccPad + lane] = make_double2(0.0, 0.0);
        const double zx = t.c_cx[c], zy = t.c_cy[c];
        const int lo = t.c_lo[c], hi = t.c_hi[c];
        for (int j = lo + lane; j < hi; j += 32) {
            if (!t.pact[j]) continue;
            const double2 w = make_double2(t.px[j] - zx, t.py[j] - zy);
            double2 wk = make_double2(t.pq[j], 0.0);
            for (int k = 0; k <= P; ++k) {
                double2* ak = &acc[k * kAccPad + lane];
                *ak = cadd(*ak, wk);
                wk = cmul(wk, w);
            }
        }
        __syncwarp();
        if (lane <= P) {
            double2 sum = make_double2(0.0, 0.0);
            for (int l = 0; l < 32; ++l) sum = cadd(sum, acc[lane * kAccPad + l]);
            a[(size_t)c * (P + 1) + lane] = sum;
        }
        __syncwarp();
    }
}

// Warps per block of the level kernels (M2M, L2L): the cooperative loops run
// one 256-thread block per SM, so a grid barrier has 148 arrivals.
constexpr int kLevelWarps = 8;

// M2M into the active non-leaf cells of level L (fmm2D.cpp:309-379). A warp
// holds G = 32/(P+1) cells, lane (g, p) computing a_p of cell g by Horner's
// rule in t = z_child - z_parent for all children at once (independent
// chains), then summing the children in order:
//   a_p += a0 t^p + sum_{k=1..p} m2m[p][k] a_k t^(p-k).
// Child expansions are read through L2 (ld.cg): in the cooperative kernel the
// level below was written by other blocks of the same launch.
__device__ __forceinline__ void m2m_level_body(const Tree2D& t, double2* __restrict__ a,
                                               const double* __restrict__ coef, int P, int L) {
    __shared__ double2 s_child[kLevelWarps][4][32];  // [warp][child][g * (P+1) + k]
    __shared__ double2 s_tt[kLevelWarps][4][16];     // [warp][child][g]
    const double* g_m2m = coef + kCoefM2M;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int Q = P + 1, G = 32 / Q, g = lane / Q, k = lane - g * Q;
    const int c0 = t.info->level_start[L], c1 = t.info->level_start[L + 1];
    const int warps = gridDim.x * (blockDim.x >> 5);
    const int gw = blockIdx.x * (blockDim.x >> 5) + wib;
    for (int cb = c0 + gw * G; cb < c1; cb += warps * G) {
        const int c = cb + g;
        bool ok = g < G && c < c1;
        if (ok) {
            const uint8_t f = t.c_flags[c];
            ok = !(f & CELL_LEAF) && (f & CELL_ACTIVE);
        }
        unsigned m = 0;
        int ch0 = -1;
        if (ok) {
            m = t.c_chmask[c];
            ch0 = t.c_child0[c];
            ok = ch0 >= 0;
        }
        const int nch = ok ? __popc(m) : 0;
        #pragma unroll
        for (int r = 0; r < 4; ++r)
            if (r < nch) s_child[wib][r][lane] = __ldcg(&a[(size_t)(ch0 + r) * Q + k]);
        if (k < nch) s_tt[wib][k][g] = make_double2(t.c_cx[ch0 + k] - t.c_cx[c], t.c_cy[ch0 + k] - t.c_cy[c]);
        __syncwarp();
        if (ok) {
            double2 acc = make_double2(0.0, 0.0);
            if (k == 0) {
                for (int r = 0; r < nch; ++r) acc = cadd(acc, s_child[wib][r][g * Q]);
            } else {
                double2 S[4], tt[4];
                #pragma unroll
                for (int r = 0; r < 4; ++r) {
                    S[r] = s_child[wib][r][g * Q];
                    tt[r] = s_tt[wib][r][g];
                }
                for (int j = k - 1; j >= 0; --j) {
                    const int kk = k - j;
                    const double cf = g_m2m[k * W + kk];
                    #pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (r < nch) S[r] = cfma(S[r], tt[r], cscale(s_child[wib][r][g * Q + kk], cf));
                }
                #pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (r < nch) acc = cadd(acc, S[r]);
            }
            a[(size_t)c * Q + k] = acc;
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(128)
m2m_level2d(Tree2D t, double2* __restrict__ a, const double* __restrict__ coef, int P, int L, unsigned* err) {
    if (block_fatal(err)) return;
    m2m_level_body(t, a, coef, P, L);
}

// All M2M levels (depth-1 down to 1) in one cooperative launch, a grid
// barrier between levels (barrier word: zeroed before every evaluation, used
// by this kernel only).
__global__ void __launch_bounds__(32 * kLevelWarps)
m2m_levels_coop(Tree2D t, double2* __restrict__ a, const double* __restrict__ coef, int P, unsigned* bar,
                unsigned* err) {
    const int depth = t.info->depth;
    for (int L = depth - 1; L >= 1; --L) {
        if (!block_fatal(err)) m2m_level_body(t, a, coef, P, L);
        grid_sync_counter(bar, err);
    }
}

// L2L pull into every cell of level L >= 3 from its parent (fmm2D.cpp:587-651,
// where each non-leaf parent at levels 2..max-1 pushes into its children):
//   b_p(c) += sum_{k=p..P} l2l[p][k] b_k(parent) t^(k-p),  t = z_c - z_parent.
// A warp holds G = 32/(P+1) cells, lane (g, p) computing b_p of cell g. The
// parent's expansion is final because level L-1 is complete (previous launch,
// or before the grid barrier in the cooperative kernel); it is read through
// L2 (ld.cg).
__device__ __forceinline__ void l2l_level_body(const Tree2D& t, double2* __restrict__ b,
                                               const double* __restrict__ coef, int P, int L) {
    __shared__ double2 s_par[kLevelWarps][32];
    const double* g_l2l = coef + kCoefL2L;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int Q = P + 1, G = 32 / Q, g = lane / Q, k = lane - g * Q;
    const int c0 = t.info->level_start[L], c1 = t.info->level_start[L + 1];
    const int warps = gridDim.x * (blockDim.x >> 5);
    const int gw = blockIdx.x * (blockDim.x >> 5) + wib;
    for (int cb = c0 + gw * G; cb < c1; cb += warps * G) {
        const int c = cb + g;
        const bool ok = g < G && c < c1;
        const int par = ok ? t.c_parent[c] : 0;
        if (ok) s_par[wib][lane] = __ldcg(&b[(size_t)par * Q + k]);
        __syncwarp();
        if (ok) {
            const double2 tt = make_double2(t.c_cx[c] - t.c_cx[par], t.c_cy[c] - t.c_cy[par]);
            const double* cf = g_l2l + k * W;
            const double2* sp = &s_par[wib][g * Q];
            double2 S = cscale(sp[P], cf[P]);
            for (int kk = P - 1; kk >= k; --kk) S = cfma(S, tt, cscale(sp[kk], cf[kk]));
            double2* bc = &b[(size_t)c * Q + k];
            *bc = cadd(__ldcg(bc), S);
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(128)
l2l_level2d(Tree2D t, double2* __restrict__ b, const double* __restrict__ coef, int P, int L, unsigned* err) {
    if (block_fatal(err)) return;
    l2l_level_body(t, b, coef, P, L);
}

// All L2L levels (3 down to the depth) in one cooperative launch.
__global__ void __launch_bounds__(32 * kLevelWarps)
l2l_levels_coop(Tree2D t, double2* __restrict__ b, const double* __restrict__ coef, int P, unsigned* bar,
                unsigned* err) {
    const int depth = t.info->depth;
    for (int L = 3; L <= depth; ++L) {
        if (!block_fatal(err)) l2l_level_body(t, b, coef, P, L);
        grid_sync_counter(bar, err);
    }
}

// ---- M2L -------------------------------------------------------------------

// One warp per target cell. The warp is split into G = 32/P groups of P lanes;
// lane (g, p-1) accumulates b_p over the sources g, g+G, ... of list 2 then
// list 4. Powers w^m = (z_src - z_tgt)^(-m), m = 1..2P, go through shared
// memory per group.
__global__ void __launch_bounds__(128)
m2l2d(Tree2D t, Lists2D l, const double2* __restrict__ a, double2* __restrict__ b, const double* __restrict__ coef,
      int P, unsigned* err) {
    const double* g_m2l = coef + kCoefM2L;
    extern __shared__ double2 sm[];
    if (fatal(err)) return;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int G = 32 / P;
    const int g = lane / P, p = lane % P + 1;
    const bool on = g < G;
    // per warp: pw[G][2P+1], as[G][P+1], part[G][P+1]
    double2* pw = sm + (size_t)wib * (G * (2 * P + 1) + 2 * G * (P + 1));
    double2* as = pw + G * (2 * P + 1);
    double2* part = as + G * (P + 1);
    const int c_begin = t.info->level_start[2], c_end = t.info->n_cells;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int c = c_begin + blockIdx.x * (blockDim.x >> 5) + wib; c < c_end; c += warps) {
        const int n2 = l.l2_n[c], n4 = l.l4_n[c];
        const int ns = n2 + n4;
        const double zx = t.c_cx[c], zy = t.c_cy[c];
        double2 acc = make_double2(0.0, 0.0);
        for (int s0 = 0; s0 < ns; s0 += G) {
            const int si = s0 + g;
            const bool has = on && si < ns;
            int src = -1;
            if (has) src = si < n2 ? l.l2_src[(size_t)c * kList2Cap + si] : l.l4_src[(size_t)c * kList4Cap + (si - n2)];
            double2 w = make_double2(0.0, 0.0);
            if (has) w = cinv(make_double2(t.c_cx[src] - zx, t.c_cy[src] - zy));
            // w^p by binary powering, then w^(p+P) = w^p * w^P.
            double2 wp = make_double2(1.0, 0.0), base = w;
            for (int e = p; e > 0; e >>= 1) {
                if (e & 1) wp = cmul(wp, base);
                base = cmul(base, base);
            }
            const double2 wP = make_double2(__shfl_sync(0xffffffffu, wp.x, on ? g * P + P - 1 : lane),
                                            __shfl_sync(0xffffffffu, wp.y, on ? g * P + P - 1 : lane));
            if (has) {
                pw[g * (2 * P + 1) + p] = wp;
                pw[g * (2 * P + 1) + p + P] = cmul(wp, wP);
                as[g * (P + 1) + p] = a[(size_t)src * (P + 1) + p];
                if (p == 1) as[g * (P + 1)] = a[(size_t)src * (P + 1)];
            }
            __syncwarp();
            if (has) {
                const double2* A = as + g * (P + 1);
                const double2* Wg = pw + g * (2 * P + 1);
                double2 s = cscale(cmul(A[0], Wg[p]), 1.0 / (double)p);
                const double* cf = g_m2l + p * W;
                for (int k = 1; k <= P; ++k) s = cfma(cscale(A[k], cf[k]), Wg[p + k], s);
                acc = csub(acc, s);
            }
            __syncwarp();
        }
        if (on) part[g * (P + 1) + p] = acc;
        __syncwarp();
        if (lane < P) {
            double2 tot = make_double2(0.0, 0.0);
            for (int gg = 0; gg < G; ++gg) tot = cadd(tot, part[gg * (P + 1) + lane + 1]);
            b[(size_t)c * (P + 1) + lane + 1] = tot;
        }
        if (lane == 0) b[(size_t)c * (P + 1)] = make_double2(0.0, 0.0);
        __syncwarp();
    }
}

// M2L with precomputed list-2 operators. For a list-2 pair the source sits
// at the integer offset tau = (dx, dy) in {-3..3}^2 cell lengths r, and with
// scaled expansions a~_k = a_k / r^k, b~_p = r^p b_p the translation
//   b~_p = sum_{k=0..P} T_tau[p][k] a~_k,
//   T_tau[p][0] = -(1/p) tau^-p,  T_tau[p][k] = -m2l[p][k] tau^-(p+k)
// does not depend on the level (the same algebra as fmm2D.cpp:471-481). The
// 49 operators (stored [slot][k][p], p fastest) replace the per-pair powers.
// List-4 sources (coarser leaves, arbitrary offsets) use the direct formula.
// One warp per target cell, split into G = 32/P groups of P lanes.
__global__ void __launch_bounds__(128)
m2l2d_op(Tree2D t, Lists2D l, const double2* __restrict__ a, double2* __restrict__ b,
         const double2* __restrict__ op, const double* __restrict__ coef, int P, unsigned* err) {
    extern __shared__ double2 sm[];
    if (fatal(err)) return;
    const double* g_m2l = coef + kCoefM2L;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int G = 32 / P;
    const int g = lane / P, p = lane % P + 1;
    const bool on = g < G;
    // per warp: as[G][P+1] (scaled sources), pw[G][2P+1] (list-4 powers), part[G][P+1]
    double2* as = sm + (size_t)wib * (G * (P + 1) * 2 + G * (2 * P + 1));
    double2* part = as + G * (P + 1);
    double2* pw = part + G * (P + 1);
    const double root = t.geom->root;
    const int c_begin = t.info->level_start[2], c_end = t.info->n_cells;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int c = c_begin + blockIdx.x * (blockDim.x >> 5) + wib; c < c_end; c += warps) {
        const int n2 = l.l2_n[c], n4 = l.l4_n[c];
        const double rinv = ldexp(1.0, (int)t.c_level[c]) / root;  // 1 / cell length
        const double zx = t.c_cx[c], zy = t.c_cy[c];
        double2 acc_s = make_double2(0.0, 0.0);  // scaled (list 2)
        double2 acc = make_double2(0.0, 0.0);    // unscaled (list 4)
        // rinv^k for the lanes' k = p (and k = 0 handled by p == 1 lanes)
        double rk = 1.0;
        for (int e = 0; e < p; ++e) rk *= rinv;  // rinv^p
        for (int s0 = 0; s0 < n2; s0 += G) {
            const int si = s0 + g;
            const bool has = on && si < n2;
            int src = 0, slot = 0;
            if (has) {
                src = l.l2_src[(size_t)c * kList2Cap + si];
                slot = l.l2_slot[(size_t)c * kList2Cap + si];
                as[g * (P + 1) + p] = cscale(a[(size_t)src * (P + 1) + p], rk);
                if (p == 1) as[g * (P + 1)] = a[(size_t)src * (P + 1)];
            }
            __syncwarp();
            if (has) {
                const double2* A = as + g * (P + 1);
                const double2* T = op + (size_t)slot * (P + 1) * P + (p - 1);
                double2 sacc = acc_s;
                for (int k = 0; k <= P; ++k) sacc = cfma(T[(size_t)k * P], A[k], sacc);
                acc_s = sacc;
            }
            __syncwarp();
        }
        for (int s0 = 0; s0 < n4; s0 += G) {
            const int si = s0 + g;
            const bool has = on && si < n4;
            int src = 0;
            if (has) src = l.l4_src[(size_t)c * kList4Cap + si];
            double2 w = make_double2(0.0, 0.0);
            if (has) w = cinv(make_double2(t.c_cx[src] - zx, t.c_cy[src] - zy));
            double2 wp = make_double2(1.0, 0.0), base = w;
            for (int e = p; e > 0; e >>= 1) {
                if (e & 1) wp = cmul(wp, base);
                base = cmul(base, base);
            }
            const double2 wP = make_double2(__shfl_sync(0xffffffffu, wp.x, on ? g * P + P - 1 : lane),
                                            __shfl_sync(0xffffffffu, wp.y, on ? g * P + P - 1 : lane));
            double2* Wg = pw + g * (2 * P + 1);
            if (has) {
                Wg[p] = wp;
                Wg[p + P] = cmul(wp, wP);
                as[g * (P + 1) + p] = a[(size_t)src * (P + 1) + p];
                if (p == 1) as[g * (P + 1)] = a[(size_t)src * (P + 1)];
            }
            __syncwarp();
            if (has) {
                const double2* A = as + g * (P + 1);
                double2 sv = cscale(cmul(A[0], Wg[p]), 1.0 / (double)p);
                const double* cf = g_m2l + p * W;
                for (int k = 1; k <= P; ++k) sv = cfma(cscale(A[k], cf[k]), Wg[p + k], sv);
                acc = csub(acc, sv);
            }
            __syncwarp();
        }
        if (on) part[g * (P + 1) + p] = cadd(cscale(acc_s, rk), acc);
        __syncwarp();
        if (lane < P) {
            double2 tot = make_double2(0.0, 0.0);
            for (int gg = 0; gg < G; ++gg) tot = cadd(tot, part[gg * (P + 1) + lane + 1]);
            b[(size_t)c * (P + 1) + lane + 1] = tot;
        }
        if (lane == 0) b[(size_t)c * (P + 1)] = make_double2(0.0, 0.0);
        __syncwarp();
    }
}

// ---- leaf evaluation: M2P (list 3), L2P --------------------------------------

// Far field of targets i of a leaf, lane-owned: M2P over list 3
// (fmm2D.cpp:1040-1066) and L2P of the leaf's complete local expansion
// (fmm2D.cpp:1076-1093). With TWO, each lane takes a second target and both
// run through the list-3 sources together (one load of every source's
// coefficients serves both, and the two chains are independent). Each
// target's sums run in the same order either way. MODE kEvalFull does both;
// kEvalM2P writes the list-3 sums alone to fx/fy; kEvalL2P starts from those
// sums (the same value the full mode reaches after its list-3 loop) and adds
// L2P, so the split gives the same bits as one pass.
constexpr int kEvalFull = 0, kEvalM2P = 1, kEvalL2P = 2;
template <bool TWO, int MODE>
__device__ __forceinline__ void eval_targets(const Tree2D& t, const Lists2D& l, const double2* __restrict__ a,
                                             const double2* s_b, int P, int i0, int i1, bool h0, bool h1, double zx,
                                             double zy, const int32_t* src3, uint32_t n3, double* fx, double* fy,
                                             const double* nx, const double* ny, double* out0, double* out1,
                                             int velocity, double u_inf, double v_inf, unsigned* err) {
    double x[2], y[2], ex[2] = {0.0, 0.0}, ey[2] = {0.0, 0.0};
    bool h[2] = {h0, h1};
    const int ii[2] = {i0, i1};
    #pragma unroll
    for (int u = 0; u < (TWO ? 2 : 1); ++u) {
        x[u] = h[u] ? t.px[ii[u]] : zx + 1.0;
        y[u] = h[u] ? t.py[ii[u]] : zy;
    }
    if (MODE == kEvalL2P) {
        #pragma unroll
        for (int u = 0; u < (TWO ? 2 : 1); ++u)
            if (h[u]) {
                ex[u] = fx[ii[u]];
                ey[u] = fy[ii[u]];
            }
        n3 = 0;
    }
    for (uint32_t k = 0; k < n3; ++k) {
        const int s = src3[k];
        const double sx = t.c_cx[s], sy = t.c_cy[s];
        const double2* A = a + (size_t)s * (P + 1);
        double2 w[2], S[2];
        #pragma unroll
        for (int u = 0; u < (TWO ? 2 : 1); ++u) {
            w[u] = cinv(make_double2(x[u] - sx, y[u] - sy));
            S[u] = A[P];
        }
        for (int pp = P - 1; pp >= 0; --pp) {
            const double2 Ap = A[pp];
            #pragma unroll
            for (int u = 0; u < (TWO ? 2 : 1); ++u) S[u] = cfma(S[u], w[u], Ap);
        }
        #pragma unroll
        for (int u = 0; u < (TWO ? 2 : 1); ++u) {
            S[u] = cmul(S[u], w[u]);
            ex[u] += S[u].x;
            ey[u] -= S[u].y;
        }
    }
    if (MODE == kEvalM2P) {
        #pragma unroll
        for (int u = 0; u < (TWO ? 2 : 1); ++u)
            if (h[u]) {
                fx[ii[u]] = ex[u];
                fy[ii[u]] = ey[u];
            }
        return;
    }
    #pragma unroll
    for (int u = 0; u < (TWO ? 2 : 1); ++u) {
        const double2 w = make_double2(x[u] - zx, y[u] - zy);
        double2 S = cscale(s_b[P], (double)P);
        for (int pp = P - 1; pp >= 1; --pp) S = cfma(S, w, cscale(s_b[pp], (double)pp));
        double fxv = ex[u] + S.x, fyv = ey[u] - S.y;
        if (!h[u]) continue;
        const int i = ii[u];
        if (nx) {
            // near field already computed: write the total in the caller's order
            fxv = nx[i] + fxv;
            fyv = ny[i] + fyv;
            const uint32_t orig = t.perm[i];
            if (orig >= (uint32_t)t.n) {
                set_err(err, ERR_INDEX);
            } else if (velocity) {
                out0[orig] = fyv + u_inf;
                out1[orig] = -fxv + v_inf;
            } else {
                out0[orig] = fxv;
                out1[orig] = fyv;
            }
        } else {
            fx[i] = fxv;
            fy[i] = fyv;
        }
    }
}

constexpr int kEvalWarps = 4;   // one warp per leaf
constexpr int kEvalThreads = 32 * kEvalWarps;

// Far field of every particle of a leaf (eval_targets), one warp per leaf,
// 64 targets per pass (two per lane). Cells above level 2 carry no local
// expansion (M2L starts at level 2).
template <int MODE>
__global__ void __launch_bounds__(kEvalThreads)
eval2d(Tree2D t, Lists2D l, const double2* __restrict__ a, const double2* __restrict__ b, double* __restrict__ fx,
       double* __restrict__ fy, int P, const double* __restrict__ nx, const double* __restrict__ ny,
       double* __restrict__ out0, double* __restrict__ out1, int velocity, double u_inf, double v_inf, int lists,
       unsigned* err) {
    __shared__ double2 s_bw[kEvalWarps][W];
    if (fatal(err)) return;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    double2* s_b = s_bw[wib];
    const int nl = t.info->n_leaves;
    for (int li = blockIdx.x * kEvalWarps + wib; li < nl; li += gridDim.x * kEvalWarps) {
        const int c = t.leaf_cells[li];
        const int L = t.c_level[c];
        if (MODE != kEvalM2P)
            for (int k = lane; k <= P; k += 32)
                s_b[k] = L >= 2 ? b[(size_t)c * (P + 1) + k] : make_double2(0.0, 0.0);
        __syncwarp();
        const int lo = t.c_lo[c], hi = t.c_hi[c];
        const double zx = t.c_cx[c], zy = t.c_cy[c];
        // list 3 of the leaf: the CSR, or (M2P) the fixed slots of
        // int_list_slots, the leaves whose list outgrew them coming in a
        // second pass from the CSR
        const int32_t* src3 = nullptr;
        uint32_t n3 = 0;
        if (MODE != kEvalL2P) {
            bool csr = lists == kP2PListCsr;
            if (!csr) {
                const uint32_t cnt = l.l3_cnt[li];
                const bool spill = cnt > (uint32_t)kListSlot3;
                if (spill != (lists == kP2PListSpill)) continue;   // the other pass takes this leaf
                csr = spill;
                if (!spill) {
                    src3 = l.l3_slot + (size_t)li * kListSlot3;
                    n3 = cnt;
                }
            }
            if (csr) {
                const uint32_t o3 = l.l3_off[li];
                src3 = l.l3_src + o3;
                n3 = l.l3_off[li + 1] - o3;
            }
        }
        for (int i0 = lo; i0 < hi; i0 += 64) {
            const int ia = i0 + lane, ib = i0 + 32 + lane;
            if (i0 + 32 < hi)   // warp-uniform
                eval_targets<true, MODE>(t, l, a, s_b, P, ia, ib, ia < hi, ib < hi, zx, zy, src3, n3, fx, fy, nx, ny,
                                         out0, out1, velocity, u_inf, v_inf, err);
            else
                eval_targets<false, MODE>(t, l, a, s_b, P, ia, ib, ia < hi, false, zx, zy, src3, n3, fx, fy, nx, ny,
                                          out0, out1, velocity, u_inf, v_inf, err);
        }
        __syncwarp();
    }
}

// ---- P2P over list 1 --------------------------------------------------------

// Writes one target's total field (near + far) in the caller's order; with
// fx == nullptr (near field computed concurrently with the far field) the
// near field alone, in tree order, into out0/out1.
__device__ __forceinline__ void p2p_store(const Tree2D& t, int ti, double ex, double ey, const double* fx,
                                          const double* fy, double* out0, double* out1, int velocity, double u_inf,
                                          double v_inf, unsigned* err) {
    if (!fx) {
        out0[ti] = ex;
        out1[ti] = ey;
        return;
    }
    ex += fx[ti];
    ey += fy[ti];
    const uint32_t orig = t.perm[ti];
    if (orig >= (uint32_t)t.n) {
        set_err(err, ERR_INDEX);
    } else if (velocity) {
        out0[orig] = ey + u_inf;
        out1[orig] = -ex + v_inf;
    } else {
        out0[orig] = ex;
        out1[orig] = ey;
    }
}

// ---- mixed form: FP32 near field ---------------------------------------------

// FP32 reciprocal (hardware approximation, ~1 ulp) of the mixed near field.
__device__ __forceinline__ float rcp_approx(float a) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}


constexpr int kP2PMeta = 64;   // list-1 cells staged per leaf at a time

// ---- FP64 near field ---------------------------------------------------------

// The plain form's field and the potential over list 1 (fmm2D.cpp:135-179 and
// 77-122), one warp per leaf. A chunk of T <= 192 of the leaf's targets is
// spread over H lanes with M = ceil(T / H) targets each, and the ns = 32 / H
// lane groups take every ns-th source of the leaf's list-1 cells, which form
// one flat sequence staged 64 at a time in shared memory (loaded a step
// ahead). M is picked per chunk for the fewest lane-cycles (near_shape): lanes
// without a target and slots without one are what the FP64 pipe loses, and a
// staged source costs the SM 24 bytes a lane of its 128 a cycle, so few
// targets per lane would be bound by shared memory. The pair itself is ten
// FP64 operations. j == i is tested only in the steps that hold the leaf's own
// cell (the reference's NaN of two coincident particles stays). Partial sums
// are added over the lane groups in a fixed order.
// 242 M pairs (778,377-particle boundary layer, caps 50/75): 249 us, 62 % of
// the FP64 pipe's cycles (this mix of operations alone, in registers, reaches
// 72 %: three 64-bit operands an FMA); the
// kernel before took four targets per lane, cell by cell from global memory,
// 379 us and a 13 us copy of the particles.
constexpr int kNear64Warps = 4;
constexpr int kNear64Stage = 64;
constexpr int kNear64MaxM = 6;
constexpr int kNear64Chunk = 32 * kNear64MaxM;

struct Near64Warp {
    union {
        struct {
            double2 xy[kNear64Stage];
            double q[kNear64Stage];
        } st;
        double red[2 * kNear64MaxM][32];
    };
    int2 meta[kP2PMeta];       // first particle and size of each list-1 cell
};

// Targets per lane of a chunk of T: the least (10 M + 3) / ns, ten operations
// per pair and about three for a step.
__device__ __forceinline__ int near_shape(int T) {
    int best = kNear64MaxM, bc = 10 * kNear64MaxM + 3, bn = 32 / ((T + kNear64MaxM - 1) / kNear64MaxM);
    #pragma unroll
    for (int M = kNear64MaxM - 1; M >= 1; --M) {
        const int H = (T + M - 1) / M;
        if (H > 32) break;
        const int ns = 32 / H, c = 10 * M + 3;
        if (c * bn < bc * ns) {
            best = M;
            bc = c;
            bn = ns;
        }
    }
    return best;
}

// log a in FP64 without branches, so that the lane's targets run side by side
// (CUDA's own log branches for its special cases: 94 us against 55 for the
// near field of 120,011 particles): a = m 2^e with m in [sqrt(1/2), sqrt(2)),
// log m = 2 atanh z, z = (m - 1) / (m + 1), by the series of atanh to z^21
// (|z| <= 0.172: the next term is below 2^-60 of the sum; relative error at
// most 3.3e-16 over 1e6 arguments). For normal a away from the ends of the
// range (log_ordinary); the others take log().
__device__ __forceinline__ bool log_ordinary(double a) {
    return (unsigned)__double2hiint(a) - 0x01000000u < 0x7e000000u;   // 2^-1007 <= a < 2^1009, no NaN
}
__device__ __forceinline__ double log_series(double a) {
    const int hi = __double2hiint(a);
    // high word of sqrt(1/2): m >= sqrt(1/2) up to 2^-20, and e = 0 next to 1
    const int e = (hi - 0x3fe6a09e) >> 20;
    const double m = __hiloint2double(hi - (e << 20), __double2loint(a));
    const double num = m - 1.0;
    const double z = num * rcp_nr(m + 1.0);
    const double z2 = z * z;
    double p = fma(z2, 2.0 / 21.0, 2.0 / 19.0);
    p = fma(p, z2, 2.0 / 17.0);
    p = fma(p, z2, 2.0 / 15.0);
    p = fma(p, z2, 2.0 / 13.0);
    p = fma(p, z2, 2.0 / 11.0);
    p = fma(p, z2, 2.0 / 9.0);
    p = fma(p, z2, 2.0 / 7.0);
    p = fma(p, z2, 2.0 / 5.0);
    p = fma(p, z2, 2.0 / 3.0);
    p = fma(p * z2, z, 2.0 * z);
    return fma((double)e, 0.69314718055994530942, p);
}

// Staged sources s0, s0 + ns, ... below cnt onto the lane's M targets; SELF:
// flat source self[k] is target k itself and adds zero whatever its strength.
// POT: sums q log(r^2) in ex.
template <int M, bool POT, bool SELF>
__device__ __forceinline__ void near64_pairs(const double2* xy, const double* q, int s0, int cnt, int ns,
                                             const double* x, const double* y, const int* self, double* ex,
                                             double* ey) {
    if (s0 >= cnt) return;
    double2 pn = xy[s0];   // the next source, loaded while this one is applied
    double wn = q[s0];
    #pragma unroll 1
    for (int s = s0; s < cnt; s += ns) {
        const double2 p = pn;
        const double w = wn;
        const int sn = min(s + ns, kNear64Stage - 1);
        pn = xy[sn];
        wn = q[sn];
        double r2[M], lg[M];
        bool odd = false;
        #pragma unroll
        for (int k = 0; k < M; ++k) {
            const double dx = x[k] - p.x, dy = y[k] - p.y;
            r2[k] = fma(dx, dx, dy * dy);
            if (POT) {
                lg[k] = log_series(r2[k]);
                odd |= !log_ordinary(r2[k]);
            } else {
                double f = w * rcp_nr(r2[k]);
                if (SELF && s == self[k]) f = 0.0;
                ex[k] = fma(f, dx, ex[k]);
                ey[k] = fma(f, dy, ey[k]);
            }
        }
        if (POT) {
            if (odd) {   // a target itself, coincident particles, or distances beyond 1e+-150
                #pragma unroll
                for (int k = 0; k < M; ++k)
                    if (!log_ordinary(r2[k])) lg[k] = SELF && s == self[k] ? 0.0 : log(r2[k]);
            }
            #pragma unroll
            for (int k = 0; k < M; ++k) ex[k] = fma(SELF && s == self[k] ? 0.0 : w, lg[k], ex[k]);
        }
    }
}

template <int M, bool POT>
__device__ __forceinline__ void near64_chunk(Near64Warp& sm, const Tree2D& t, const int32_t* __restrict__ src1, int c,
                                             int lo, int n1, int tb, int T, const double* fx, const double* fy,
                                             double* out0, double* out1, int velocity, double u_inf, double v_inf,
                                             unsigned* err) {
    const int lane = threadIdx.x & 31;
    const int H = (T + M - 1) / M, ns = 32 / H;
    const int tt = lane % H, split = lane / H;   // target k of this lane is chunk slot tt + k H
    double x[M], y[M], ex[M], ey[M];
    #pragma unroll
    for (int k = 0; k < M; ++k) {
        const int i = tt + k * H;
        x[k] = t.px[tb + (i < T ? i : 0)];
        y[k] = t.py[tb + (i < T ? i : 0)];
        ex[k] = ey[k] = 0.0;
    }
    for (int seg = 0; seg < n1; seg += kP2PMeta) {
        const int nseg = min(kP2PMeta, n1 - seg);
        __syncwarp();
        // ranges and flat starts of the segment's cells (two per lane), and
        // the leaf's own flat range
        int sz[2] = {0, 0}, inc[2];
        bool own[2] = {false, false};
        #pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = lane + 32 * h;
            if (k < nseg) {
                const int sc = src1[seg + k];
                const int slo = t.c_lo[sc];
                sz[h] = t.c_hi[sc] - slo;
                own[h] = sc == c;
                sm.meta[k] = make_int2(slo, sz[h]);
            }
            inc[h] = sz[h];
        }
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a0 = __shfl_up_sync(0xffffffffu, inc[0], o), a1 = __shfl_up_sync(0xffffffffu, inc[1], o);
            if (lane >= o) {
                inc[0] += a0;
                inc[1] += a1;
            }
        }
        const int tot0 = __shfl_sync(0xffffffffu, inc[0], 31);
        const int total = tot0 + __shfl_sync(0xffffffffu, inc[1], 31);
        const int start0 = inc[0] - sz[0], start1 = tot0 + inc[1] - sz[1];
        const unsigned b0 = __ballot_sync(0xffffffffu, own[0]), b1 = __ballot_sync(0xffffffffu, own[1]);
        int own0 = -(1 << 30);
        if (b0) own0 = __shfl_sync(0xffffffffu, start0, __ffs(b0) - 1);
        else if (b1) own0 = __shfl_sync(0xffffffffu, start1, __ffs(b1) - 1);
        const int self0 = own0 + (tb - lo) + tt;   // flat source that is target 0 of this lane
        __syncwarp();
        // per-lane walkers over the flat sequence: the lane stages flat sources
        // cb + lane and cb + 32 + lane of step cb
        int kw[2] = {0, 0}, ow[2] = {lane, lane + 32};
        auto settle = [&](int h) {
            while (kw[h] < nseg && ow[h] >= sm.meta[kw[h]].y) {
                ow[h] -= sm.meta[kw[h]].y;
                ++kw[h];
            }
        };
        double vx[2], vy[2], vq[2];
        auto fetch = [&](int h) {
            vx[h] = vy[h] = vq[h] = 0.0;
            if (kw[h] < nseg) {
                const int j = sm.meta[kw[h]].x + ow[h];
                vx[h] = t.px[j];
                vy[h] = t.py[j];
                vq[h] = t.pq[j];
            }
        };
        #pragma unroll
        for (int h = 0; h < 2; ++h) {
            settle(h);
            fetch(h);
        }
        for (int cb = 0; cb < total; cb += kNear64Stage) {
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                sm.st.xy[lane + 32 * h] = make_double2(vx[h], vy[h]);
                sm.st.q[lane + 32 * h] = vq[h];
            }
            __syncwarp();
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                ow[h] += kNear64Stage;
                settle(h);
                fetch(h);
            }
            const int cnt = min(kNear64Stage, total - cb);
            const int s0 = split < ns ? split : cnt;
            if (own0 < cb + kNear64Stage && own0 + (tb - lo) + T > cb) {   // warp-uniform
                int self[M];
                #pragma unroll
                for (int k = 0; k < M; ++k) self[k] = tt + k * H < T ? self0 + k * H - cb : -1;
                near64_pairs<M, POT, true>(sm.st.xy, sm.st.q, s0, cnt, ns, x, y, self, ex, ey);
            } else {
                near64_pairs<M, POT, false>(sm.st.xy, sm.st.q, s0, cnt, ns, x, y, nullptr, ex, ey);
            }
            __syncwarp();
        }
    }
    // sum over the lane groups: lane tt + g H holds group g's parts of target slots tt + k H
    __syncwarp();
    #pragma unroll
    for (int k = 0; k < M; ++k) {
        sm.red[2 * k][lane] = ex[k];
        if (!POT) sm.red[2 * k + 1][lane] = ey[k];
    }
    __syncwarp();
    for (int i = lane; i < T; i += 32) {
        const int k = i / H, l0 = i - k * H;
        double sx = 0.0, sy = 0.0;
        for (int g = 0; g < ns; ++g) {
            sx += sm.red[2 * k][l0 + g * H];
            if (!POT) sy += sm.red[2 * k + 1][l0 + g * H];
        }
        if (POT) {
            const uint32_t orig = t.perm[tb + i];
            if (orig >= (uint32_t)t.n) set_err(err, ERR_INDEX);
            else out0[orig] = 0.5 * sx + fx[tb + i];
        } else {
            p2p_store(t, tb + i, sx, sy, fx, fy, out0, out1, velocity, u_inf, v_inf, err);
        }
    }
    __syncwarp();
}

// List 1 from the CSR, or from the fixed slots (kP2PListSlots; the leaves
// whose list outgrew them come in a second pass, kP2PListSpill, from the CSR).
template <bool POT>
__global__ void __launch_bounds__(32 * kNear64Warps, 3)
near2d_f64(Tree2D t, Lists2D l, const double* __restrict__ fx, const double* __restrict__ fy,
           double* __restrict__ out0, double* __restrict__ out1, int velocity, double u_inf, double v_inf, int lists,
           unsigned* err) {
    __shared__ Near64Warp sm[kNear64Warps];
    if (fatal(err)) return;
    const int wib = threadIdx.x >> 5;
    const int nl = t.info->n_leaves;
    // A tree of few leaves leaves most of the GPU's 148 x 12 warps without one:
    // 2, 4 or 8 warps then share a leaf's targets (2,001 particles, 64 leaves:
    // 24 -> 12 us), up to half the GPU's places. Each part stages the leaf's
    // sources again, which costs other solves the GPU when they share it: with
    // all places taken, 256 leaves in four parts in place of two, a captured batch
    // of 24 solves of 6,000 particles took 782 us (735 with this line, 711 with a
    // quarter of the places, 706 without parts), one of 48 1,408 (1,316, 1,263,
    // 1,250); alone, 12,000 particles of as many leaves 169, 170, 174 and 174 us
    // eager. 20,001 particles, about 1,024 leaves: 133 us in one part, 144 in two.
    int parts = 1;
    while (parts < 8 && (long long)nl * parts * 2 <= 148 * 6) parts *= 2;
    for (int it = blockIdx.x * kNear64Warps + wib; it < nl * parts; it += gridDim.x * kNear64Warps) {
        const int li = it / parts, part = it - li * parts;
        const int32_t* src1;
        int n1;
        if (lists == kP2PListCsr) {
            src1 = l.l1_src + l.l1_off[li];
            n1 = (int)(l.l1_off[li + 1] - l.l1_off[li]);
        } else {
            const uint32_t cnt = l.l1_cnt[li];
            const bool spill = cnt > (uint32_t)kListSlot1;
            if (spill != (lists == kP2PListSpill)) continue;
            src1 = spill ? l.l1_src + l.l1_off[li] : l.l1_slot + (size_t)li * kListSlot1;
            n1 = spill ? (int)(l.l1_off[li + 1] - l.l1_off[li]) : (int)cnt;
        }
        const int c = t.leaf_cells[li];
        const int lo = t.c_lo[c], leaf_hi = t.c_hi[c];
        const int slice = (leaf_hi - lo + parts - 1) / parts;
        const int hi = min(leaf_hi, lo + (part + 1) * slice);
        for (int tb = lo + part * slice; tb < hi; tb += kNear64Chunk) {
            const int T = min(kNear64Chunk, hi - tb);
            switch (near_shape(T)) {
#define VPM_NEAR_CASE(MM)                                                                                            \
    case MM:                                                                                                         \
        near64_chunk<MM, POT>(sm[wib], t, src1, c, lo, n1, tb, T, fx, fy, out0, out1, velocity, u_inf, v_inf, err);   \
        break;
                VPM_NEAR_CASE(1) VPM_NEAR_CASE(2) VPM_NEAR_CASE(3) VPM_NEAR_CASE(4) VPM_NEAR_CASE(5) VPM_NEAR_CASE(6)
#undef VPM_NEAR_CASE
                default: break;
            }
        }
    }
}

// Warp-per-leaf FP32 near field (the mixed form's default). A chunk of
// T <= 192 targets of the warp's leaf is spread over H lanes (the smallest
// power of two with M = ceil(T/H) <= 12 targets per lane), so all 32 lanes
// are busy and at most H - 1 target slots idle. The leaf's list-1 cells form
// one flat sequence of sources; every step the warp stages the next
// kTileStage of them in shared memory (loads issued a step ahead, moved into
// the target leaf's frame: scaled by the exact power of two between the two
// leaves' sizes plus the FP32 cell offset; stored with x, y and q duplicated
// so that they feed packed FP32x2 instructions directly), and
// lane group ("split") s of the ns = 32/H groups applies staged sources
// s, s + ns, ... to its M targets. Every kTileFlush sources the per-lane FP32
// sums are reduced over the splits with shuffles into FP64 accumulators in
// shared memory (target k is kept by split k mod ns); the sums are in units
// of the leaf size and are scaled back on the store.
//
// i == j needs no test: r^2 is formed as dx dx + dy dy + kTileEps, and a
// particle of the leaf meets itself at dx = dy = 0 exactly (the own cell's
// offset is zero, its scale one), so q / kTileEps multiplies zero offsets.
// In leaf units, the smallest non-zero FP32 offset squared is about 1e-15,
// so kTileEps changes no other pair, and q / kTileEps stays finite for
// |q| < 3e14.
constexpr int kTileWarps = 8;
constexpr int kTileFlush = 128;
constexpr int kTileMaxM = 6;
constexpr int kTileChunk = 16 * kTileMaxM;      // targets per chunk (H <= 16, so ns >= 2)
constexpr int kTileSlots = kTileMaxM / 2;       // FP64 target slots per lane (ns >= 2)
constexpr int kTileStage = 64;                  // sources staged per step (two per lane)
constexpr float kTileEps = 1e-24f;

struct TileShared {
    float4 xy[kTileWarps][kTileStage];             // (x, x, y, y) of the staged sources
    float2 qq[kTileWarps][kTileStage];             // (q, q)
    int2 meta[kTileWarps][kP2PMeta];               // (lo, size) per list-1 cell
    int cs[kTileWarps][kP2PMeta + 1];              // flat start of each cell, then the total
    double acc[kTileWarps][2 * kTileSlots][32];    // FP64 accumulators: row 2i x, 2i+1 y of slot i
};

// Two targets (packed: low half the first) against one source, on the
// packed FP32x2 instructions: d = -t + s, r2 = d.d + eps, f = q rcp(r2),
// p += f d.
__device__ __forceinline__ void tile_pair2(uint64_t nx, uint64_t ny, uint64_t sx, uint64_t sy, uint64_t sq,
                                           uint64_t eps, uint64_t& px, uint64_t& py) {
    asm("{\n\t"
        ".reg .b64 dx, dy, r2, rr, fq;\n\t"
        ".reg .f32 a, b;\n\t"
        "add.rn.f32x2 dx, %2, %4;\n\t"
        "add.rn.f32x2 dy, %3, %5;\n\t"
        "fma.rn.f32x2 r2, dx, dx, %7;\n\t"
        "fma.rn.f32x2 r2, dy, dy, r2;\n\t"
        "mov.b64 {a, b}, r2;\n\t"
        "rcp.approx.ftz.f32 a, a;\n\t"
        "rcp.approx.ftz.f32 b, b;\n\t"
        "mov.b64 rr, {a, b};\n\t"
        "mul.rn.f32x2 fq, %6, rr;\n\t"
        "fma.rn.f32x2 %0, fq, dx, %0;\n\t"
        "fma.rn.f32x2 %1, fq, dy, %1;\n\t"
        "}"
        : "+l"(px), "+l"(py)
        : "l"(nx), "l"(ny), "l"(sx), "l"(sy), "l"(sq), "l"(eps));
}

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    return ((uint64_t)__float_as_uint(hi) << 32) | (uint64_t)__float_as_uint(lo);
}
__device__ __forceinline__ float lo2(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi2(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }

// Staged sources split, split + NS, ... below cnt applied to the lane's M
// targets: a loop with constant bounds and strides (NS = 32 >> HS), so no
// index arithmetic is left between the pair updates.
template <int M, int HS>
__device__ __forceinline__ void tile_pairs(const ulonglong2* xy, const uint64_t* qq, int split, int cnt,
                                           const uint64_t* nx, const uint64_t* ny, float nxo, float nyo, uint64_t* px,
                                           uint64_t* py, float& pxo, float& pyo) {
    constexpr int MP = M / 2, NS = 32 >> HS, PER = kTileStage / NS;
    constexpr bool ODD = (M & 1) != 0;
    const uint64_t eps = pack2(kTileEps, kTileEps);
    const ulonglong2* xs = xy + split;
    const uint64_t* qs = qq + split;
    const int nrun = (cnt - split + NS - 1) / NS;   // sources of this split in the stage
    #pragma unroll
    for (int u = 0; u < PER; ++u) {
        if (u >= nrun) break;
        const ulonglong2 sv = xs[u * NS];   // (x, x), (y, y)
        const uint64_t sq = qs[u * NS];     // (q, q)
        #pragma unroll
        for (int h = 0; h < MP; ++h) tile_pair2(nx[h], ny[h], sv.x, sv.y, sq, eps, px[h], py[h]);
        if (ODD) {
            const float dx = nxo + lo2(sv.x), dy = nyo + lo2(sv.y);
            const float fq = lo2(sq) * rcp_approx(fmaf(dy, dy, fmaf(dx, dx, kTileEps)));
            pxo = fmaf(fq, dx, pxo);
            pyo = fmaf(fq, dy, pyo);
        }
    }
}

// Coordinate of a particle in the target leaf's frame, in units of its size:
// formed in FP64 and rounded once (a particle of the leaf gets the same value
// as a target and as a source).
__device__ __forceinline__ float leaf_unit(double x, double c, double ih) { return (float)((x - c) * ih); }

template <int M, int HS>
__device__ __forceinline__ void tile_chunk(TileShared& sm, const Tree2D& t, const int32_t* __restrict__ src1, int c,
                                           double ccx, double ccy, double ih, int n1, int tb, int T,
                                           const double* fx, const double* fy, double* out0, double* out1,
                                           int velocity, double u_inf, double v_inf, unsigned* err) {
    constexpr int MP = M / 2;
    constexpr int NP = MP > 0 ? MP : 1;
    constexpr int hs = HS, H = 1 << HS, ns = 32 >> HS;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int tt = lane & (H - 1), split = lane >> hs;
    // negated target coordinates (leaf frame); target k of this lane is chunk slot tt + k H
    uint64_t nx[NP], ny[NP], px[NP], py[NP];
    float nxo = 0.f, nyo = 0.f, pxo = 0.f, pyo = 0.f;
    #pragma unroll
    for (int h = 0; h < MP; ++h) {
        const int i0 = tt + ((2 * h) << hs), i1 = tt + ((2 * h + 1) << hs);
        const int j0 = tb + (i0 < T ? i0 : 0), j1 = tb + (i1 < T ? i1 : 0);
        nx[h] = pack2(-leaf_unit(t.px[j0], ccx, ih), -leaf_unit(t.px[j1], ccx, ih));
        ny[h] = pack2(-leaf_unit(t.py[j0], ccy, ih), -leaf_unit(t.py[j1], ccy, ih));
        px[h] = py[h] = 0ull;
    }
    if (M & 1) {
        const int i0 = tt + ((M - 1) << hs);
        const int j0 = tb + (i0 < T ? i0 : 0);
        nxo = -leaf_unit(t.px[j0], ccx, ih);
        nyo = -leaf_unit(t.py[j0], ccy, ih);
    }
    double* acc = &sm.acc[wib][0][lane];
    #pragma unroll
    for (int i = 0; i < 2 * kTileSlots; ++i) acc[32 * i] = 0.0;
    // reduce the FP32 partials over the splits into the FP64 slots
    auto flush = [&]() {
        #pragma unroll
        for (int k = 0; k < M; ++k) {
            float vx = (k < 2 * MP) ? ((k & 1) ? hi2(px[k >> 1]) : lo2(px[k >> 1])) : pxo;
            float vy = (k < 2 * MP) ? ((k & 1) ? hi2(py[k >> 1]) : lo2(py[k >> 1])) : pyo;
            for (int o = H; o < 32; o <<= 1) {
                vx += __shfl_xor_sync(0xffffffffu, vx, o);
                vy += __shfl_xor_sync(0xffffffffu, vy, o);
            }
            if ((k & (ns - 1)) == split) {
                const int slot = k >> (5 - hs);
                acc[32 * (2 * slot)] -= (double)vx;
                acc[32 * (2 * slot + 1)] -= (double)vy;
            }
        }
        #pragma unroll
        for (int h = 0; h < MP; ++h) px[h] = py[h] = 0ull;
        pxo = pyo = 0.f;
    };
    int steps = 0;   // staged sources since the last flush (each lane applied steps / ns of them)
    for (int seg = 0; seg < n1; seg += kP2PMeta) {
        const int nseg = min(kP2PMeta, n1 - seg);
        __syncwarp();
        // metadata and flat prefix of the segment
        {
            int sz[2] = {0, 0};
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = lane + 32 * h;
                if (k < nseg) {
                    const int sc = src1[seg + k];
                    const int slo = t.c_lo[sc];
                    sz[h] = t.c_hi[sc] - slo;
                    sm.meta[wib][k] = make_int2(slo, sz[h]);
                }
            }
            int inc0 = sz[0], inc1 = sz[1];
            #pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int a0 = __shfl_up_sync(0xffffffffu, inc0, o), a1 = __shfl_up_sync(0xffffffffu, inc1, o);
                if (lane >= o) {
                    inc0 += a0;
                    inc1 += a1;
                }
            }
            const int tot0 = __shfl_sync(0xffffffffu, inc0, 31);
            const int tot1 = __shfl_sync(0xffffffffu, inc1, 31);
            if (lane < nseg) sm.cs[wib][lane] = inc0 - sz[0];
            if (lane + 32 < nseg) sm.cs[wib][lane + 32] = tot0 + inc1 - sz[1];
            if (lane == 0) sm.cs[wib][nseg] = tot0 + tot1;
        }
        __syncwarp();
        const int total = sm.cs[wib][nseg];
        // per-lane walkers over the flat sequence: the lane stages flat sources
        // cb + lane and cb + 32 + lane of step cb
        int k0 = 0, q0 = lane, k1 = 0, q1 = lane + 32;
        while (k0 < nseg && q0 >= sm.meta[wib][k0].y) {
            q0 -= sm.meta[wib][k0].y;
            ++k0;
        }
        while (k1 < nseg && q1 >= sm.meta[wib][k1].y) {
            q1 -= sm.meta[wib][k1].y;
            ++k1;
        }
        auto fetch = [&](int k, int o) -> float4 {
            if (k >= nseg) return make_float4(0.f, 0.f, 0.f, 0.f);
            const int j = sm.meta[wib][k].x + o;
            return make_float4(leaf_unit(t.px[j], ccx, ih), leaf_unit(t.py[j], ccy, ih), (float)t.pq[j], 0.f);
        };
        auto advance = [&](int& k, int& o) {
            o += kTileStage;
            while (k < nseg && o >= sm.meta[wib][k].y) {
                o -= sm.meta[wib][k].y;
                ++k;
            }
        };
        float4 pv0 = fetch(k0, q0), pv1 = fetch(k1, q1);
        for (int cb = 0; cb < total; cb += kTileStage) {
            sm.xy[wib][lane] = make_float4(pv0.x, pv0.x, pv0.y, pv0.y);
            sm.qq[wib][lane] = make_float2(pv0.z, pv0.z);
            sm.xy[wib][lane + 32] = make_float4(pv1.x, pv1.x, pv1.y, pv1.y);
            sm.qq[wib][lane + 32] = make_float2(pv1.z, pv1.z);
            __syncwarp();
            advance(k0, q0);
            advance(k1, q1);
            pv0 = fetch(k0, q0);
            pv1 = fetch(k1, q1);
            tile_pairs<M, HS>(reinterpret_cast<const ulonglong2*>(sm.xy[wib]),
                              reinterpret_cast<const uint64_t*>(sm.qq[wib]), split, min(kTileStage, total - cb), nx,
                              ny, nxo, nyo, px, py, pxo, pyo);
            __syncwarp();
            steps += kTileStage;
            if (steps >= kTileFlush * ns) {
                flush();
                steps = 0;
            }
        }
    }
    flush();
    __syncwarp();
    #pragma unroll
    for (int i = 0; i < kTileSlots; ++i) {
        const int kk = split + (i << (5 - hs));
        const int ti = tt + (kk << hs);
        if (kk < M && ti < T)
            p2p_store(t, tb + ti, acc[32 * (2 * i)] * ih, acc[32 * (2 * i + 1)] * ih, fx, fy, out0, out1, velocity, u_inf,
                      v_inf, err);
    }
    __syncwarp();
}

__global__ void __launch_bounds__(32 * kTileWarps, 3)
p2p2d_tile_f32(Tree2D t, Lists2D l, const double* __restrict__ fx,
               const double* __restrict__ fy, double* __restrict__ out0, double* __restrict__ out1, int velocity,
               double u_inf, double v_inf, int lists, unsigned* err) {
    __shared__ TileShared sm;
    if (fatal(err)) return;
    const int wib = threadIdx.x >> 5;
    const int nl = t.info->n_leaves;
    for (int li = blockIdx.x * kTileWarps + wib; li < nl; li += gridDim.x * kTileWarps) {
        // list 1 of the leaf: CSR, or the fixed slots of int_list_slots (the
        // leaves whose list outgrew them come in a second pass, from the CSR)
        const int32_t* src1;
        int n1;
        if (lists == kP2PListCsr) {
            src1 = l.l1_src + l.l1_off[li];
            n1 = (int)(l.l1_off[li + 1] - l.l1_off[li]);
        } else {
            const uint32_t cnt = l.l1_cnt[li];
            const bool spill = cnt > (uint32_t)kListSlot1;
            if (spill != (lists == kP2PListSpill)) continue;
            src1 = spill ? l.l1_src + l.l1_off[li] : l.l1_slot + (size_t)li * kListSlot1;
            n1 = spill ? (int)(l.l1_off[li + 1] - l.l1_off[li]) : (int)cnt;
        }
        const int c = t.leaf_cells[li];
        const int lo = t.c_lo[c], hi = t.c_hi[c];
        const double ccx = t.c_cx[c], ccy = t.c_cy[c];
        const int lev = t.c_level[c];
        const double ih = ldexp(1.0, lev) / t.geom->root;   // 1 / leaf size
        for (int tb = lo; tb < hi; tb += kTileChunk) {
            const int T = min(kTileChunk, hi - tb);
            int hs = 0;   // the smallest H = 2^hs with ceil(T / H) <= kTileMaxM (H <= 16)
            while (((T + (1 << hs) - 1) >> hs) > kTileMaxM) ++hs;
            const int M = (T + (1 << hs) - 1) >> hs;
            switch ((hs << 4) | M) {
#define VPM_TILE_CASE(HH, MM)                                                                                       \
    case (HH << 4) | MM:                                                                                            \
        tile_chunk<MM, HH>(sm, t, src1, c, ccx, ccy, ih, n1, tb, T, fx, fy, out0, out1, velocity, u_inf, v_inf, err); \
        break;
#define VPM_TILE_ROW(HH) VPM_TILE_CASE(HH, 1) VPM_TILE_CASE(HH, 2) VPM_TILE_CASE(HH, 3) VPM_TILE_CASE(HH, 4)         \
    VPM_TILE_CASE(HH, 5) VPM_TILE_CASE(HH, 6)
                VPM_TILE_ROW(0) VPM_TILE_ROW(1) VPM_TILE_ROW(2) VPM_TILE_ROW(3) VPM_TILE_ROW(4)
#undef VPM_TILE_ROW
#undef VPM_TILE_CASE
                default: break;
            }
        }
    }
}

}  // namespace

cudaError_t set_coefficients2d(int P, bool exact, double* dst, cudaStream_t st) {
    std::vector<double> tab(3 * W * W, 0.0);
    double* m2m = tab.data() + kCoefM2M;
    double* m2l = tab.data() + kCoefM2L;
    double* l2l = tab.data() + kCoefL2L;
    for (int p = 0; p <= P; ++p) {
        for (int k = 1; k <= p; ++k) m2m[p * W + k] = (double)binom_host(p - 1, k - 1, exact) * ((double)p / (double)k);
        for (int k = 1; k <= P; ++k)
            m2l[p * W + k] = (double)binom_host(p + k - 1, k - 1, exact) * ((k & 1) ? -1.0 : 1.0) / (double)k;
        for (int k = p; k <= P; ++k) l2l[p * W + k] = (double)binom_host(k, p, exact);
    }
    cudaError_t e = cudaMemcpyAsync(dst, tab.data(), sizeof(double) * tab.size(), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    // The host vectors go out of scope: wait for the copies.
    return cudaStreamSynchronize(st);
}

// ---- upward pass in two launches ----------------------------------------------
//
// The multipole of any cell is a_k = sum of q_j (z_j - z_c)^k over the active
// particles of its subtree (P2M at a leaf, fmm2D.cpp:237-284), and M2M
// (fmm2D.cpp:309-379) shifts the children's moments with the binomial
// coefficients C(p, k) = C(p-1, k-1) p / k, which gives the same moments
// whenever those coefficients are exact (orders up to 18 with the reference's
// 32-bit binComb, any order with exact binomials). Every cell covers a
// contiguous range of the sorted particles, so a cell of at most kDirectMax
// particles takes its moments straight from that range (upward_direct2d: one
// warp per cell, all levels at once, no ordering between cells). The larger
// cells (the top of the tree, about n / kDirectMax per level) follow by M2M
// from their children in the cooperative level loop m2m_big_levels_coop,
// from the deepest level holding one. Sums run in a fixed order (lane order
// over the particles, then lanes in order; children in child order). A large
// cell without active particles gets zero moments from the first launch, so
// every cell's moments are written in every evaluation.
constexpr int kUpWarps = 8;
constexpr int kDirectMax = 1024;
constexpr int kUpMaxP = 18;

template <int P>
__global__ void __launch_bounds__(32 * kUpWarps)
upward_direct2d(Tree2D t, double2* __restrict__ a, unsigned* __restrict__ top_level, unsigned* err) {
    constexpr int Q = P + 1, CS = 2 * Q + 1;   // components per lane, padded row stride
    extern __shared__ double up_sm[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    double* red = up_sm + (size_t)wib * 32 * CS;   // [lane][component]
    if (fatal(err)) return;
    const int c_begin = t.info->level_start[1], c_end = t.info->n_cells;
    const int nw = gridDim.x * kUpWarps;
    for (int c = c_begin + blockIdx.x * kUpWarps + wib; c < c_end; c += nw) {
        const int lo = t.c_lo[c], hi = t.c_hi[c];
        const uint8_t f = t.c_flags[c];
        if (hi - lo > kDirectMax && !(f & CELL_LEAF)) {
            if (f & CELL_ACTIVE) {   // by M2M afterwards (m2m_big_levels_coop)
                if (lane == 0) atomicMax(top_level, (unsigned)t.c_level[c]);
            } else {                 // no active particle: zero moments (its parent's M2M reads them)
                for (int comp = lane; comp < 2 * Q; comp += 32) reinterpret_cast<double*>(a + (size_t)c * Q)[comp] = 0.0;
            }
            continue;
        }
        double re[Q], im[Q];
        #pragma unroll
        for (int k = 0; k < Q; ++k) re[k] = im[k] = 0.0;
        if (f & CELL_ACTIVE) {
            const double zx = t.c_cx[c], zy = t.c_cy[c];
            for (int j = lo + lane; j < hi; j += 32) {
                if (!t.pact[j]) continue;
                const double wx = t.px[j] - zx, wy = t.py[j] - zy;
                double pr = t.pq[j], pi = 0.0;
                re[0] += pr;
                #pragma unroll
                for (int k = 1; k < Q; ++k) {
                    const double nr = pr * wx - pi * wy, ni = pr * wy + pi * wx;
                    pr = nr;
                    pi = ni;
                    re[k] += pr;
                    im[k] += pi;
                }
            }
        }
        #pragma unroll
        for (int k = 0; k < Q; ++k) {
            red[lane * CS + 2 * k] = re[k];
            red[lane * CS + 2 * k + 1] = im[k];
        }
        __syncwarp();
        for (int comp = lane; comp < 2 * Q; comp += 32) {
            double sum = 0.0;
            for (int l = 0; l < 32; ++l) sum += red[l * CS + comp];
            reinterpret_cast<double*>(a + (size_t)c * Q)[comp] = sum;
        }
        __syncwarp();
    }
}

bool upward_direct_ok(int P, bool exact) { return P >= 1 && P <= kUpMaxP && (exact || P <= 18); }
static_assert(kUpMaxP <= 18, "the reference's 32-bit M2M binomials wrap from order 19");

template <int P>
cudaError_t launch_upward_direct(const Tree2D& t, Expansions2D& e, unsigned* err, cudaStream_t st, cudaEvent_t mid) {
    const size_t smem = sizeof(double) * kUpWarps * 32 * (2 * (P + 1) + 1);
    cudaError_t r = cudaFuncSetAttribute(upward_direct2d<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (r != cudaSuccess) return r;
    upward_direct2d<P><<<148 * 4, 32 * kUpWarps, smem, st>>>(t, e.a, t.gbar + 3, err);
    if (mid) {
        r = cudaEventRecord(mid, st);
        if (r != cudaSuccess) return r;
    }
    // A small grid: the large cells are a few hundred per level, and the
    // blocks of this loop wait at its barriers most of the time while the
    // near field runs beside it on the other streams, so every block it does
    // not hold is SM room for that (16 blocks: mixed step 0.442 -> 0.430 ms
    // at 778k against one block per SM).
    r = fmm2d_m2m_big(t, e, P, kDirectMax, std::max(16, t.n >> 16), err, st);
    return r != cudaSuccess ? r : cudaGetLastError();
}

// Upward pass of orders the direct form covers (upward_direct_ok): one launch.
// Otherwise the P2M + M2M level loop below.
cudaError_t fmm2d_upward_direct(const Tree2D& t, Expansions2D& e, int P, bool exact, unsigned* err, cudaStream_t st,
                                int* launches, cudaEvent_t mid) {
    // the level loop over all cells: every moment is final only at its end
    auto full = [&]() -> cudaError_t {
        cudaError_t r = fmm2d_upward(t, e, P, err, st, launches);
        if (r == cudaSuccess && mid) r = cudaEventRecord(mid, st);
        return r;
    };
    if (!upward_direct_ok(P, exact) || !t.gbar) return full();
    cudaError_t r;
    switch (P) {
#define VPM_UP_CASE(PP) \
    case PP: r = launch_upward_direct<PP>(t, e, err, st, mid); break;
        VPM_UP_CASE(1) VPM_UP_CASE(2) VPM_UP_CASE(3) VPM_UP_CASE(4) VPM_UP_CASE(5) VPM_UP_CASE(6)
        VPM_UP_CASE(7) VPM_UP_CASE(8) VPM_UP_CASE(9) VPM_UP_CASE(10) VPM_UP_CASE(11) VPM_UP_CASE(12)
        VPM_UP_CASE(13) VPM_UP_CASE(14) VPM_UP_CASE(15) VPM_UP_CASE(16) VPM_UP_CASE(17) VPM_UP_CASE(18)
#undef VPM_UP_CASE
        default: return full();
    }
    if (r != cudaSuccess) {   // cooperative launch refused: the level loop over all cells instead
        (void)cudaGetLastError();
        return full();
    }
    *launches += 2;
    return r;
}

// Upward pass: P2M of every active leaf, then M2M level by level from the
// deepest possible level up to level 1 (levels below the tree's depth exit
// at once; the launch count does not depend on the data, so the sequence can
// be captured in a CUDA graph).
cudaError_t fmm2d_upward(const Tree2D& t, Expansions2D& e, int P, unsigned* err, cudaStream_t st, int* launches) {
    cudaError_t r = cudaMemsetAsync(e.a, 0, sizeof(double2) * (size_t)t.cap_cells * (P + 1), st);
    if (r != cudaSuccess) return r;
    const size_t smem = sizeof(double2) * kP2MWarps * (P + 1) * kAccPad;
    p2m2d<<<148 * 16, 32 * kP2MWarps, smem, st>>>(t, e.a, P, err);
    *launches += 1;
    if (t.gbar) {
        int grid = 0;
        r = launch_coop(m2m_levels_coop, 32 * kLevelWarps, 0, st, 1, &grid, t, e.a, (const double*)e.coef, P,
                        t.gbar + 2, err);
        if (r == cudaSuccess) {
            *launches += 1;
            return cudaGetLastError();
        }
        (void)cudaGetLastError();  // cooperative launch refused: one launch per level instead
    }
    for (int L = t.key_levels - 1; L >= 1; --L) {
        m2m_level2d<<<148 * 4, 128, 0, st>>>(t, e.a, e.coef, P, L, err);
        *launches += 1;
    }
    return cudaGetLastError();
}

// List-2 operators T_tau (see m2l2d_op) for the 49 offset slots, from the
// same M2L coefficients as the direct formula (so the reference's binomials
// carry over). Upload synchronises `st`.
cudaError_t set_m2l_operators2d(int P, bool exact, double2* dst, cudaStream_t st) {
    std::vector<double2> op((size_t)49 * (P + 1) * P);
    for (int slot = 0; slot < 49; ++slot) {
        const int dx = slot % 7 - 3, dy = slot / 7 - 3;
        std::complex<double> tau(dx, dy), inv = (dx == 0 && dy == 0) ? 0.0 : 1.0 / tau;
        std::vector<std::complex<double>> ip(2 * P + 2);
        ip[0] = 1.0;
        for (int m = 1; m <= 2 * P; ++m) ip[m] = ip[m - 1] * inv;
        for (int p = 1; p <= P; ++p) {
            for (int k = 0; k <= P; ++k) {
                std::complex<double> v;
                if (k == 0) v = -(1.0 / (double)p) * ip[p];
                else v = -((double)binom_host(p + k - 1, k - 1, exact) * ((k & 1) ? -1.0 : 1.0) / (double)k) * ip[p + k];
                op[((size_t)slot * (P + 1) + k) * P + (p - 1)] = make_double2(v.real(), v.imag());
            }
        }
    }
    cudaError_t e = cudaMemcpyAsync(dst, op.data(), sizeof(double2) * op.size(), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(st);
}

cudaError_t fmm2d_m2l_only(const Tree2D& t, const Lists2D& l, Expansions2D& e, int P, unsigned* err,
                           cudaStream_t st, int* launches) {
    const int G = 32 / P;
    if (e.op) {
        const size_t smem = sizeof(double2) * 4 * (size_t)(2 * G * (P + 1) + G * (2 * P + 1));
        m2l2d_op<<<148 * 16, 128, smem, st>>>(t, l, e.a, e.b, e.op, e.coef, P, err);
    } else {
        const size_t smem = sizeof(double2) * 4 * (size_t)(G * (2 * P + 1) + 2 * G * (P + 1));
        m2l2d<<<148 * 16, 128, smem, st>>>(t, l, e.a, e.b, e.coef, P, err);
    }
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t fmm2d_l2l(const Tree2D& t, Expansions2D& e, int P, unsigned* err, cudaStream_t st, int* launches) {
    if (t.gbar) {
        int grid = 0;
        cudaError_t r = launch_coop(l2l_levels_coop, 32 * kLevelWarps, 0, st, 1, &grid, t, e.b,
                                    (const double*)e.coef, P, t.gbar + 4, err);
        if (r == cudaSuccess) {
            *launches += 1;
            return cudaGetLastError();
        }
        (void)cudaGetLastError();  // cooperative launch refused: one launch per level instead
    }
    for (int L = 3; L <= t.key_levels; ++L) {
        l2l_level2d<<<148 * 4, 128, 0, st>>>(t, e.b, e.coef, P, L, err);
        *launches += 1;
    }
    return cudaGetLastError();
}

cudaError_t fmm2d_m2l(const Tree2D& t, const Lists2D& l, Expansions2D& e, int P, unsigned* err, cudaStream_t st,
                      int* launches) {
    cudaError_t r = fmm2d_m2l_only(t, l, e, P, err, st, launches);
    if (r != cudaSuccess) return r;
    return fmm2d_l2l(t, e, P, err, st, launches);
}

cudaError_t fmm2d_eval(const Tree2D& t, const Lists2D& l, Expansions2D& e, int P, unsigned* err, cudaStream_t st,
                       int* launches) {
    eval2d<kEvalFull><<<148 * 16, kEvalThreads, 0, st>>>(t, l, e.a, e.b, e.fx, e.fy, P, nullptr, nullptr, nullptr,
                                                         nullptr, 0, 0.0, 0.0, kP2PListCsr, err);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t fmm2d_m2p(const Tree2D& t, const Lists2D& l, Expansions2D& e, int P, unsigned* err, cudaStream_t st,
                      int* launches, int lists) {
    eval2d<kEvalM2P><<<148 * 16, kEvalThreads, 0, st>>>(t, l, e.a, e.b, e.fx, e.fy, P, nullptr, nullptr, nullptr,
                                                        nullptr, 0, 0.0, 0.0, lists, err);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t fmm2d_eval_combine(const Tree2D& t, const Lists2D& l, Expansions2D& e, int P, const double* nx,
                               const double* ny, double* out0, double* out1, int velocity, double u_inf, double v_inf,
                               unsigned* err, cudaStream_t st, int* launches, bool m2p_done) {
    if (m2p_done)
        eval2d<kEvalL2P><<<148 * 16, kEvalThreads, 0, st>>>(t, l, e.a, e.b, e.fx, e.fy, P, nx, ny, out0, out1, velocity,
                                                            u_inf, v_inf, kP2PListCsr, err);
    else
        eval2d<kEvalFull><<<148 * 16, kEvalThreads, 0, st>>>(t, l, e.a, e.b, e.fx, e.fy, P, nx, ny, out0, out1,
                                                             velocity, u_inf, v_inf, kP2PListCsr, err);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t fmm2d_p2p_f32(const Tree2D& t, const Lists2D& l, const Expansions2D& e, double* out0, double* out1,
                          int velocity, double u_inf, double v_inf, unsigned* err, cudaStream_t st, int* launches,
                          bool near_only, int lists) {
    Expansions2D en = e;
    if (near_only) en.fx = en.fy = nullptr;
    // Many short blocks (a leaf or a few per warp) rather than one persistent
    // wave: blocks retire all through the launch, so the far-field kernels
    // running concurrently on the other streams get SM room as they queue.
    // the pass over the few leaves whose list 1 outgrew its slots: one wave
    const int grid = lists == kP2PListSpill ? 148 : 148 * 3 * 8;
    p2p2d_tile_f32<<<grid, 32 * kTileWarps, 0, st>>>(t, l, en.fx, en.fy, out0, out1, velocity, u_inf, v_inf, lists,
                                                    err);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t fmm2d_p2p_f64(const Tree2D& t, const Lists2D& l, const Expansions2D& e, double* out0, double* out1,
                          int velocity, double u_inf, double v_inf, unsigned* err, cudaStream_t st, int* launches,
                          bool near_only, int lists) {
    // Short blocks, as above.
    const int grid = lists == kP2PListSpill ? 148 * 2 : 148 * 3 * 16;
    near2d_f64<false><<<grid, 32 * kNear64Warps, 0, st>>>(t, l, near_only ? nullptr : e.fx, near_only ? nullptr : e.fy,
                                                          out0, out1, velocity, u_inf, v_inf, lists, err);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t fmm2d_p2p_potential(const Tree2D& t, const Lists2D& l, const Expansions2D& e, double* out, unsigned* err,
                                cudaStream_t st, int* launches) {
    near2d_f64<true><<<148 * 3 * 16, 32 * kNear64Warps, 0, st>>>(t, l, e.fx, nullptr, out, nullptr, 0, 0.0, 0.0,
                                                                 kP2PListCsr, err);
    *launches += 1;
    return cudaGetLastError();
}

}  // namespace vpm
