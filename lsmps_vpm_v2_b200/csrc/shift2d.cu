// M2M of the large cells and L2L of the leaves (2D), with one lane per
// expansion: a lane holds all P + 1 coefficients in registers and shifts them
// in place by repeated synthetic division (Horner's scheme for a polynomial
// about a new centre),
//   L2L  b_p <- sum_{k >= p} C(k, p) t^(k-p) b_k   : P (P + 1) / 2 steps b_k += t b_(k+1)
//   M2M  a_p <- sum_{k <= p} C(p, k) t^(p-k) a_k   : as many steps a_k += t a_(k-1)
// (fmm2D.cpp:587-651 and 309-379, with exact binomials), which needs no
// coefficient table, no powers and no other lane. A lane per coefficient, as
// before, left P + 1 of 32 lanes on a cell, half of them idle in the
// triangular sums, and walked a chain of dependent loads per term.
#include "fmm2d.cuh"

namespace vpm {

static_assert(kL2LMaxP == kMaxP, "an order per instantiation");

namespace {

constexpr int kShiftWarps = 8;

// One lane per child of a large cell (eight cells per warp), levels *top_level
// .. 1 with a grid barrier between them: the cells of more than min_count
// particles, the others are final already. A warp looks through 32 cells at a
// time and works off the large ones. Children are added pairwise, (0 + 1) +
// (2 + 3). Bound by the barriers and one round of loads and shifts per level:
// 6 to 8 us a level. 778,377-particle boundary layer, P = 10: 50 us (94 with a
// lane per coefficient); 530,888 particles, P = 16: 63 us (149).
template <int P>
__global__ void __launch_bounds__(32 * kShiftWarps)
m2m_big_levels_coop(Tree2D t, double2* __restrict__ a, int min_count, const unsigned* __restrict__ top_level,
                    unsigned* bar, unsigned* err) {
    constexpr int Q = P + 1;
    __shared__ int s_big[kShiftWarps][32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int g = lane >> 2, q = lane & 3;
    const int warps = gridDim.x * kShiftWarps, gw = blockIdx.x * kShiftWarps + wib;
    const int top = (int)*top_level;
    for (int L = top; L >= 1; --L) {
        const bool skip = block_fatal(err);
        const int c0 = skip ? 0 : t.info->level_start[L], c1 = skip ? 0 : t.info->level_start[L + 1];
        for (int cb = c0 + gw * 32; cb < c1; cb += warps * 32) {
            const int cc = cb + lane;
            bool big = false;
            if (cc < c1) {
                const uint8_t f = t.c_flags[cc];
                big = !(f & CELL_LEAF) && (f & CELL_ACTIVE) && t.c_hi[cc] - t.c_lo[cc] > min_count;
            }
            const unsigned m = __ballot_sync(0xffffffffu, big);
            if (big) s_big[wib][__popc(m & ((1u << lane) - 1u))] = cc;
            __syncwarp();
            const int nb = __popc(m);
            for (int i = 0; i < nb; i += 8) {   // warp-uniform
                const int c = i + g < nb ? s_big[wib][i + g] : -1;
                double2 v[Q];
                #pragma unroll
                for (int k = 0; k < Q; ++k) v[k] = make_double2(0.0, 0.0);
                if (c >= 0) {
                    const unsigned cm = t.c_chmask[c];
                    const int ch0 = t.c_child0[c];
                    if (ch0 >= 0 && ((cm >> q) & 1u)) {
                        const int ch = ch0 + __popc(cm & ((1u << q) - 1u));
                        const double2 tt = make_double2(t.c_cx[ch] - t.c_cx[c], t.c_cy[ch] - t.c_cy[c]);
                        #pragma unroll
                        for (int k = 0; k < Q; ++k) v[k] = __ldcg(&a[(size_t)ch * Q + k]);
                        #pragma unroll
                        for (int s = 1; s < Q; ++s)
                            #pragma unroll
                            for (int k = P; k >= s; --k) v[k] = cfma(tt, v[k - 1], v[k]);
                    }
                }
                #pragma unroll
                for (int k = 0; k < Q; ++k) {
                    v[k].x += __shfl_xor_sync(0xffffffffu, v[k].x, 1);
                    v[k].y += __shfl_xor_sync(0xffffffffu, v[k].y, 1);
                    v[k].x += __shfl_xor_sync(0xffffffffu, v[k].x, 2);
                    v[k].y += __shfl_xor_sync(0xffffffffu, v[k].y, 2);
                    if (c >= 0 && (k & 3) == q) a[(size_t)c * Q + k] = v[k];
                }
            }
            __syncwarp();
        }
        if (L > 1) grid_sync_counter(bar, err);
    }
}

// Full local expansion of every leaf from the M2L parts of its ancestors at
// levels 2 .. L-1, one lane per leaf: the coarsest ancestor's expansion is
// shifted to the next one's centre, that one's part added, and so on down to
// the leaf. Equal to the level-by-level pull of fmm2D.cpp:587-651 up to
// rounding (shifts of a degree-P polynomial compose exactly), without a level
// loop or a grid barrier. Ancestors come from the dense grid (written for
// every cell of levels <= dense_levels by the tree build, so an ancestor's
// entry is always current) and, below it, the parent chain, walked once. The
// next ancestor's index and centre are loaded while the current part is shifted.
// 778,377-particle boundary layer, P = 10: 14 us (37 with a lane per
// coefficient, P + 1 of 32 lanes on a leaf); 530,888 particles, P = 16: 20 us
// (80). Above P = 16 the registers of two expansions grow, and from 27 on they
// spill: 600,000 particles, P = 17, 20, 24, 27, 30: 18, 23, 29, 35, 41 us (57, 57,
// 72, 72, 76); 100,000: 12, 14, 16, 18, 23 (18, 18, 21, 23, 23). Leaves down to
// level 27 (6,000 particles in eight nested blobs), P = 16: 37 us (38, and 41
// with a walk of the chain for every level).
constexpr int kLeafShiftWarps = 2;   // few leaves per SM: small blocks spread them

template <int P>
__global__ void __launch_bounds__(32 * kLeafShiftWarps)
l2l_leaves2d(Tree2D t, double2* __restrict__ b, const unsigned* err) {
    constexpr int Q = P + 1;
    if (fatal(err)) return;   // n_leaves is then set, leaf_cells and the cell records need not be
    const int nl = t.info->n_leaves, nc = t.info->n_cells;
    const int dlev = t.dense ? t.dense_levels : 1;
    for (int li = blockIdx.x * blockDim.x + threadIdx.x; li < nl; li += gridDim.x * blockDim.x) {
        const int c = t.leaf_cells[li];
        const int L = t.c_level[c];
        if (L <= 2) continue;
        const int ix = t.c_ix[c], iy = t.c_iy[c];
        int chain[kMaxLevels2D];   // ancestors below the dense grid, from one walk up
        for (int l = L - 1, a = c; l > dlev && l >= 2; --l) chain[l] = a = t.c_parent[a];
        auto ancestor = [&](int m) {
            const int sh = L - m;
            const int a = m <= dlev ? t.dense[start_id2(m) + (ix >> sh) + ((int64_t)(iy >> sh) << m)] : chain[m];
            return a >= 0 && a < nc ? a : c;   // always a cell; c itself would add nothing wrong to read
        };
        auto centre = [&](int a) { return make_double2(t.c_cx[a], t.c_cy[a]); };
        int an = ancestor(2);
        double2 zn = centre(an), z = zn;
        double2 v[Q];
        #pragma unroll
        for (int k = 0; k < Q; ++k) v[k] = make_double2(0.0, 0.0);
        for (int m = 2; m <= L; ++m) {
            const int a = an;
            const double2 tt = make_double2(zn.x - z.x, zn.y - z.y);
            z = zn;
            double2 w[Q];
            #pragma unroll
            for (int k = 0; k < Q; ++k) w[k] = b[(size_t)a * Q + k];
            if (m < L) {
                an = m + 1 < L ? ancestor(m + 1) : c;
                zn = centre(an);
            }
            if (m > 2) {
                #pragma unroll
                for (int s = 0; s < P; ++s)
                    #pragma unroll
                    for (int k = P - 1; k >= s; --k) v[k] = cfma(tt, v[k + 1], v[k]);
            }
            #pragma unroll
            for (int k = 0; k < Q; ++k) v[k] = cadd(v[k], w[k]);
        }
        #pragma unroll
        for (int k = 0; k < Q; ++k) b[(size_t)c * Q + k] = v[k];
    }
}

template <int P>
cudaError_t launch_m2m_big(const Tree2D& t, Expansions2D& e, int min_count, int max_grid, unsigned* err,
                           cudaStream_t st) {
    int grid = 0;
    return launch_coop_max(m2m_big_levels_coop<P>, 32 * kShiftWarps, 0, st, 1, max_grid, &grid, t, e.a, min_count,
                           (const unsigned*)(t.gbar + 3), t.gbar + 2, err);
}

template <int P>
cudaError_t launch_l2l_leaves(const Tree2D& t, Expansions2D& e, unsigned* err, cudaStream_t st) {
    l2l_leaves2d<P><<<148 * 8, 32 * kLeafShiftWarps, 0, st>>>(t, e.b, err);
    return cudaGetLastError();
}

}  // namespace

#define VPM_SHIFT_CASES                                                                                          \
    VPM_CASE(1) VPM_CASE(2) VPM_CASE(3) VPM_CASE(4) VPM_CASE(5) VPM_CASE(6) VPM_CASE(7) VPM_CASE(8) VPM_CASE(9)  \
    VPM_CASE(10) VPM_CASE(11) VPM_CASE(12) VPM_CASE(13) VPM_CASE(14) VPM_CASE(15) VPM_CASE(16) VPM_CASE(17)      \
    VPM_CASE(18)

cudaError_t fmm2d_m2m_big(const Tree2D& t, Expansions2D& e, int P, int min_count, int max_grid, unsigned* err,
                          cudaStream_t st) {
    switch (P) {
#define VPM_CASE(PP) case PP: return launch_m2m_big<PP>(t, e, min_count, max_grid, err, st);
        VPM_SHIFT_CASES
#undef VPM_CASE
        default: return cudaErrorInvalidValue;
    }
}

bool l2l_direct_ok(int P, bool exact) { return P >= 1 && P <= kL2LMaxP && (exact || P <= 17); }

cudaError_t fmm2d_l2l_leaves(const Tree2D& t, Expansions2D& e, int P, unsigned* err, cudaStream_t st, int* launches) {
    *launches += 1;
    switch (P) {
#define VPM_CASE(PP) case PP: return launch_l2l_leaves<PP>(t, e, err, st);
        VPM_SHIFT_CASES VPM_CASE(19) VPM_CASE(20) VPM_CASE(21) VPM_CASE(22) VPM_CASE(23) VPM_CASE(24) VPM_CASE(25)
        VPM_CASE(26) VPM_CASE(27) VPM_CASE(28) VPM_CASE(29) VPM_CASE(30)
#undef VPM_CASE
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace vpm
