// List-2 M2L of the plain form per parent cell, FP64 (orders 1..16).
//
// The contraction of m2l_parent_f32 (m2l_tc.cu): with scaled expansions
// a~_k = a_k / r^k, b~_p = r^p b_p, the operator at offset tau factors as
//   T_tau[p][k] = tau^-p C[p][k] tau^-k,  C[p][0] = -1/p, C[p][k] = -m2l[p][k]
// (fmm2D.cpp:471-481; C from the reference's or the exact binomials), so one
// (child, source) pair is a diagonal complex scaling, one real P x (P + 1)
// matrix on the real and imaginary parts and another diagonal scaling: 300
// FP64 operations at P = 10 against 440 for the dense operator, and no
// operator to read: C and the powers of the 49 offsets are kernel parameters
// (constant bank). A block takes 32 parents, one per lane. The 32
// positions of the sources (children of the parent's neighbours) come into
// shared memory by cp.async, eight at a time and a step ahead; warp (child q,
// part h) applies the positions of its part that are not adjacent to its
// child (the scaling by 1 / r^k goes with tau^-k). The parts' sums are added
// in order, so the result does not depend on the schedule.
// Missing children and sources count as zero; a tree whose list 2 is not of
// this shape (l2_irregular) is left to m2l_list4_add.
// 778,377-particle boundary layer, P = 10: 72 us with list 4, against 133
// for a warp per target cell reading the 49 dense operators; in the captured
// graph, beside the near field, 581 us become 509.
#include <complex>

#include "fmm2d.cuh"

namespace vpm {

namespace {

constexpr int kPosAll = 32;    // positions of the 6 x 6 block around the children
constexpr int kPosStep = 8;    // positions staged at a time

template <int P>
struct ParF64Args {
    double C[P][P + 1];      // C[p - 1][k]
    double2 tp[49][P + 1];   // tau^-k, slot = (tau_y + 3) 7 + tau_x + 3
};

constexpr int kParts = 2;      // parts of the positions per child: eight warps

// 16 bytes global -> shared, zeros where there is no source.
__device__ __forceinline__ void cp_async16z(void* dst, const void* src, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(on ? 16 : 0)
                 : "memory");
}

// Offset of position j of the block from child (qx, qy), in cells.
__device__ __forceinline__ void offset(int j, int qx, int qy, int& tx, int& ty) {
    const int k8 = j >> 2, d = j & 3, nb = k8 < 4 ? k8 : k8 + 1;
    tx = 2 * (nb % 3 - 1) + (d & 1) - qx;
    ty = 2 * (nb / 3 - 1) + (d >> 1) - qy;
}

// Staged position jj (of the step from j0) onto the lane's sums. One at a
// time: with two, an entry of C feeds four FMAs, but both sources and the sums
// outgrow the registers above P = 10 and gain nothing below.
template <int P>
__device__ __forceinline__ void apply(const ParF64Args<P>& args, const double2* st, const double (*s_rp)[32], int jj,
                                      int slot, double* accr, double* acci) {
    constexpr int Q = P + 1;
    const int lane = threadIdx.x & 31;
    double ar[Q], ai[Q];
    {
        const double2 v = st[jj * Q * 32 + lane];
        ar[0] = v.x;
        ai[0] = v.y;
    }
    #pragma unroll
    for (int k = 1; k < Q; ++k) {
        const double2 v = st[(jj * Q + k) * 32 + lane];
        const double2 w = cscale(args.tp[slot][k], s_rp[k][lane]);
        ar[k] = v.x * w.x - v.y * w.y;
        ai[k] = v.x * w.y + v.y * w.x;
    }
    #pragma unroll
    for (int p = 0; p < P; ++p) {
        double br = 0.0, bi = 0.0;
        #pragma unroll
        for (int k = 0; k < Q; ++k) {
            br = fma(args.C[p][k], ar[k], br);
            bi = fma(args.C[p][k], ai[k], bi);
        }
        const double2 w = args.tp[slot][p + 1];
        accr[p] = fma(w.x, br, fma(-w.y, bi, accr[p]));
        acci[p] = fma(w.x, bi, fma(w.y, br, acci[p]));
    }
}

template <int P>
__global__ void __launch_bounds__(128 * kParts)
m2l_parent_f64(Tree2D t, const int32_t* __restrict__ blk, const double2* __restrict__ a, double2* __restrict__ b,
               const __grid_constant__ ParF64Args<P> args, unsigned* err) {
    constexpr int Q = P + 1, NP = kParts, PER = kPosStep / NP, kStage = kPosStep * Q * 32;
    extern __shared__ double2 sm_a[];               // 2 x [kPosStep][Q][32], then the sums [4][2 P][32]
    __shared__ int s_src[kPosAll][32];              // [position][parent]
    __shared__ double s_rp[Q][32];                  // [k][parent]: (1 / child length)^k
    if (fatal(err)) return;
    const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
    const int q = wq & 3, h = wq >> 2;
    const int qx = q & 1, qy = q >> 1;
    const int np = t.info->n_cells - t.info->n_leaves;   // non-leaf cells; the root is the first
    const bool irregular = t.info->l2_irregular != 0;
    const double root = t.geom->root;
    for (int tile = blockIdx.x; 1 + tile * 32 < np; tile += gridDim.x) {
        const int pi = 1 + tile * 32 + lane;
        const int par = pi < np ? t.nonleaf[pi] : -1;
        if (wq == 0) {
            const double rinv = par >= 0 ? ldexp(1.0, (int)t.c_level[par] + 1) / root : 0.0;
            double r = 1.0;
            #pragma unroll
            for (int k = 0; k < Q; ++k) {
                s_rp[k][lane] = r;
                r *= rinv;
            }
        }
        for (int j4 = wq; j4 < kPosAll / 4; j4 += 4 * NP) {
            int4 v = make_int4(-1, -1, -1, -1);
            if (par >= 0 && !irregular) v = __ldg(reinterpret_cast<const int4*>(blk + (size_t)par * kPosAll) + j4);
            s_src[4 * j4][lane] = v.x;
            s_src[4 * j4 + 1][lane] = v.y;
            s_src[4 * j4 + 2][lane] = v.z;
            s_src[4 * j4 + 3][lane] = v.w;
        }
        double accr[P], acci[P];
        #pragma unroll
        for (int p = 0; p < P; ++p) accr[p] = acci[p] = 0.0;
        __syncthreads();   // s_src is written
        auto fetch = [&](int j0) {
            // item (j, m, k), k fastest (a source's moments are contiguous)
            double2* st = sm_a + ((j0 / kPosStep) & 1) * kStage;
            if (j0 < kPosAll)
                for (int idx = threadIdx.x; idx < kStage; idx += 128 * NP) {
                    const int jm = idx / Q, k = idx - jm * Q;
                    const int j = jm >> 5, m = jm & 31;
                    const int src = s_src[j0 + j][m];
                    cp_async16z(&st[(j * Q + k) * 32 + m], a + (size_t)max(src, 0) * Q + k, src >= 0);
                }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        fetch(0);
        for (int j0 = 0; j0 < kPosAll; j0 += kPosStep) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();   // this step's sources have landed; the last step's are read
            fetch(j0 + kPosStep);
            const double2* st = sm_a + ((j0 / kPosStep) & 1) * kStage;
            #pragma unroll 1
            for (int jj = h * PER; jj < (h + 1) * PER; ++jj) {
                const int j = j0 + jj;
                int tx, ty;
                offset(j, qx, qy, tx, ty);
                if (tx >= -1 && tx <= 1 && ty >= -1 && ty <= 1) continue;   // adjacent: not in this child's list 2
                if (!__any_sync(0xffffffffu, s_src[j][lane] >= 0)) continue;
                apply<P>(args, st, s_rp, jj, (ty + 3) * 7 + tx + 3, accr, acci);
            }
        }
        // the parts' sums, in order
        double* sum = reinterpret_cast<double*>(sm_a) + (size_t)q * 2 * P * 32 + lane;
        #pragma unroll 1
        for (int hh = 0; hh < NP; ++hh) {
            __syncthreads();
            if (hh == h) {
                #pragma unroll
                for (int p = 0; p < P; ++p) {
                    if (hh > 0) {
                        accr[p] = sum[p * 32] + accr[p];
                        acci[p] = sum[(P + p) * 32] + acci[p];
                    }
                    if (hh < NP - 1) {
                        sum[p * 32] = accr[p];
                        sum[(P + p) * 32] = acci[p];
                    }
                }
            }
        }
        if (h == NP - 1 && par >= 0) {
            const unsigned m = t.c_chmask[par];
            if (m & (1u << q)) {
                const int ch = t.c_child0[par] + __popc(m & ((1u << q) - 1u));
                double2* bc = b + (size_t)ch * Q;
                bc[0] = make_double2(0.0, 0.0);
                #pragma unroll
                for (int p = 0; p < P; ++p) {
                    const double rk = s_rp[p + 1][lane];
                    bc[p + 1] = make_double2(accr[p] * rk, acci[p] * rk);
                }
            }
        }
        __syncthreads();
    }
}

template <int P>
cudaError_t launch_m2l_parent_f64(const Tree2D& t, const Lists2D& l, Expansions2D& e, bool exact, unsigned* err,
                                  cudaStream_t st) {
    constexpr int Q = P + 1;
    ParF64Args<P> args;
    for (int p = 1; p <= P; ++p) {
        args.C[p - 1][0] = -1.0 / (double)p;
        for (int k = 1; k <= P; ++k)
            args.C[p - 1][k] = -((double)binom_m2l_host(p + k - 1, k - 1, exact) * ((k & 1) ? -1.0 : 1.0) / (double)k);
    }
    for (int slot = 0; slot < 49; ++slot) {
        const int dx = slot % 7 - 3, dy = slot / 7 - 3;
        const std::complex<double> inv = (dx == 0 && dy == 0) ? 0.0 : 1.0 / std::complex<double>(dx, dy);
        std::complex<double> w = 1.0;
        for (int k = 0; k <= P; ++k) {
            args.tp[slot][k] = make_double2(w.real(), w.imag());
            w *= inv;
        }
    }
    constexpr size_t stage = sizeof(double2) * 2 * kPosStep * Q * 32, sums = sizeof(double) * 4 * 2 * P * 32;
    constexpr size_t smem = stage > sums ? stage : sums;
    cudaError_t r = cudaFuncSetAttribute(m2l_parent_f64<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (r != cudaSuccess) return r;
    m2l_parent_f64<P><<<148 * 2, 128 * kParts, smem, st>>>(t, l.l2_blk, e.a, e.b, args, err);
    return cudaGetLastError();
}

}  // namespace

bool m2l_parent_f64_supported(const Tree2D& t, const Lists2D& l, int P) {
    return P >= 1 && P <= 16 && l.l2_blk && t.nonleaf;
}

cudaError_t fmm2d_m2l_parent_f64(const Tree2D& t, const Lists2D& l, Expansions2D& e, int P, bool exact, unsigned* err,
                                 cudaStream_t st, int* launches) {
    if (!m2l_parent_f64_supported(t, l, P)) return cudaErrorInvalidValue;
    cudaError_t r;
    switch (P) {
#define VPM_CASE(PP) \
    case PP: r = launch_m2l_parent_f64<PP>(t, l, e, exact, err, st); break;
        VPM_CASE(1) VPM_CASE(2) VPM_CASE(3) VPM_CASE(4) VPM_CASE(5) VPM_CASE(6) VPM_CASE(7) VPM_CASE(8)
        VPM_CASE(9) VPM_CASE(10) VPM_CASE(11) VPM_CASE(12) VPM_CASE(13) VPM_CASE(14) VPM_CASE(15) VPM_CASE(16)
#undef VPM_CASE
        default: return cudaErrorInvalidValue;
    }
    if (r != cudaSuccess) return r;
    *launches += 1;
    return fmm2d_m2l_list4(t, l, e, P, err, st, launches);
}

}  // namespace vpm
