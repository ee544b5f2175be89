// 3D treecode evaluation (fastFMM3Dutils::evaluateFMM, src/FMM/fast3DFMM.cpp:318-472):
// every particle is a target; from the root's children down, each active
// child k of a cell on the target's list is
//   far   if R^2 > (s size_k)^2   -> M2P with the derivative multipliers of
//                                    fmm3D::M2P_mul_calc (fmm3D.cpp:147-200)
//   else a non-leaf               -> onto the target's list for the next level
//   else a leaf                   -> P2P  u += (alpha_j x r) / |r|^3, j != i,
//                                    active j only (fast3DFMM.cpp:440-460)
// The reference's TreeCell path (fmm3D::calcVelocity, VELOCITY_CALCULATION_TYPE
// 2, fmm3D.cpp:1264-1360; calcVelocityNearBody, fmm3D.cpp:1406-1606) walks
// its TreeCell the same way, with every particle of a near leaf a source.
// (level-1 cells themselves are never evaluated, as in the reference).
// s is the reference's support factor 2 (fast3DFMM.cpp:4) unless the caller
// asks for a stricter far test (a larger s: more accurate, slower).
//
// One block per 64 consecutive particles in leaf order (a few neighbouring
// leaves); every lane holds two of them as its targets, the same ones in every
// warp. The block walks the tree once for all its targets, depth first; an
// entry carries the mask of the targets whose own walk holds it, so every
// target makes exactly its own reference decisions, whichever others share
// its block.
//
// What bounds it: the pairs (about 75 FP64 operations per M2P, 22 per P2P;
// FP32 alike in the mixed form) against the 128 bytes a cycle that an SM reads
// from shared memory, and everything else kept off their path. Candidates are
// classified one per lane against the box of the block's targets: the test's
// operations are rounded one by one and each is monotone in the target's
// coordinates, so the values formed from the box's faces bound those of every
// target inside it exactly, and a cell that is far (near) by its bound is far
// (near) for every target by the reference's own rounded test. Only the cells
// in between are tested target by target. Far cells and near leaves go to
// lists that the warps then share out, all lanes on one cell, with moments and
// sources staged in shared memory ahead of their use. A record read by 32
// lanes costs the SM 8 bytes a lane of its 128 a cycle, more than the
// arithmetic of one target per lane takes (42 doubles a record and one target
// per lane: 84 cycles against 36, the whole kernel 2.17 ms on the 222,688-
// particle ring): hence two targets per lane and a record of 30 doubles.
// A walk that tested, summed and descended cell by cell, one target per lane,
// took 5.17 ms there (FP64) and 30.5 ms on the 2,009,183-particle ring
// (mixed), waiting for dependent loads; this one takes 1.96 and 21.2 ms.
#include "fmm3d.cuh"

#include <cmath>

namespace vpm {

namespace {

constexpr int kStack3D = 1024;   // walk entries per block
constexpr int kStageM = 4;       // far cells staged per warp: two in use, two ahead

// Record of a far cell as the evaluation stages it: centre, then the moments.
// FP64 (pack3d_f64): 30 doubles, see m2p64. Mixed (prep3d_f32): 3 doubles and
// 30 floats.
constexpr int kRec64Bytes = kMom3D * 8;
constexpr int kRec32Bytes = kRec32Floats * 4;
static_assert(kRec64Bytes % 16 == 0 && kRec32Bytes % 16 == 0, "staged with 16-byte copies");

// The two targets of a lane and their sums.
struct Targets {
    double x[2], y[2], z[2];
    double vx[2], vy[2], vz[2];
    int slot[2];
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// 1 / sqrt(a) in FP64: the hardware's approximation (about 20 bits) and one
// step of Halley's method, y + y e (1/2 + 3/8 e) with e = 1 - a y^2, whose
// error is of order e^3.
__device__ __forceinline__ double rsqrt_halley(double a) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-(a * y), y, 1.0);
    return fma(fma(e, 0.375, 0.5), y * e, y);
}

// v += s (a, b, c) where `on`, as three predicated operations: what leads up
// to them runs for every lane, without a branch between independent pairs,
// and a lane that is not `on` keeps its sums whatever the values are.
__device__ __forceinline__ void add3_if(bool on, double s, double a, double b, double c, double& vx, double& vy,
                                        double& vz) {
    asm("{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.s32 p, %3, 0;\n\t"
        "@p fma.rn.f64 %0, %5, %4, %0;\n\t"
        "@p fma.rn.f64 %1, %6, %4, %1;\n\t"
        "@p fma.rn.f64 %2, %7, %4, %2;\n\t"
        "}"
        : "+d"(vx), "+d"(vy), "+d"(vz)
        : "r"((int)on), "d"(s), "d"(a), "d"(b), "d"(c));
}

// M2P of one far cell, FP64 (fast3DFMM.cpp:395-425 with the multipliers of
// fmm3D.cpp:147-200). With r = target - centre and, for source component c,
// F_c = sum_m M_c,m g_m (g the derivatives of r / |r|^3), the velocity is
// (F_y,z - F_z,y, F_z,x - F_x,z, F_x,y - F_y,x). The derivative tensors are
// symmetric and (being those of a harmonic function) blind to the trace of
// the second moments, so with traceless second moments q_c
//   F_c = r S_c + D_c / R^3 - 3 / R^5 W_c,
//   S_c = M0_c / R^3 - 3 / R^5 (D_c . r) + 15 / R^7 P_c,
//   P_c = r . q_c r,   W_c,i = 2 q_ii r_i + sum_{k != i} q_ik r_k,
// and the antisymmetric combination of D and W is a vector A of differences
// of D and a 3 x 3 matrix K of differences of q:
//   u = 1/R^3 [ A - 3 K r / R^2 + S~ x r ],
//   S~_c = M0_c - 3 / R^2 (D_c . r - 5 P_c / R^2).
// 73 operations per target and 14 per cell, against about 230 for the thirty
// multipliers and their products. K and A cost fewer cycles formed here, once
// for both targets, than read from a longer record.
// Record: [0..2] centre, [3..5] M0, [6..14] D by component, [15..29] per
// component -5 (q_xx, q_yy, q_xy, q_yz, q_xz).
// Targets first .. last; one that is not `on` (its cell is near) adds nothing.
template <int FIRST, int LAST>
__device__ __forceinline__ void m2p64(const double2* __restrict__ rec, const bool* on, Targets& t) {
    double M[kMom3D];
    #pragma unroll
    for (int i = 0; i < kMom3D / 2; ++i) {
        const double2 v = rec[i];
        M[2 * i] = v.x;
        M[2 * i + 1] = v.y;
    }
    const double *Dx = M + 6, *Dy = M + 9, *Dz = M + 12, *qx = M + 15, *qy = M + 20, *qz = M + 25;
    const double Ax = Dy[2] - Dz[1], Ay = Dz[0] - Dx[2], Az = Dx[1] - Dy[0];
    // entries of q: 0 xx, 1 yy, 2 xy, 3 yz, 4 xz; zz = -(xx + yy)
    const double Kxx = qy[4] - qz[2], Kxy = fma(-2.0, qz[1], qy[3]), Kxz = fma(-2.0, qy[0] + qy[1], -qz[3]);
    const double Kyx = fma(2.0, qz[0], -qx[4]), Kyy = qz[2] - qx[3], Kyz = fma(2.0, qx[0] + qx[1], qz[4]);
    const double Kzx = fma(-2.0, qy[0], qx[2]), Kzy = fma(2.0, qx[1], -qy[2]), Kzz = qx[3] - qy[4];
    #pragma unroll
    for (int h = FIRST; h <= LAST; ++h) {
        const double x = t.x[h] - M[0], y = t.y[h] - M[1], z = t.z[h] - M[2];
        const double xx = x * x, yy = y * y, zz = z * z;
        const double iR = rsqrt_halley(xx + yy + zz);
        const double i2 = iR * iR, i3 = i2 * iR, i2a = -3.0 * i2, i2k = 0.6 * i2;
        const double a = xx - zz, b = yy - zz, xy = x * y, yz = y * z, xz = x * z;
        double S[3];
        #pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double* D = M + 6 + 3 * c;
            const double* q = M + 15 + 5 * c;
            const double P = fma(q[0], a, fma(q[1], b, fma(q[2], xy, fma(q[3], yz, q[4] * xz))));
            S[c] = fma(i2a, fma(D[0], x, fma(D[1], y, fma(D[2], z, i2 * P))), M[3 + c]);
        }
        const double wx = fma(i2k, fma(Kxx, x, fma(Kxy, y, Kxz * z)), Ax);
        const double wy = fma(i2k, fma(Kyx, x, fma(Kyy, y, Kyz * z)), Ay);
        const double wz = fma(i2k, fma(Kzx, x, fma(Kzy, y, Kzz * z)), Az);
        add3_if(on[h], i3, fma(S[1], z, fma(-S[2], y, wx)), fma(S[2], x, fma(-S[0], z, wy)),
                fma(S[0], y, fma(-S[1], x, wz)), t.vx[h], t.vy[h], t.vz[h]);
    }
}

// The same in FP32 (mixed form), by the thirty multipliers: offsets rounded to
// float after the FP64 subtraction, moments from their FP32 copy, the cell's
// sum formed in FP32 and added to the FP64 total. Where a sum of products can
// be contracted in more than one way the form is written out, so the result
// does not depend on how the compiler combines it with its surroundings.
__device__ __forceinline__ void m2p32(const float* __restrict__ M, double dxd, double dyd, double dzd,
                                      double& vx, double& vy, double& vz) {
    const float dx = (float)dxd, dy = (float)dyd, dz = (float)dzd;
    const float R2 = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
    const float iR = rsqrtf(R2);
    const float i2 = iR * iR;
    const float i3 = i2 * iR;
    const float i5 = i3 * i2, i7 = i5 * i2;
    const float a5x = 3.f * i5 * dx, a5y = 3.f * i5 * dy, a5z = 3.f * i5 * dz;
    const float b7 = 15.f * i7;
    float gx[10], gy[10], gz[10];
    gx[0] = dx * i3;
    gx[1] = -(a5x * dx) + i3;
    gx[2] = -(a5x * dy);
    gx[3] = -(a5x * dz);
    gx[4] = __fmaf_rn(b7 * dx * dx, dx, -__fmul_rn(3.f, a5x));
    gx[5] = (b7 * dx * dy * dy) - a5x;
    gx[6] = (b7 * dx * dz * dz) - a5x;
    gx[7] = (b7 * dx * dx * dy) - a5y;
    gx[8] = (b7 * dx * dy * dz);
    gx[9] = (b7 * dx * dx * dz) - a5z;
    gy[0] = dy * i3;
    gy[1] = -(a5y * dx);
    gy[2] = -(a5y * dy) + i3;
    gy[3] = -(a5y * dz);
    gy[4] = (b7 * dy * dx * dx) - a5y;
    gy[5] = __fmaf_rn(b7 * dy * dy, dy, -__fmul_rn(3.f, a5y));
    gy[6] = (b7 * dy * dz * dz) - a5y;
    gy[7] = (b7 * dy * dx * dy) - a5x;
    gy[8] = (b7 * dy * dy * dz) - a5z;
    gy[9] = (b7 * dy * dx * dz);
    gz[0] = dz * i3;
    gz[1] = -(a5z * dx);
    gz[2] = -(a5z * dy);
    gz[3] = -(a5z * dz) + i3;
    gz[4] = (b7 * dz * dx * dx) - a5z;
    gz[5] = (b7 * dz * dy * dy) - a5z;
    gz[6] = __fmaf_rn(b7 * dz * dz, dz, -__fmul_rn(3.f, a5z));
    gz[7] = (b7 * dz * dx * dy);
    gz[8] = (b7 * dz * dy * dz) - a5y;
    gz[9] = (b7 * dz * dx * dz) - a5x;
    float sx = 0.f, sy = 0.f, sz = 0.f;
    #pragma unroll
    for (int m = 0; m < 10; ++m) {
        const float mx = M[m], my = M[10 + m], mz = M[20 + m];
        sx = __fadd_rn(sx, __fmaf_rn(my, gz[m], -__fmul_rn(mz, gy[m])));
        sy = __fadd_rn(sy, __fmaf_rn(mz, gx[m], -__fmul_rn(mx, gz[m])));
        sz = __fadd_rn(sz, __fmaf_rn(mx, gy[m], -__fmul_rn(my, gx[m])));
    }
    vx += sx;
    vy += sy;
    vz += sz;
}

// One warp per cell: for a leaf (no children), the offsets from its centre
// and the alphas of its particles; then every cell's record (grid-stride).
__global__ void __launch_bounds__(256) prep3d_f32_kernel(Tree3D t, unsigned* err) {
    if (fatal(err)) return;
    const int lane = threadIdx.x & 31;
    const int nc = t.info->n_cells;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < nc; c += warps) {
        const double cx = t.c_x[c], cy = t.c_y[c], cz = t.c_z[c];
        float* rec = t.rec32 + (size_t)c * kRec32Floats;
        if (lane < 3) reinterpret_cast<double*>(rec)[lane] = lane == 0 ? cx : lane == 1 ? cy : cz;
        if (lane < 30) rec[6 + lane] = (float)t.mom[(size_t)c * kMom3D + lane];
        if (t.c_chmask[c] != 0) continue;
        for (int j = t.c_lo[c] + lane; j < t.c_hi[c]; j += 32) {
            t.ps32[j] = make_float4((float)(t.px[j] - cx), (float)(t.py[j] - cy), (float)(t.pz[j] - cz),
                                    t.pact[j] ? 1.f : 0.f);
            t.as32[j] = make_float4((float)t.ax[j], (float)t.ay[j], (float)t.az[j], 0.f);
        }
    }
}

// The thirty moments of every cell (three components of 1, x, y, z, xx, yy,
// zz, xy, yz, xz) rewritten in place as the record of m2p64, eight cells per
// warp through shared memory. Runs once after M2M, which needs the moments as
// they are; bound by its 480 bytes of traffic per cell.
constexpr int kPackWarps = 4, kPackCells = 8;
__global__ void __launch_bounds__(32 * kPackWarps) pack3d_f64_kernel(Tree3D t, unsigned* err) {
    __shared__ double s_in[kPackWarps][kPackCells][kMom3D + 1], s_out[kPackWarps][kPackCells][kMom3D + 1];
    if (fatal(err)) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nc = t.info->n_cells;
    const int step = gridDim.x * kPackWarps * kPackCells;
    for (int c0 = (blockIdx.x * kPackWarps + w) * kPackCells; c0 < nc; c0 += step) {
        const int m = min(kPackCells, nc - c0);
        for (int k = 0; k < m; ++k)
            if (lane < kMom3D) s_in[w][k][lane] = t.mom[(size_t)(c0 + k) * kMom3D + lane];
        __syncwarp();
        const int k = lane >> 2, c = lane & 3;   // cell of the batch, component
        if (k < m && c < 3) {
            const double* Mc = s_in[w][k] + 10 * c;
            double* out = s_out[w][k];
            const double tr = (Mc[4] + Mc[5] + Mc[6]) * (1.0 / 3.0);
            out[c] = c == 0 ? t.c_x[c0 + k] : c == 1 ? t.c_y[c0 + k] : t.c_z[c0 + k];
            out[3 + c] = Mc[0];
            #pragma unroll
            for (int d = 0; d < 3; ++d) out[6 + 3 * c + d] = Mc[1 + d];
            out[15 + 5 * c] = -5.0 * (Mc[4] - tr);
            out[16 + 5 * c] = -5.0 * (Mc[5] - tr);
            #pragma unroll
            for (int d = 0; d < 3; ++d) out[17 + 5 * c + d] = -5.0 * Mc[7 + d];
        }
        __syncwarp();
        for (int q = 0; q < m; ++q)
            if (lane < kMom3D) t.mom[(size_t)(c0 + q) * kMom3D + lane] = s_out[w][q][lane];
        __syncwarp();
    }
}

// Per-warp staging: records of far cells, or 32 sources of near leaves, or
// the candidates tested target by target.
struct Src64 {
    double2 xy[32], zax[32], ayz[32];
};
struct Src32 {
    float4 p[32], a[32];
};
struct Open3D {
    double2 xy[32];
    double2 zr[32];                   // z, (s size)^2
    uint2 m[32];                      // masks
};
template <bool F32>
union alignas(16) Stage3D {
    unsigned char rec[kStageM][F32 ? kRec32Bytes : kRec64Bytes];
    Src64 s64;
    Src32 s32;
    Open3D open;
};
// W warps. A step adds at most 32 W entries to the far and near lists, which
// are worked off above half of their capacity.
template <bool F32, int W>
struct alignas(16) Block3D {
    static constexpr int kList = 64 * W;
    Stage3D<F32> st[W];
    uint4 stack[kStack3D];            // (children - 1) << 29 | first child, masks
    uint4 far[kList], near[kList];    // cell, masks
    int start[W][32];                 // flat start of a near leaf's sources in the warp's batch
    int count[W][3];                  // far cells, near leaves and walk entries a warp adds
};

// Far cells w, w + W, ... of the list. Records are copied one pair of cells
// ahead of their use.
template <bool F32, int W>
__device__ __forceinline__ void far_flush(Block3D<F32, W>& s, const Tree3D& t, int nf, int w, Targets& tg) {
    const int lane = threadIdx.x & 31;
    constexpr size_t kBytes = F32 ? kRec32Bytes : kRec64Bytes;
    constexpr int kChunks = (int)kBytes / 16;
    const char* base = F32 ? (const char*)t.rec32 : (const char*)t.mom;
    Stage3D<F32>& st = s.st[w];
    const int cnt = nf > w ? (nf - w + W - 1) / W : 0;
    auto fetch = [&](int i) {
        // lanes 0-15 the first cell's chunks, 16-31 the second's (at most 16 each)
        static_assert(kChunks <= 16, "one record per half warp");
        const int k = i + (lane >> 4), c = lane & 15;
        if (k < cnt && c < kChunks)
            cp_async16(st.rec[k & (kStageM - 1)] + 16 * c, base + (size_t)s.far[w + k * W].x * kBytes + 16 * c);
        cp_async_commit();
    };
    fetch(0);
    for (int i = 0; i < cnt; i += 2) {
        cp_async_wait<0>();
        __syncwarp();   // records i, i + 1 have landed for every lane; the two before are read
        fetch(i + 2);
        #pragma unroll
        for (int k = i; k < i + 2; ++k) {
            if (k >= cnt) break;
            const unsigned char* rec = st.rec[k & (kStageM - 1)];
            const uint4 e = s.far[w + k * W];
            const bool on[2] = {((e.y >> lane) & 1u) != 0, ((e.z >> lane) & 1u) != 0};
            if (F32) {
                const double* c = reinterpret_cast<const double*>(rec);
                #pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (on[h])
                        m2p32(reinterpret_cast<const float*>(rec) + 6, xsub(tg.x[h], c[0]), xsub(tg.y[h], c[1]),
                              xsub(tg.z[h], c[2]), tg.vx[h], tg.vy[h], tg.vz[h]);
            } else {
                const double2* r = reinterpret_cast<const double2*>(rec);
                if (e.y && e.z) m2p64<0, 1>(r, on, tg);   // warp-uniform
                else if (e.y) m2p64<0, 0>(r, on, tg);
                else m2p64<1, 1>(r, on, tg);
            }
        }
    }
    cp_async_wait<0>();
    __syncwarp();
}

// Sources i0 .. i1 - 1 of the warp's staged batch, all of one near leaf, onto
// targets FIRST .. LAST; j0 is the slot of staged source 0, `act` the batch's
// mask of sources that count, sum[] the mixed form's FP32 sums of the leaf.
template <int FIRST, int LAST>
__device__ __forceinline__ void pairs64(const Src64& s, int i0, int i1, int j0, unsigned act, const bool* in,
                                        Targets& t) {
    #pragma unroll 2
    for (int i = i0; i < i1; ++i) {
        const bool live = (act >> i) & 1u;
        const double2 xy = s.xy[i], za = s.zax[i], yz = s.ayz[i];
        #pragma unroll
        for (int h = FIRST; h <= LAST; ++h) {
            const bool on = in[h] && live && j0 + i != t.slot[h];
            const double ex = t.x[h] - xy.x, ey = t.y[h] - xy.y, ez = t.z[h] - za.x;
            const double ir = rsqrt_halley(ex * ex + ey * ey + ez * ez);
            add3_if(on, ir * ir * ir, fma(yz.x, ez, -(yz.y * ey)), fma(yz.y, ex, -(za.y * ez)),
                    fma(za.y, ey, -(yz.x * ex)), t.vx[h], t.vy[h], t.vz[h]);
        }
    }
}

struct Sums32 {
    float tx[2], ty[2], tz[2];        // targets in the leaf's frame
    float sx[2], sy[2], sz[2];
};
template <int FIRST, int LAST>
__device__ __forceinline__ void pairs32(const Src32& s, int i0, int i1, int j0, unsigned act, const bool* in,
                                        const int* slot, Sums32& f) {
    for (int i = i0; i < i1; ++i) {
        if (!((act >> i) & 1u)) continue;   // warp-uniform
        const float4 sp = s.p[i], al = s.a[i];
        #pragma unroll
        for (int h = FIRST; h <= LAST; ++h) {
            const float ex = f.tx[h] - sp.x, ey = f.ty[h] - sp.y, ez = f.tz[h] - sp.z;
            const float ir = rsqrtf(__fmaf_rn(ez, ez, __fmaf_rn(ey, ey, __fmul_rn(ex, ex))));
            const float ir3 = ir * ir * ir;
            if (in[h] && j0 + i != slot[h]) {
                f.sx[h] = __fmaf_rn(__fmaf_rn(al.y, ez, -__fmul_rn(al.z, ey)), ir3, f.sx[h]);
                f.sy[h] = __fmaf_rn(__fmaf_rn(al.z, ex, -__fmul_rn(al.x, ez)), ir3, f.sy[h]);
                f.sz[h] = __fmaf_rn(__fmaf_rn(al.x, ey, -__fmul_rn(al.y, ex)), ir3, f.sz[h]);
            }
        }
    }
}

// Near leaves w, w + W, ... of the list, 32 of them at a time: their sources
// as one flat sequence, staged 32 at a time and applied leaf by leaf.
// ALL: inactive particles are sources too (TreeCell path). Mixed form: the
// target's offset from the leaf's centre is formed in FP64 and rounded once,
// the sources' offsets and alphas are FP32 copies (prep3d_f32), a leaf's sum
// is FP32 and is added to the FP64 total.
template <bool F32, bool ALL, int W>
__device__ __forceinline__ void near_flush(Block3D<F32, W>& s, const Tree3D& t, int nn, int w, Targets& tg) {
    const int lane = threadIdx.x & 31;
    Stage3D<F32>& st = s.st[w];
    int* start = s.start[w];
    for (int first = w; first < nn; first += 32 * W) {
        const int mine = first + lane * W;
        int lo = 0, sz = 0;
        if (mine < nn) {
            const int k = (int)s.near[mine].x;
            lo = t.c_lo[k];
            sz = t.c_hi[k] - lo;
        }
        int incl = sz;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        start[lane] = incl - sz;
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        int cur = -1;                   // mixed: list entry the FP32 sums belong to
        Sums32 f;
        auto flush32 = [&]() {
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (cur >= 0) {
                    tg.vx[h] += f.sx[h];
                    tg.vy[h] += f.sy[h];
                    tg.vz[h] += f.sz[h];
                }
                f.sx[h] = f.sy[h] = f.sz[h] = 0.f;
            }
        };
        if (F32) flush32();
        for (int b = 0; b < total; b += 32) {
            __syncwarp();               // start[] is written; the last batch is read
            const int q = b + lane;
            int e = 0;                  // the last entry that starts at or before q
            #pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                if (start[e + o] <= q) e += o;
            const int j = __shfl_sync(0xffffffffu, lo, e) + q - start[e];
            const bool in = q < total;
            bool live = false;
            if (in) {
                if constexpr (F32) {
                    const float4 p = t.ps32[j];
                    live = ALL || p.w != 0.f;
                    st.s32.p[lane] = p;
                    st.s32.a[lane] = t.as32[j];
                } else {
                    live = ALL || t.pact[j];
                    st.s64.xy[lane] = make_double2(t.px[j], t.py[j]);
                    st.s64.zax[lane] = make_double2(t.pz[j], t.ax[j]);
                    st.s64.ayz[lane] = make_double2(t.ay[j], t.az[j]);
                }
            }
            const unsigned act = __ballot_sync(0xffffffffu, live);   // and the staged sources are written
            const int c = min(32, total - b);
            for (int i = 0; i < c;) {   // one leaf's share of the batch at a time
                const int le = __shfl_sync(0xffffffffu, e, i), jl = __shfl_sync(0xffffffffu, j, i) - i;
                const unsigned same = __ballot_sync(0xffffffffu, in && e == le);
                const int i1 = 32 - __clz(same);
                const uint4 en = s.near[first + le * W];
                const bool on[2] = {((en.y >> lane) & 1u) != 0, ((en.z >> lane) & 1u) != 0};
                if constexpr (F32) {
                    if (le != cur) {
                        flush32();
                        cur = le;
                        const double cx = t.c_x[en.x], cy = t.c_y[en.x], cz = t.c_z[en.x];
                        #pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            f.tx[h] = (float)(tg.x[h] - cx);
                            f.ty[h] = (float)(tg.y[h] - cy);
                            f.tz[h] = (float)(tg.z[h] - cz);
                        }
                    }
                    if (en.y && en.z) pairs32<0, 1>(st.s32, i, i1, jl, act, on, tg.slot, f);
                    else if (en.y) pairs32<0, 0>(st.s32, i, i1, jl, act, on, tg.slot, f);
                    else pairs32<1, 1>(st.s32, i, i1, jl, act, on, tg.slot, f);
                } else {
                    if (en.y && en.z) pairs64<0, 1>(st.s64, i, i1, jl, act, on, tg);
                    else if (en.y) pairs64<0, 0>(st.s64, i, i1, jl, act, on, tg);
                    else pairs64<1, 1>(st.s64, i, i1, jl, act, on, tg);
                }
                i = i1;
            }
        }
        if (F32) flush32();
        __syncwarp();
    }
}

__device__ __forceinline__ double warp_min(double v) {
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// One block of W warps per 64 targets. The walk's stack holds non-leaf cells
// as (first child, number of children); a step pops up to 4 W entries, warp w
// classifies the children of four of them, and the block appends the results
// in warp and lane order. A step that pops p entries adds at most 7 p to the
// stack, so near its top only one is popped: depth first, that adds at most 7
// for each of the tree's kMaxLevels3D levels, which the rest of it holds.
template <bool F32, bool ALL, int W>
__global__ void __launch_bounds__(32 * W, W > 4 ? 1 : F32 ? 5 : 4)
eval3d_kernel(Tree3D t, const uint8_t* __restrict__ target, double support, double* __restrict__ u,
              double* __restrict__ v, double* __restrict__ w, double uinf, double vinf, double winf, unsigned* err) {
    extern __shared__ __align__(16) unsigned char sm3[];
    Block3D<F32, W>& s = *reinterpret_cast<Block3D<F32, W>*>(sm3);
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (block_fatal(err)) return;
    Targets tg;
    bool has[2], tgt[2];
    unsigned full[2];
    #pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int slot = blockIdx.x * 64 + 32 * h + lane;
        has[h] = slot < t.n;
        tgt[h] = has[h] && (target == nullptr || target[t.perm[slot]] != 0);
        tg.slot[h] = slot;
        tg.x[h] = has[h] ? t.px[slot] : 0.0;
        tg.y[h] = has[h] ? t.py[slot] : 0.0;
        tg.z[h] = has[h] ? t.pz[slot] : 0.0;
        tg.vx[h] = tg.vy[h] = tg.vz[h] = 0.0;
        full[h] = __ballot_sync(0xffffffffu, tgt[h]);
    }
    const unsigned below = (1u << lane) - 1u;
    auto walk_entry = [](unsigned cm, int c0, unsigned ma, unsigned mb) {
        return make_uint4((unsigned)(__popc(cm) - 1) << 29 | (unsigned)c0, ma, mb, 0u);
    };
    int top = 0, nf = 0, nn = 0;   // the same in every thread
    // the level-1 cells are walked through but never evaluated themselves
    if (full[0] | full[1]) {
        const int r0 = t.c_child0[0], nr = __popc(t.c_chmask[0]);
        unsigned cm = 0;
        if (lane < nr) cm = t.c_chmask[r0 + lane];
        const unsigned push = __ballot_sync(0xffffffffu, cm != 0);
        if (cm && wib == 0) s.stack[__popc(push & below)] = walk_entry(cm, t.c_child0[r0 + lane], full[0], full[1]);
        top = __popc(push);
    }
    auto box = [&](const double* p, double& lo, double& hi) {
        lo = warp_min(fmin(tgt[0] ? p[0] : HUGE_VAL, tgt[1] ? p[1] : HUGE_VAL));
        hi = warp_max(fmax(tgt[0] ? p[0] : -HUGE_VAL, tgt[1] ? p[1] : -HUGE_VAL));
    };
    double bx0, bx1, by0, by1, bz0, bz1;
    box(tg.x, bx0, bx1);
    box(tg.y, by0, by1);
    box(tg.z, bz0, bz1);
    // least and largest |fl(p - c)| over the box's axis
    auto span = [](double c, double lo, double hi, double& mn, double& mx) {
        const double a = xsub(lo, c), b = xsub(hi, c);
        mn = fmax(0.0, fmax(a, -b));
        mx = fmax(-a, b);
    };
    auto dist2 = [](double x, double y, double z) { return xadd(xadd(xmul(x, x), xmul(y, y)), xmul(z, z)); };
    while (top > 0) {
        const int room = kStack3D - top;
        if (room < 7) {
            if (threadIdx.x == 0) set_err(err, ERR_QUEUE);
            break;   // block-uniform
        }
        const int npop = min(min(4 * W, top), room >= 7 * 4 * W + 7 * kMaxLevels3D ? 4 * W : 1);
        top -= npop;
        __syncthreads();   // the entries popped are written; counts of the last step are read
        const int pe = 4 * wib + (lane >> 3), r = lane & 7;
        unsigned cm = 0, fa = 0, fb = 0, ra = 0, rb = 0;   // far masks, near masks of the lane's candidate
        int k = 0, c0 = 0;
        bool cand = false;
        if (pe < npop) {
            const uint4 e = s.stack[top + pe];
            cand = r <= (int)(e.x >> 29);
            k = (int)(e.x & 0x1fffffffu) + r;
            ra = e.y;
            rb = e.z;
        }
        bool open = false;
        double cx = 0.0, cy = 0.0, cz = 0.0, rc2 = 0.0;
        if (cand) {
            cand = t.c_active[k] != 0;
            cx = t.c_x[k];
            cy = t.c_y[k];
            cz = t.c_z[k];
            cm = t.c_chmask[k];
            c0 = t.c_child0[k];
            const double rc = xmul(t.c_size[k], support);
            rc2 = xmul(rc, rc);
            double x0, x1, y0, y1, z0, z1;
            span(cx, bx0, bx1, x0, x1);
            span(cy, by0, by1, y0, y1);
            span(cz, bz0, bz1, z0, z1);
            if (dist2(x0, y0, z0) > rc2) {
                fa = ra;
                fb = rb;
                ra = rb = 0;
            } else {
                open = cand && dist2(x1, y1, z1) > rc2;
            }
        }
        if (!cand) fa = fb = ra = rb = 0;
        const unsigned b_open = __ballot_sync(0xffffffffu, open);
        if (b_open) {
            Open3D& o = s.st[wib].open;
            if (open) {
                const int i = __popc(b_open & below);
                o.xy[i] = make_double2(cx, cy);
                o.zr[i] = make_double2(cz, rc2);
            }
            __syncwarp();
            const int nopen = __popc(b_open);
            #pragma unroll 2
            for (int i = 0; i < nopen; ++i) {
                const double2 xy = o.xy[i], zr = o.zr[i];
                const unsigned ma = __ballot_sync(
                    0xffffffffu, dist2(xsub(tg.x[0], xy.x), xsub(tg.y[0], xy.y), xsub(tg.z[0], zr.x)) > zr.y);
                const unsigned mb = __ballot_sync(
                    0xffffffffu, dist2(xsub(tg.x[1], xy.x), xsub(tg.y[1], xy.y), xsub(tg.z[1], zr.x)) > zr.y);
                if (lane == i) o.m[i] = make_uint2(ma, mb);
            }
            __syncwarp();
            if (open) {
                const uint2 m = o.m[__popc(b_open & below)];
                fa = ra & m.x;
                fb = rb & m.y;
                ra &= ~m.x;
                rb &= ~m.y;
            }
        }
        const bool p_far = (fa | fb) != 0, p_near = (ra | rb) != 0 && cm == 0, p_down = (ra | rb) != 0 && cm != 0;
        const unsigned b_far = __ballot_sync(0xffffffffu, p_far);
        const unsigned b_near = __ballot_sync(0xffffffffu, p_near);
        const unsigned b_down = __ballot_sync(0xffffffffu, p_down);
        if (lane == 0) {
            s.count[wib][0] = __popc(b_far);
            s.count[wib][1] = __popc(b_near);
            s.count[wib][2] = __popc(b_down);
        }
        __syncthreads();   // the popped entries are read too
        int at[3] = {nf, nn, top};
        #pragma unroll
        for (int i = 0; i < W; ++i) {
            #pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int q = s.count[i][c];
                if (i < wib) at[c] += q;
                (c == 0 ? nf : c == 1 ? nn : top) += q;
            }
        }
        if (p_far) s.far[at[0] + __popc(b_far & below)] = make_uint4((unsigned)k, fa, fb, 0u);
        if (p_near) s.near[at[1] + __popc(b_near & below)] = make_uint4((unsigned)k, ra, rb, 0u);
        if (p_down) s.stack[at[2] + __popc(b_down & below)] = walk_entry(cm, c0, ra, rb);
        constexpr int kFull = Block3D<F32, W>::kList / 2;
        if (nf > kFull || nn > kFull) {
            __syncthreads();
            if (nf > kFull) {
                far_flush<F32, W>(s, t, nf, wib, tg);
                nf = 0;
            }
            if (nn > kFull) {
                near_flush<F32, ALL, W>(s, t, nn, wib, tg);
                nn = 0;
            }
            __syncthreads();
        }
    }
    __syncthreads();
    far_flush<F32, W>(s, t, nf, wib, tg);
    near_flush<F32, ALL, W>(s, t, nn, wib, tg);
    // the warps' sums, added in warp order: warp 0 target 0, warp 1 target 1 of every lane
    __syncthreads();
    double* sum = reinterpret_cast<double*>(sm3);   // [W][6][32]
    static_assert(sizeof(Block3D<F32, W>) >= W * 6 * 32 * sizeof(double), "the sums reuse the lists");
    #pragma unroll
    for (int h = 0; h < 2; ++h) {
        sum[(wib * 6 + 3 * h + 0) * 32 + lane] = tg.vx[h];
        sum[(wib * 6 + 3 * h + 1) * 32 + lane] = tg.vy[h];
        sum[(wib * 6 + 3 * h + 2) * 32 + lane] = tg.vz[h];
    }
    __syncthreads();
    if (wib > 1) return;
    const bool hs = wib ? has[1] : has[0], tt = wib ? tgt[1] : tgt[0];
    if (!hs) return;
    double a[3] = {0.0, 0.0, 0.0};
    #pragma unroll
    for (int i = 0; i < W; ++i)
        #pragma unroll
        for (int c = 0; c < 3; ++c) a[c] += sum[(i * 6 + 3 * wib + c) * 32 + lane];
    const uint32_t i = t.perm[blockIdx.x * 64 + 32 * wib + lane];
    u[i] = tt ? a[0] + uinf : 0.0;
    v[i] = tt ? a[1] + vinf : 0.0;
    w[i] = tt ? a[2] + winf : 0.0;
}

}  // namespace

cudaError_t prep3d(const Tree3D& t, bool mixed, unsigned* err, cudaStream_t st, int* launches) {
    if (mixed) prep3d_f32_kernel<<<148 * 8, 256, 0, st>>>(t, err);
    else pack3d_f64_kernel<<<148 * 8, 32 * kPackWarps, 0, st>>>(t, err);
    *launches += 1;
    return cudaGetLastError();
}

template <bool F32, bool ALL, int W>
static cudaError_t launch_eval3d_w(const Tree3D& t, const uint8_t* target, double support, double* u, double* v,
                                   double* w, double uinf, double vinf, double winf, unsigned* err, cudaStream_t st) {
    constexpr int smem = (int)sizeof(Block3D<F32, W>);
    if (smem > 48 * 1024) {
        const cudaError_t e =
            cudaFuncSetAttribute(eval3d_kernel<F32, ALL, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
    }
    eval3d_kernel<F32, ALL, W><<<ceil_div(t.n, 64), 32 * W, smem, st>>>(t, target, support, u, v, w, uinf, vinf, winf,
                                                                        err);
    return cudaGetLastError();
}

cudaError_t eval3d(const Tree3D& t, bool mixed, bool all_src, const uint8_t* target, double support, double* u,
                   double* v, double* w, double uinf, double vinf, double winf, unsigned* err, cudaStream_t st,
                   int* launches) {
    // Warps per block: with at most two blocks per SM the work of one block is
    // the kernel's time, so eight warps share it; with more blocks than that
    // four, whose barriers and uneven shares cost less. A whole call with eight
    // warps against four, FP64 (mixed): 5,202 particles 228 us against 254 (244,
    // 288), 14,200 313 and 326 (346, 354), 19,500, where the line lies, 375 and 377
    // (418, 413), 27,872 424 and 410 (490, 434), 222,688 2,574 and 2,161 (3,239,
    // 2,238).
    const bool wide = ceil_div(t.n, 64) <= 2 * 148;
#define VPM_LAUNCH(F, A)                                                                              \
    (wide ? launch_eval3d_w<F, A, 8>(t, target, support, u, v, w, uinf, vinf, winf, err, st)          \
          : launch_eval3d_w<F, A, 4>(t, target, support, u, v, w, uinf, vinf, winf, err, st))
    *launches += 1;
    if (mixed) return all_src ? VPM_LAUNCH(true, true) : VPM_LAUNCH(true, false);
    return all_src ? VPM_LAUNCH(false, true) : VPM_LAUNCH(false, false);
#undef VPM_LAUNCH
}

}  // namespace vpm
