// fia_advect32.cu -- the chosen form of the flux pass: FP32 arithmetic in local cell
// coordinates, double-float psi, compensated face and cell sums.
//
// Same kernels as fia_advect.cu (psi column scan, unique-vertex backtrace, unique-face
// clip + quadrature + WENO6, deterministic gather), with these differences:
//  * all geometry is in cell units relative to an integer anchor (fia_local.cuh);
//  * psi is stored as (hi, lo) float pairs in the reference's units (density x length):
//    the WENO6 weights are not scale invariant (alpha = C / (1e-6 + beta)^2), so psi must
//    carry the same scale as in the reference for the same interpolant;
//  * a face interpolates psi - Psi0(f), Psi0(f) = the psi node at the face's anchor, and
//    stores (Ft, Ny): the compensated flux of psi - Psi0 plus the density terms, and the
//    sum of the pieces' scaled y-normals;
//  * the gather forms, per cell c with base node Psi_c,
//        rho' = sum_f s_f [ Ft(f) + (Psi0(f) - Psi_c) Ny(f) ],
//    which equals sum_f s_f F(f) - Psi_c sum_f s_f Ny(f); the last sum is the y-component
//    of the vector area of the closed surface of the backtraced cell, zero in exact
//    arithmetic, and is dropped so that no O(psi) term survives in FP32.
#include "fia_advect.cuh"
#include "fia_local.cuh"
#include "fia_clip32.cuh"
#include "fia_weno_rec.cuh"
#include "fia_trace.cuh"

#include <algorithm>
#include <climits>

namespace fia {

namespace {

inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// ---------------------------------------------------------------------------------
// psi as hi/lo pairs: the cells' increments, then their running sums along y
// ---------------------------------------------------------------------------------
// The increment of cell (i, c, k) goes to psi row c + 1 as a (sum, compensation) pair.  A thread
// takes kPsiRun cells of a column.  WENO6: cell c spans [c + oy - 1/2, c + oy + 1/2], so its points
// lie below node c in the first half and above it in the second, at offsets that no cell changes:
// the coefficients are formed once a block, and the stencil data of the second half serve the first
// half of the next cell too.  The three psi of a density step at 128^3 took 360 us as one thread
// a column, which evaluated every point from its samples and summed as it went (16384 threads, each a
// chain of 128 cells): 78 us now, 30 of them these increments (bound by FP32 issue).  Runs of 8 cells
// measure the same there, and 3% of a whole step more at 16^3.
constexpr int kPsiRun = 4, kPsiThreads = 128;
template <int MODE>
__global__ void __launch_bounds__(kPsiThreads) k_psi_inc32(PassDesc d, const float* __restrict__ a,
                                                           float2* __restrict__ psi) {
    __shared__ WenoCoef<float> coef[2 * kMaxGauss];
    const float hf = d.hf, oy = d.A.oyf;
    if constexpr (MODE == PSI_WENO6) {
        if (threadIdx.x < 2 * d.k) {
            const int half = (int)threadIdx.x >= d.k, q = threadIdx.x - half * d.k;
            const float y = ((oy - 0.5f) + 0.5f * float(half)) + 0.25f * (1.0f + d.gxf[q]);
            int by;
            float sy, t[6];
            locate(0, y, oy, by, sy);
#pragma unroll
            for (int i = 0; i < 6; ++i) t[i] = sy + float(2 - i);
            coef[threadIdx.x] = weno_coef(t);
        }
        __syncthreads();
    }
    const int Mx = d.A.Mx, My = d.A.My, Mz = d.A.Mz;
    const int runs = (My + kPsiRun - 1) / kPsiRun;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)Mx * runs * Mz) return;
    const int k = (int)(id % Mz);
    const long long t = id / Mz;
    const int j0 = (int)(t % runs) * kPsiRun, i = (int)(t / runs);
    const int j1 = min(j0 + kPsiRun, My);
    if constexpr (MODE == PSI_WENO6) {
        const float* col = a + idx3(d.A, i, 0, k);
        float f[6];
#pragma unroll
        for (int m = 0; m < 6; ++m) f[m] = __ldg(col + (long long)clampi(j0 - 3 + m, My - 1) * Mz);
        Weno6Data w = weno6_data(f);
#pragma unroll 1
        for (int j = j0; j < j1; ++j) {
            Kahan inc;
#pragma unroll 1
            for (int q = 0; q < d.k; ++q) inc.add(weno6_at(w, coef[q]) * (0.5f * hf) * d.gwf[q]);
#pragma unroll
            for (int m = 0; m < 5; ++m) f[m] = f[m + 1];
            f[5] = __ldg(col + (long long)clampi(j + 3, My - 1) * Mz);
            w = weno6_data(f);
#pragma unroll 1
            for (int q = 0; q < d.k; ++q) inc.add(weno6_at(w, coef[d.k + q]) * (0.5f * hf) * d.gwf[q]);
            psi[idx3(d.P, i, j + 1, k)] = make_float2(inc.s, inc.c);
        }
    } else {
        const PlainLoad L{a};
        const float q0[3] = {d.A.oxf, 0.25f + oy - 0.5f, d.A.ozf};
        const float q1[3] = {d.A.oxf, 0.75f + oy - 0.5f, d.A.ozf};
        for (int j = j0; j < j1; ++j) {
            const int anc[3] = {i, j, k};
            Kahan inc;
            inc.add(lin3d_loc(L, d.A, anc, q0) * (0.5f * hf));
            inc.add(lin3d_loc(L, d.A, anc, q1) * (0.5f * hf));
            psi[idx3(d.P, i, j + 1, k)] = make_float2(inc.s, inc.c);
        }
    }
}
// The running sums, one thread per (x, z) column; the cells' increments are loaded kScanAhead at a
// time (PLAIN: formed from the field).
constexpr int kScanAhead = 16, kScanThreads = 64;
template <bool PLAIN>
__global__ void __launch_bounds__(kScanThreads) k_psi_scan32(PassDesc d, const float* __restrict__ a,
                                                             float2* __restrict__ psi) {
    const int My = d.A.My, Mz = d.A.Mz;
    const long long col = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= (long long)d.A.Mx * Mz) return;
    const int i = (int)(col / Mz), k = (int)(col % Mz);
    float2* P = psi + idx3(d.P, i, 0, k);
    const float* A = a + idx3(d.A, i, 0, k);
    float hi = 0.f, lo = 0.f;
    *P = make_float2(0.f, 0.f);
    auto add = [&](int j, float2 v) {
        Kahan inc;
        if (PLAIN) inc.add(v.x * d.hf);
        else inc = Kahan{v.x, v.y};
        // (hi, lo) += inc
        float s, e;
        two_sum(hi, inc.s, s, e);
        e += lo + inc.c;
        two_sum(s, e, hi, lo);
        P[(long long)j * Mz] = make_float2(hi, lo);
    };
    auto at = [&](int j) {
        return PLAIN ? make_float2(__ldg(A + (long long)(j - 1) * Mz), 0.f) : P[(long long)j * Mz];
    };
    int j = 1;
    for (; j + kScanAhead - 1 <= My; j += kScanAhead) {
        float2 v[kScanAhead];
#pragma unroll
        for (int m = 0; m < kScanAhead; ++m) v[m] = at(j + m);
#pragma unroll
        for (int m = 0; m < kScanAhead; ++m) add(j + m, v[m]);
    }
    for (; j <= My; ++j) add(j, at(j));
}
void psi32(const PassDesc& d, const float* a, float2* psi, cudaStream_t s) {
    const long long cols = (long long)d.A.Mx * d.A.Mz;
    const unsigned inc = nblk(cols * ((d.A.My + kPsiRun - 1) / kPsiRun), kPsiThreads);
    if (d.psi_mode == PSI_WENO6) k_psi_inc32<PSI_WENO6><<<inc, kPsiThreads, 0, s>>>(d, a, psi);
    else if (d.psi_mode == PSI_LINEAR) k_psi_inc32<PSI_LINEAR><<<inc, kPsiThreads, 0, s>>>(d, a, psi);
    if (d.psi_mode == PSI_PLAIN) k_psi_scan32<true><<<nblk(cols, kScanThreads), kScanThreads, 0, s>>>(d, a, psi);
    else k_psi_scan32<false><<<nblk(cols, kScanThreads), kScanThreads, 0, s>>>(d, a, psi);
}

// ---------------------------------------------------------------------------------
// backtrace: displacement in cells of every unique vertex, clamped to the domain (one thread a
// vertex: linear interpolation)
// ---------------------------------------------------------------------------------
__global__ void k_backtrace32(PassDesc d, const float* __restrict__ u, const float* __restrict__ v,
                              const float* __restrict__ w, NodeField fu, NodeField fv, NodeField fw,
                              float* __restrict__ disp) {
    const int Lx = d.A.Mx + 1, Ly = d.A.My + 1, Lz = d.A.Mz + 1;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)Lx * Ly * Lz) return;
    const int k = (int)(id % Lz);
    const int j = (int)((id / Lz) % Ly);
    const int i = (int)(id / ((long long)Lz * Ly));
    const int anc[3] = {i, j, k};
    float q[3] = {0.f, 0.f, 0.f};
    if (d.comp >= 0) q[d.comp] = -0.5f;
    float dx[3] = {0.f, 0.f, 0.f};
    bool pinned = false;
    if (d.comp >= 0) {
        const int vi = anc[d.comp];
        pinned = (vi <= 1 || vi >= d.N[d.comp]);
    }
    if (!pinned) {
        const float s = d.dthf;   // dt/h converts the velocity to cells per step
        dx[0] = -interp_loc(d.interp, PlainLoad{u}, fu, anc, q) * s;
        dx[1] = -interp_loc(d.interp, PlainLoad{v}, fv, anc, q) * s;
        dx[2] = -interp_loc(d.interp, PlainLoad{w}, fw, anc, q) * s;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float e = (c == d.comp) ? 0.5f : 0.f;
        const float rest = float(anc[c]) + q[c];          // exact (small integers and halves)
        const float lo = -e, hi = float(d.N[c]) + e;
        if (rest + dx[c] < lo) dx[c] = lo - rest;
        if (rest + dx[c] > hi) dx[c] = hi - rest;
    }
    disp[3 * id + 0] = dx[0]; disp[3 * id + 1] = dx[1]; disp[3 * id + 2] = dx[2];
}

// The same with WENO6, a tile of vertices and one velocity component a block (fia_trace.cuh).
template <int N>
__global__ void __launch_bounds__(kTraceThreads) k_trace32(PassDesc d, const float* __restrict__ u,
                                                           const float* __restrict__ v, const float* __restrict__ w,
                                                           NodeField fu, NodeField fv, NodeField fw,
                                                           float* __restrict__ disp, TraceTiles tiles) {
    extern __shared__ float trace_sm[];
    const int c = blockIdx.y;
    const float* a = c == 0 ? u : (c == 1 ? v : w);
    const NodeField F = c == 0 ? fu : (c == 1 ? fv : fw);
    const float off[3] = {F.oxf, F.oyf, F.ozf};
    const int L[3] = {d.A.Mx + 1, d.A.My + 1, d.A.Mz + 1};
    const float q[3] = {d.comp == 0 ? -0.5f : 0.f, d.comp == 1 ? -0.5f : 0.f, d.comp == 2 ? -0.5f : 0.f};
    const float qc = c == d.comp ? -0.5f : 0.f, e = c == d.comp ? 0.5f : 0.f;
    const float lo = -e, hi = float(c == 0 ? d.N[0] : (c == 1 ? d.N[1] : d.N[2])) + e, s = d.dthf;
    const int Np = d.comp == 0 ? d.N[0] : (d.comp == 1 ? d.N[1] : d.N[2]);
    trace_tile<N, TraceCoef32>(a, F, off, L, q, tiles, trace_sm, [&](int i, int j, int k, float val) {
        const int vi = d.comp == 0 ? i : (d.comp == 1 ? j : k);
        float dx = d.comp >= 0 && (vi <= 1 || vi >= Np) ? 0.f : -val * s;
        const float rest = float(c == 0 ? i : (c == 1 ? j : k)) + qc;   // exact (small integers and halves)
        if (rest + dx < lo) dx = lo - rest;
        if (rest + dx > hi) dx = hi - rest;
        disp[3 * (((long long)i * L[1] + j) * L[2] + k) + c] = dx;
    });
}
// Tiles of 8 x 8 vertices, of 4 x 4 (a quarter more evaluations for a density vertex) where those
// would leave SMs without a block.  Whole density steps: 128^3 4883 us with 8 x 8, 4935 with 4 x 4;
// 16^3 323 and 314.
void backtrace32(const PassDesc& d, const VelocityFields& vel, float* disp, cudaStream_t s) {
    const int L[3] = {d.A.Mx + 1, d.A.My + 1, d.A.Mz + 1};
    const float *u = (const float*)vel.u, *v = (const float*)vel.v, *w = (const float*)vel.w;
    if (d.interp != INTERP_WENO6) {
        const long long nv = (long long)L[0] * L[1] * L[2];
        k_backtrace32<<<nblk(nv, 128), 128, 0, s>>>(d, u, v, w, vel.fu, vel.fv, vel.fw, disp);
        return;
    }
    const TraceTiles t8 = trace_tiles(L, 8, 32), t4 = trace_tiles(L, 4, 32);
    if (3 * trace_blocks(L, 8, t8) >= 152 * 2) {
        const dim3 g(trace_blocks(L, 8, t8), 3);
        k_trace32<8><<<g, kTraceThreads, trace_smem(8, t8, 4), s>>>(d, u, v, w, vel.fu, vel.fv, vel.fw, disp, t8);
    } else {
        const dim3 g(trace_blocks(L, 4, t4), 3);
        k_trace32<4><<<g, kTraceThreads, trace_smem(4, t4, 4), s>>>(d, u, v, w, vel.fu, vel.fv, vel.fw, disp, t4);
    }
}

// Second trace of the flux MacCormack scheme: from the backtraced position (rest + disp),
// disp2 = disp + dt/h u(rest + disp), the pin rule and clamp of k_backtrace32
// (calc_backtraced_face_3D.cpp:9-160, time direction "backward").
__global__ void k_forward32(PassDesc d, const float* __restrict__ u, const float* __restrict__ v,
                            const float* __restrict__ w, NodeField fu, NodeField fv, NodeField fw,
                            const float* __restrict__ disp, float* __restrict__ disp2) {
    const int Lx = d.A.Mx + 1, Ly = d.A.My + 1, Lz = d.A.Mz + 1;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)Lx * Ly * Lz) return;
    const int k = (int)(id % Lz);
    const int j = (int)((id / Lz) % Ly);
    const int i = (int)(id / ((long long)Lz * Ly));
    const int anc[3] = {i, j, k};
    float q0[3] = {0.f, 0.f, 0.f};
    if (d.comp >= 0) q0[d.comp] = -0.5f;
    float dx[3] = {disp[3 * id], disp[3 * id + 1], disp[3 * id + 2]};
    bool pinned = false;
    if (d.comp >= 0) {
        const int vi = anc[d.comp];
        pinned = (vi <= 1 || vi >= d.N[d.comp]);
    }
    if (!pinned) {
        const float q[3] = {q0[0] + dx[0], q0[1] + dx[1], q0[2] + dx[2]};
        const float s = d.dthf;
        const float v0 = interp_loc(d.interp, PlainLoad{u}, fu, anc, q);
        const float v1 = interp_loc(d.interp, PlainLoad{v}, fv, anc, q);
        const float v2 = interp_loc(d.interp, PlainLoad{w}, fw, anc, q);
        dx[0] += v0 * s; dx[1] += v1 * s; dx[2] += v2 * s;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float e = (c == d.comp) ? 0.5f : 0.f;
        const float rest = float(anc[c]) + q0[c];
        const float lo = -e, hi = float(d.N[c]) + e;
        if (rest + dx[c] < lo) dx[c] = lo - rest;
        if (rest + dx[c] > hi) dx[c] = hi - rest;
    }
    disp2[3 * id + 0] = dx[0]; disp2[3 * id + 1] = dx[1]; disp2[3 * id + 2] = dx[2];
}

// ---------------------------------------------------------------------------------
// faces
// ---------------------------------------------------------------------------------
// One record per node row and stencil base (fia_weno_rec.cuh): of the advected field, and of psi
// (WenoNewton; the pairs' differences, free of psi's magnitude).  One thread per record, coalesced
// in both directions: bound by the 32 or 36 bytes written.
template <bool PSI>
__global__ void k_records_newton(NodeField F, const void* __restrict__ field, float4* __restrict__ rec) {
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= weno_rec_count(F)) return;
    const long long row = id / (F.Mz + 1);
    const int b = (int)(id - row * (F.Mz + 1)) - 1;
    float f[6], lo[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const long long n = row * F.Mz + clampi(b - 2 + i, F.Mz - 1);
        if (PSI) {
            const float2 v = __ldg(static_cast<const float2*>(field) + n);
            f[i] = v.x; lo[i] = v.y;
        } else {
            f[i] = __ldg(static_cast<const float*>(field) + n);
        }
    }
    float D[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) D[i] = PSI ? (f[i + 1] - f[i]) + (lo[i + 1] - lo[i]) : f[i + 1] - f[i];
    const WenoRec<float> r = weno_record(f[2], D[0], D[1], D[2], D[3], D[4]);
    rec[2 * id] = make_float4(r.f, r.d, r.s1, r.s2);
    rec[2 * id + 1] = make_float4(r.t0, r.t2, r.q0, r.q2);
}
__global__ void k_records_samples(NodeField F, const float* __restrict__ field, float4* __restrict__ rec,
                                  float* __restrict__ rec2) {
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= weno_rec_count(F)) return;
    const long long row = id / (F.Mz + 1);
    const int b = (int)(id - row * (F.Mz + 1)) - 1;
    float f[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) f[i] = __ldg(field + row * F.Mz + clampi(b - 2 + i, F.Mz - 1));
    const Weno6Data w = weno6_data(f);
    rec[2 * id] = make_float4(f[0], f[1], f[2], f[3]);
    rec[2 * id + 1] = make_float4(f[4], f[5], w.r0, w.r1);
    rec2[id] = w.r2;
}

// The y-interval below a piece's centroid (polygon_3D.cpp:275-286): the y-face ylo = fl + oy and
// the fraction f of the cell up to the centroid.  The density points are k on [ylo, cy] when f <
// 1/2, else k on each of [ylo, ylo + 1/2] and [ylo + 1/2, cy].
struct YSpan {
    float ylo, f;
    int fl;
};
__device__ __forceinline__ YSpan y_span(const PassDesc& d, float cy) {
    const float oy = (d.comp == 1) ? -0.5f : 0.f;
    const float r = snap_int(cy - oy);
    const float fl = floorf(r);
    return YSpan{fl + oy, r - fl, (int)fl};
}

constexpr int kQuadThreads = 128;

// The WENO6 quadrature of one piece (polygon_3D.cpp:257-487); returns the number of 1D WENO6
// evaluations.  The advected field's nodes sit half a cell from the y-faces, so the points of
// one half share their six y-rows, the points of the other half the rows one further up.
//
// Density: bound by the L1 data path (72% busy) and issue (67%; 16 warps per SM by registers): a
// piece reads 42 + 6 records of 32 bytes, and the lanes of a warp spread over several cells.  One
// launch on the main pass at 128^3 (18.6M pieces): 4.99 ms evaluating every 1D interpolant from its
// samples, 2.12 ms now; a density step's launches at 256^3: 44.5 -> 21.0 ms.  Measured beside it, with
// 2.58 and 21.3 ms at that time:
// five CTAs per SM 2.88 against 2.58 ms a step (spills), three 2.84; the records as two planes of
// 16 bytes 2.50 (but 21.8 against 21.3 ms at 256^3); the pieces of a warp's faces interleaved
// in the store 2.67, with planes 2.48 and 21.7.
// Velocity: by its registers and FP32 issue (psi from its samples, coefficients of 12 words); the
// launches of a velocity step on 120 x 161 x 77 cells: 11.95 -> 7.47 ms.  Two points of a half at a
// time 8.13, three 8.6 (spills), three CTAs per SM 8.3.
template <class W>
__device__ __forceinline__ int piece_quad32(const PassDesc& d, const int* anc, float cx, float cy, float cz, float ny,
                                            const typename W::Records& ar, const float4* __restrict__ prec,
                                            const PsiLoad& pl, Kahan& F, float* zs) {
    const float nyh = ny * d.invhf;   // psi carries a length; the face terms are per cell volume
    int bx, bz;
    float sx, sz;
    locate(anc[0], cx, d.A.oxf, bx, sx);     // psi has the field's x and z offsets
    locate(anc[2], cz, d.A.ozf, bz, sz);
    const typename W::Coef kz = W::coef(sz);
    if (!d.use_integral) {
        // psi at the centroid; on an unmoved y-face (the zero-velocity pass) the centroid lies
        // on a psi node row
        int by;
        float sy;
        locate(anc[1], cy, d.P.oyf, by, sy);
        if (sy == 0.f) {
            F.add(psi_noderow<W>(W::psi_rows(prec, pl, d.P.Mz, bz), d.P, bx, by, kz, W::coef(sx)) * nyh);
            return 7;
        }
        const float q[3] = {cx, cy, cz};
        F.add(weno6_3d_loc(pl, d.P, anc, q) * nyh);
        return 43;
    }
    const YSpan Y = y_span(d, cy);
    const bool two = !(Y.f < 0.5f);
    const int jlo = anc[1] + Y.fl;             // the y-face below the centroid: psi row jlo
    rec_zpass<W, kQuadThreads>(ar, d.A, bx, clampi(bz + 1, d.A.Mz), jlo - 1, kz, zs);
    const typename W::Coef kx = W::coef(sx);
    const int k = d.k;
#pragma unroll 1
    for (int half = 0; half < (two ? 2 : 1); ++half) {
        const float lo = half ? Y.ylo + 0.5f : Y.ylo;
        const float hl = half ? (cy - lo) * 0.5f : (two ? 0.25f : (cy - Y.ylo) * 0.5f);
        const float wf = half ? ny * (Y.f - 0.5f) : (two ? ny * 0.5f : ny * Y.f);
        const float base = float(Y.fl - 1 + half);   // the half's third row, relative to the anchor
#pragma unroll 1
        for (int q0 = 0; q0 < k; q0 += W::kGroup) {
            const int n = min(W::kGroup, k - q0);
            typename W::Coef ky[W::kGroup];
#pragma unroll
            for (int q = 0; q < W::kGroup; ++q) {
                const float y = hl * d.gxf[q < n ? q0 + q : q0] + hl + lo;
                ky[q] = W::coef((y - d.A.oyf) - base);
            }
            float v[W::kGroup];
            rec_yx<W, kQuadThreads>(zs, half, ky, n, kx, v);
#pragma unroll
            for (int q = 0; q < W::kGroup; ++q)
                if (q < n) F.add(v[q] * (wf * d.gwf[q0 + q]));
        }
    }
    // the psi point lies on the psi node row of the y-face below the centroid
    F.add(psi_noderow<W>(W::psi_rows(prec, pl, d.P.Mz, bz), d.P, bx, jlo, kz, kx) * nyh);
    return two ? 49 + 14 * k : 49 + 7 * k;
}

// The same with every value interpolated on its own: linear interpolation (main passes with
// interpolation_method linear), linear in y with the nearest column (the error pass).
template <int METHOD, class L>
__device__ __forceinline__ float plain_loc(const L& load, const NodeField& F, const int* anc, const float* q) {
    if constexpr (METHOD == INTERP_LINEAR) return lin3d_loc(load, F, anc, q);
    else return lin1dy_loc(load, F, anc, q);
}
template <int METHOD>
__device__ __forceinline__ void piece_quad32_plain(const PassDesc& d, const int* anc, float cx, float cy, float cz,
                                                   float ny, const float* __restrict__ a, const PsiLoad& pl, Kahan& F) {
    const PlainLoad al{a};
    float yp = cy;
    if (d.use_integral) {
        const YSpan Y = y_span(d, cy);
        const bool two = !(Y.f < 0.5f);
        const int k = d.k, np = two ? 2 * k : k;
        for (int m = 0; m < np; ++m) {
            const bool second = m >= k;
            const int q = second ? m - k : m;
            const float lo = second ? Y.ylo + 0.5f : Y.ylo;
            const float hl = second ? (cy - lo) * 0.5f : (two ? 0.25f : (cy - Y.ylo) * 0.5f);
            const float w = (second ? ny * (Y.f - 0.5f) : (two ? ny * 0.5f : ny * Y.f)) * d.gwf[q];
            const float qq[3] = {cx, hl * d.gxf[q] + hl + lo, cz};
            F.add(plain_loc<METHOD>(al, d.A, anc, qq) * w);
        }
        yp = Y.ylo;
    }
    const float qp[3] = {cx, yp, cz};
    F.add(plain_loc<METHOD>(pl, d.P, anc, qp) * (ny * d.invhf));
}

__device__ __forceinline__ void corners(int fam, int i, int j, int k, int* ci, int* cj, int* ck) {
    if (fam == 0) {
        ci[0] = i; cj[0] = j; ck[0] = k;   ci[1] = i; cj[1] = j + 1; ck[1] = k;
        ci[2] = i; cj[2] = j + 1; ck[2] = k + 1;   ci[3] = i; cj[3] = j; ck[3] = k + 1;
    } else if (fam == 1) {
        ci[0] = i; cj[0] = j; ck[0] = k;   ci[1] = i; cj[1] = j; ck[1] = k + 1;
        ci[2] = i + 1; cj[2] = j; ck[2] = k + 1;   ci[3] = i + 1; cj[3] = j; ck[3] = k;
    } else {
        ci[0] = i; cj[0] = j; ck[0] = k;   ci[1] = i + 1; cj[1] = j; ck[1] = k;
        ci[2] = i + 1; cj[2] = j + 1; ck[2] = k;   ci[3] = i; cj[3] = j + 1; ck[3] = k;
    }
}

// psi base node of a face / cell anchored at (i,j,k), clamped into the psi array
__device__ __forceinline__ long long psi_node(const NodeField& P, int i, int j, int k) {
    return idx3(P, clampi(i, P.Mx - 1), clampi(j, P.My - 1), clampi(k, P.Mz - 1));
}

// a family's arrays of the store, selected without indexing the kernel parameter (an indexed
// parameter array is copied to the stack frame)
__device__ __forceinline__ int2* range_of(const PieceStore& ps, int fam) {
    return fam == 0 ? ps.range[0] : (fam == 1 ? ps.range[1] : ps.range[2]);
}
__device__ __forceinline__ float2* normal_of(const PieceStore& ps, int fam) {
    return fam == 0 ? ps.normal[0] : (fam == 1 ? ps.normal[1] : ps.normal[2]);
}

// a face's range word: pieces of the lower cell's clip and of the upper cell's, second clip or not
__device__ __forceinline__ int range_bits(int nfwd, int nrev, bool multi) {
    return nfwd | (nrev << 15) | ((multi ? 1 : 0) << 30);
}

// Face pipeline of the chosen form, per pass:
//  k_clip32     one thread per unique face: backtraced corners, clip in shared memory (twice
//               when an iso-line crosses a piece more than twice), pieces appended
//               contiguously per face (warp prefix sum + one atomic per warp), y-normal sums;
//               a face the shared pool cannot hold goes to a list
//  k_clip32_deferred  the listed faces in a larger shared pool, appended the same way
//  k_clip32_local  those that outgrow it too, in local memory
//  k_quad32     one thread per piece: quadrature + WENO6 (uniform work per thread, no clip
//               code, so fewer registers and no divergence from the piece count);
//  k_facesum32  one thread per face: compensated sum of its pieces in emission order.
// lattice index of face id of family fam (ids are below 2^29): two 32-bit divisions
__device__ __forceinline__ void face_of32(int fam, const NodeField& A, unsigned id, int& i, int& j, int& k) {
    const unsigned Fy = A.My + (fam == 1), Fz = A.Mz + (fam == 2);
    const unsigned t = id / Fz;
    k = (int)(id - t * Fz);
    const unsigned ii = t / Fy;
    i = (int)ii;
    j = (int)(t - ii * Fy);
}

// corners of face id of family fam, in cells relative to its anchor, backtraced by disp
__device__ __forceinline__ void face_geometry(const PassDesc& d, int fam, long long id, const float* __restrict__ disp,
                                              LocalFace& g) {
    int i, j, k;
    face_of32(fam, d.A, (unsigned)id, i, j, k);
    int ci[4], cj[4], ck[4];
    corners(fam, i, j, k, ci, cj, ck);
    g.anc[0] = i; g.anc[1] = j; g.anc[2] = k;
    const int Ly = d.A.My + 1, Lz = d.A.Mz + 1;
    const float sx = d.comp == 0 ? -0.5f : 0.f, sy = d.comp == 1 ? -0.5f : 0.f, sz = d.comp == 2 ? -0.5f : 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        float dx = 0.f, dy = 0.f, dz = 0.f;
        if (!d.zero_velocity) {
            const long long vid = ((long long)ci[q] * Ly + cj[q]) * Lz + ck[q];
            dx = disp[3 * vid]; dy = disp[3 * vid + 1]; dz = disp[3 * vid + 2];
        }
        g.x[q] = float(ci[q] - i) + sx + dx;
        g.y[q] = float(cj[q] - j) + sy + dy;
        g.z[q] = float(ck[q] - k) + sz + dz;
    }
}

__device__ __forceinline__ void warp_counters(unsigned long long pc, unsigned fc, unsigned mc, unsigned st, int lane,
                                              unsigned* status, unsigned long long* counters) {
    for (int o = 16; o > 0; o >>= 1) {
        pc += __shfl_down_sync(0xffffffffu, pc, o);
        fc += __shfl_down_sync(0xffffffffu, fc, o);
        mc += __shfl_down_sync(0xffffffffu, mc, o);
        st |= __shfl_down_sync(0xffffffffu, st, o);
    }
    if (lane == 0) {
        if (fc) { atomicAdd(&counters[0], (unsigned long long)fc); atomicAdd(&counters[1], pc); }
        if (mc) atomicAdd(&counters[2], (unsigned long long)mc);
        if (st) atomicOr(status, st);
    }
}

// Both clips of a face into a pool; false: it does not fit.
template <class Pool>
__device__ __forceinline__ bool clip_both(const PassDesc& d, const LocalFace& g, const Pool& P, int& npieces, bool& multi,
                                          int& nst, int& nfwd, float& N, float& Nr) {
    Kahan ny;
    if (!clip32_fast(d, g, npieces, multi, nst, ny, P)) return false;
    nfwd = nst;
    N = ny.value();
    Nr = -N;
    if (multi) {
        ny = Kahan();
        int np2 = 0;
        bool m2 = false;
        if (!clip32_fast(d, reversed_face(g), np2, m2, nst, ny, P)) return false;
        Nr = ny.value();
    }
    return true;
}

// fast = 0 sends every face to the list
__global__ void __launch_bounds__(kClipThreads, kClipBlocks) k_clip32(PassDesc d, FamilyBlocks fb,
                                                                      const float* __restrict__ disp, PieceStore ps,
                                                                      unsigned* status, unsigned long long* counters,
                                                                      int fast) {
    extern __shared__ float clip_smem[];
    const FastPool P{clip_smem + threadIdx.x};
    const int fam = fb.family(blockIdx.x);
    const long long id = (long long)(blockIdx.x - fb.start(fam)) * blockDim.x + threadIdx.x;
    const long long nface = family_faces(d, fam);
    const int lane = threadIdx.x & 31;
    int npieces = 0, nst = 0, nfwd = 0;
    bool multi = false, ok = false;
    if (id < nface) {
        LocalFace g;
        face_geometry(d, fam, id, disp, g);
        float N = 0.f, Nr = 0.f;
        ok = fast != 0 && clip_both(d, g, P, npieces, multi, nst, nfwd, N, Nr);
        if (ok) {
            normal_of(ps, fam)[id] = make_float2(N, Nr);
        } else {
            npieces = 0;
            const unsigned q = atomicAdd(ps.count + 1, 1u);
            ps.deferred[q] = (fam << 29) | (int)id;
        }
    }
    const int cnt = ok ? nst : 0;
    const long long start = warp_slots(ps.count, cnt, lane);
    if (ok) {
        if (start + cnt <= ps.cap) {
            const int tag = (fam << 29) | (int)id;
            for (int q = 0; q < cnt; ++q) { ps.rec[start + q] = P.piece(q); ps.face[start + q] = tag; }
        }
        // a range beyond the capacity is kept as it is: the host sees the count, grows the
        // store and runs the pass again
        range_of(ps, fam)[id] = make_int2((int)start, range_bits(nfwd, cnt - nfwd, multi));
    }
    warp_counters((unsigned long long)npieces, ok ? 1u : 0u, (ok && multi) ? 1u : 0u, 0u, lane, status, counters);
}

// f(entry of a list of nd, or -1) by whole warps; a short list is spread over the warps: the faces of
// one would wait for each other.
template <class Body>
__device__ __forceinline__ void for_listed(long long nd, const Body& body) {
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    const long long warps = (long long)gridDim.x * wpb;
    const int per = (int)min(32LL, (nd + warps - 1) / warps);
    for (long long base = ((long long)blockIdx.x * wpb + (threadIdx.x >> 5)) * per; base < nd; base += warps * per)
        body(lane < per && base + lane < nd ? base + lane : -1);
}

// One listed face a lane (tag -1: none), clipped by clip32 in local memory.
__device__ __forceinline__ void clip_local(const PassDesc& d, int tag, const float* __restrict__ disp,
                                           const PieceStore& ps, unsigned* status, unsigned long long* counters) {
    const int fam = tag >> 29, lane = threadIdx.x & 31;
    const long long id = tag & ((1 << 29) - 1);
    unsigned st = 0;
    int npieces = 0, nfwd = 0;
    bool multi = false;
    PieceSink sink;
    if (tag >= 0) {
        LocalFace g;
        face_geometry(d, fam, id, disp, g);
        clip32(d, g, st, npieces, multi, sink);
        nfwd = sink.n;
        const float N = sink.ny.value();
        float Nr = -N;
        if (multi) {
            int np2 = 0;
            bool m2 = false;
            sink.ny = Kahan();
            clip32(d, reversed_face(g), st, np2, m2, sink);
            Nr = sink.ny.value();
        }
        normal_of(ps, fam)[id] = make_float2(N, Nr);
    }
    const int cnt = sink.n;
    const long long start = warp_slots(ps.count, cnt, lane);
    if (tag >= 0) {
        if (start + cnt <= ps.cap)
            for (int q = 0; q < cnt; ++q) { ps.rec[start + q] = sink.p[q]; ps.face[start + q] = tag; }
        range_of(ps, fam)[id] = make_int2((int)start, range_bits(nfwd, cnt - nfwd, multi));
    }
    warp_counters((unsigned long long)npieces, tag >= 0 ? 1u : 0u, (tag >= 0 && multi) ? 1u : 0u, st, lane, status, counters);
}

// The faces k_clip32 listed (all families), ps.count[1] of them, in a larger pool.  Those that outgrow it
// too are for the local-memory clipper.  Of a short list (a face a warp) they are clipped here; of a longer
// one they are moved to the back of the list array and counted in ps.count[2], or keep their place
// where the array has no room left, the other places blanked.
//
// The local-memory clipper then has a kernel of its own, because a warp in which one face needs it waits
// for that face, and because the pools leave 8 warps on an SM here: with it in this kernel for every
// list, a density step at 64^3 took 7.7 ms at CFL 16 (two faces in five listed, one in fifty past the larger
// pool) and 23 ms at CFL 24, and 3.6 and 6.6 ms so.  Faces over kDeferCells cells or more (clip_cells) are moved
// without an attempt: of those over 20 to 30 half would fit, of larger ones hardly any.
constexpr int kDeferBlocks = 152 * 4, kDeferCells = 20;
__host__ __device__ __forceinline__ bool short_list(unsigned listed) {
    return listed <= (unsigned)(kDeferBlocks * (kDeferThreads / 32));
}
__global__ void __launch_bounds__(kDeferThreads) k_clip32_deferred(PassDesc d, const float* __restrict__ disp, PieceStore ps,
                                                                   unsigned* status, unsigned long long* counters,
                                                                   int fast) {
    __shared__ float pool[DeferPool::kWords * kDeferThreads];
    const DeferPool P{pool + threadIdx.x};
    const unsigned nd = ps.count[1];
    const bool few = short_list(nd);
    const int lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && threadIdx.x == 0 && nd > 0) atomicAdd(&counters[4], (unsigned long long)nd);
    for_listed(nd, [&](long long t) {
        const int tag = t >= 0 ? ps.deferred[t] : 0;
        const int fam = tag >> 29;
        const long long id = tag & ((1 << 29) - 1);
        int npieces = 0, cnt = 0, nfwd = 0;
        bool multi = false, ok = false;
        if (t >= 0) {
            LocalFace g;
            face_geometry(d, fam, id, disp, g);
            float N = 0.f, Nr = 0.f;
            ok = fast != 0 && (few || clip_cells(d, g) < kDeferCells) && clip_both(d, g, P, npieces, multi, cnt, nfwd, N, Nr);
            if (ok) normal_of(ps, fam)[id] = make_float2(N, Nr);
        }
        if (!ok) npieces = cnt = 0;
        const long long start = warp_slots(ps.count, cnt, lane);
        if (ok) {
            if (start + cnt <= ps.cap)
                for (int q = 0; q < cnt; ++q) { ps.rec[start + q] = P.piece(q); ps.face[start + q] = tag; }
            range_of(ps, fam)[id] = make_int2((int)start, range_bits(nfwd, cnt - nfwd, multi));
        }
        warp_counters((unsigned long long)npieces, ok ? 1u : 0u, (ok && multi) ? 1u : 0u, 0u, lane, status, counters);
        const bool left = t >= 0 && !ok;
        if (few) {
            if (__any_sync(0xffffffffu, left)) clip_local(d, left ? tag : -1, disp, ps, status, counters);
        } else if (t >= 0) {
            const long long q = left ? (long long)atomicAdd(ps.count + 2, 1u) : 0;
            const bool keep = left && nd + q >= ps.listcap;
            if (left && !keep) ps.deferred[ps.listcap - 1 - q] = tag;
            if (!keep) ps.deferred[t] = -1;
        }
    });
}

// The faces that k_clip32_deferred leaves: ps.count[2] of them, those past the room in their old places.
__global__ void __launch_bounds__(128) k_clip32_local(PassDesc d, const float* __restrict__ disp, PieceStore ps,
                                                      unsigned* status, unsigned long long* counters) {
    const long long nd = ps.count[1], left = ps.count[2], room = ps.listcap - nd, moved = min(left, room);
    for_listed(left > room ? moved + nd : moved, [&](long long t) {
        const int tag = t < 0 ? -1 : (t < moved ? ps.deferred[ps.listcap - 1 - t] : ps.deferred[t - moved]);
        clip_local(d, tag, disp, ps, status, counters);
    });
}

// Faces at rest (the zero-velocity pass, the MacCormack face at rest) are the same square in
// every face's local coordinates, so they all have the same pieces: k_rest_clip32 clips one
// with clip32 (one thread) into ps.rest -- [0] (count, range bits, pieces with area, status)
// as ints, [1] (N, Nr), [2..] the pieces -- and k_rest_fill32 gives every face of the family a
// copy, face-major (face id's pieces at id * count): the pieces, order and sums of a clip per
// face.  Only y-faces emit pieces at rest.
__global__ void k_rest_clip32(PassDesc d, int fam, PieceStore ps) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    LocalFace g;
    face_geometry(d, fam, 0, nullptr, g);
    // in a shared pool, or else in local memory (12 us a launch)
    typedef ClipPool<36, 28, 1, unsigned long long> RestPool;
    __shared__ float pool[RestPool::kWords];
    const RestPool P{pool};
    unsigned st = 0;
    int npieces = 0, nst = 0, nfwd = 0;
    bool multi = false;
    float N = 0.f, Nr = 0.f;
    if (clip_both(d, g, P, npieces, multi, nst, nfwd, N, Nr)) {
        reinterpret_cast<int4*>(ps.rest)[0] = make_int4(nst, range_bits(nfwd, nst - nfwd, multi), npieces, 0);
        ps.rest[1] = make_float4(N, Nr, 0.f, 0.f);
        for (int q = 0; q < nst; ++q) ps.rest[2 + q] = P.piece(q);
        return;
    }
    npieces = 0;
    multi = false;
    PieceSink sink;
    clip32(d, g, st, npieces, multi, sink);
    nfwd = sink.n;
    N = sink.ny.value();
    Nr = -N;
    if (multi) {
        int np2 = 0;
        bool m2 = false;
        sink.ny = Kahan();
        clip32(d, reversed_face(g), st, np2, m2, sink);
        Nr = sink.ny.value();
    }
    reinterpret_cast<int4*>(ps.rest)[0] =
        make_int4(sink.n, range_bits(nfwd, sink.n - nfwd, multi), npieces, (int)st);
    ps.rest[1] = make_float4(N, Nr, 0.f, 0.f);
    for (int q = 0; q < sink.n; ++q) ps.rest[2 + q] = sink.p[q];
}

__global__ void k_rest_fill32(PassDesc d, int fam, PieceStore ps, unsigned* status, unsigned long long* counters) {
    const long long nface = (long long)(d.A.Mx + (fam == 0)) * (d.A.My + (fam == 1)) * (d.A.Mz + (fam == 2));
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int4 hd = reinterpret_cast<const int4*>(ps.rest)[0];
    const int cnt = hd.x;
    if (id == 0) {
        atomicAdd(ps.count, (unsigned)(cnt * nface));
        atomicAdd(&counters[0], (unsigned long long)nface);
        atomicAdd(&counters[1], (unsigned long long)hd.z * (unsigned long long)nface);
        if ((hd.y >> 30) & 1) atomicAdd(&counters[2], (unsigned long long)nface);
        if (hd.w) atomicOr(status, (unsigned)hd.w);
    }
    if (id >= nface) return;
    const long long start = id * cnt;
    if (start + cnt <= ps.cap) {
        const int tag = (fam << 29) | (int)id;
        for (int q = 0; q < cnt; ++q) { ps.rec[start + q] = ps.rest[2 + q]; ps.face[start + q] = tag; }
    }
    range_of(ps, fam)[id] = make_int2((int)start, hd.y);
    const float4 nr = ps.rest[1];
    normal_of(ps, fam)[id] = make_float2(nr.x, nr.y);
}

// Tiles of kQuadThreads pieces, `run` (up to 8) consecutive ones at a time per CTA: pieces are stored
// nearly in face order, so a run covers neighbouring z-lines and finds their records in L1.  The number
// of pieces is the store's own, so a stage whose pieces surely fit is launched without waiting for it.
// The next tile's piece is loaded before the present one is integrated.  Each piece's flux takes
// the place of its face tag.
template <class Body>
__device__ __forceinline__ void for_pieces(const PassDesc& d, const PieceStore& ps, const Body& body) {
    const long long npc = min((long long)ps.count[0], (long long)ps.cap);
    const long long ntile = (npc + kQuadThreads - 1) / kQuadThreads;
    const int run = (int)max(1LL, min(8LL, ntile / (4LL * gridDim.x)));
    long long tile = (long long)blockIdx.x * run;
    int left = run;
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    long long t = tile * kQuadThreads + threadIdx.x;
    bool on = tile < ntile && t < npc;
    float4 p = on ? ps.rec[t] : none;
    int tag = on ? ps.face[t] : 0;
    while (tile < ntile) {
        if (--left > 0) ++tile;
        else { left = run; tile += (long long)(gridDim.x - 1) * run + 1; }
        const long long tn = tile * kQuadThreads + threadIdx.x;
        const bool next = tile < ntile && tn < npc;
        const float4 pn = next ? ps.rec[tn] : none;
        const int tagn = next ? ps.face[tn] : 0;
        if (on) {
            int anc[3];
            face_of32(tag >> 29, d.A, (unsigned)(tag & ((1 << 29) - 1)), anc[0], anc[1], anc[2]);
            ps.face[t] = __float_as_int(body(p, anc));
        }
        p = pn; tag = tagn; t = tn; on = next;
    }
}

template <class W>
__global__ void __launch_bounds__(kQuadThreads, 4) k_quad32(PassDesc d, typename W::Records ar,
                                                            const float4* __restrict__ prec,
                                                            const float2* __restrict__ psi, PieceStore ps,
                                                            unsigned long long* counters) {
    __shared__ float zcol[42 * kQuadThreads];   // each thread's z-pass column (rec_zpass)
    unsigned long long ec = 0;
    for_pieces(d, ps, [&](const float4& p, const int* anc) {
        const float2 b = __ldg(psi + psi_node(d.P, anc[0], anc[1], anc[2]));
        Kahan F;
        ec += (unsigned long long)piece_quad32<W>(d, anc, p.x, p.y, p.z, p.w, ar, prec, PsiLoad{psi, b.x, b.y}, F,
                                                  zcol + threadIdx.x);
        return F.value();
    });
    for (int o = 16; o > 0; o >>= 1) ec += __shfl_down_sync(0xffffffffu, ec, o);
    if ((threadIdx.x & 31) == 0 && ec) atomicAdd(&counters[3], ec);
}

template <int METHOD>
__global__ void __launch_bounds__(kQuadThreads) k_quad32_plain(PassDesc d, const float* __restrict__ a,
                                                               const float2* __restrict__ psi, PieceStore ps) {
    for_pieces(d, ps, [&](const float4& p, const int* anc) {
        const float2 b = __ldg(psi + psi_node(d.P, anc[0], anc[1], anc[2]));
        Kahan F;
        piece_quad32_plain<METHOD>(d, anc, p.x, p.y, p.z, p.w, a, PsiLoad{psi, b.x, b.y}, F);
        return F.value();
    });
}

// flux = wgt (F, N) (acc = 0) or flux + wgt (F, N) (acc = 1): the weighted faces of the flux
// MacCormack scheme accumulate into one (flux, y-normal sum) pair per face
// With fvol: (M, Mr) = sums of y n_y of the face's pieces in cells (y relative to the face
// anchor), the same weighting, for the cell volumes of the cell-volume correction.
struct FaceSums {
    float2 *flux[3], *flux_rev[3], *fvol[3];
};
__global__ void k_facesum32(PassDesc d, FamilyBlocks fb, PieceStore ps, FaceSums fs, unsigned* status, float wgt, int acc) {
    const int fam = fb.family(blockIdx.x);
    const long long id = (long long)(blockIdx.x - fb.start(fam)) * blockDim.x + threadIdx.x;
    if (id >= family_faces(d, fam)) return;
    float2* const flux = fam == 0 ? fs.flux[0] : (fam == 1 ? fs.flux[1] : fs.flux[2]);
    float2* const flux_rev = fam == 0 ? fs.flux_rev[0] : (fam == 1 ? fs.flux_rev[1] : fs.flux_rev[2]);
    float2* const fvol = fam == 0 ? fs.fvol[0] : (fam == 1 ? fs.fvol[1] : fs.fvol[2]);
    const int2 r = range_of(ps, fam)[id];
    const int nf = r.y & 0x7fff, nr = (r.y >> 15) & 0x7fff;
    const bool multi = (r.y >> 30) & 1;
    Kahan F, Fr;
    for (int q = 0; q < nf; ++q) F.add(__int_as_float(ps.face[(long long)r.x + q]));
    for (int q = 0; q < nr; ++q) Fr.add(__int_as_float(ps.face[(long long)r.x + nf + q]));
    const float f = F.value(), fr = multi ? Fr.value() : -f;
    const float2 nrm = normal_of(ps, fam)[id];
    float2 a = make_float2(wgt * f, wgt * nrm.x), b = make_float2(wgt * fr, wgt * nrm.y);
    if (acc) {
        const float2 a0 = flux[id], b0 = flux_rev[id];
        a.x += a0.x; a.y += a0.y; b.x += b0.x; b.y += b0.y;
    }
    flux[id] = a;
    flux_rev[id] = b;
    if (!isfinite(f) || !isfinite(fr)) atomicOr(status, (unsigned)ST_NONFINITE);
    if (fvol) {
        Kahan M, Mr;
        for (int q = 0; q < nf; ++q) { const float4 p = ps.rec[(long long)r.x + q]; M.add(p.y * p.w); }
        for (int q = 0; q < nr; ++q) { const float4 p = ps.rec[(long long)r.x + nf + q]; Mr.add(p.y * p.w); }
        const float m = M.value(), mr = multi ? Mr.value() : -m;
        float2 v = make_float2(wgt * m, wgt * mr);
        if (acc) { const float2 v0 = fvol[id]; v.x += v0.x; v.y += v0.y; }
        fvol[id] = v;
    }
}

// Advected cell volumes in cells (cell-volume correction, density only): the volume points
// y n_y of a cell's pieces, from the per-face sums with y relative to each face's anchor.  The
// faces of cell (i, j, k) are anchored at row j except its upper y-face (row j + 1), which
// adds its y-normal sum; the term j sum_f s_f N_f of the common row is zero for a closed
// surface and is dropped (in FP32 it would only carry rounding).
__global__ void k_volume_gather32(PassDesc d, const float2* __restrict__ vx, const float2* __restrict__ vy,
                                  const float2* __restrict__ vz, const float2* __restrict__ fy, float* __restrict__ vol) {
    const int Mx = d.A.Mx, My = d.A.My, Mz = d.A.Mz;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)Mx * My * Mz) return;
    const int k = (int)(id % Mz);
    const int j = (int)((id / Mz) % My);
    const int i = (int)(id / ((long long)Mz * My));
    Kahan s;
    s.add(vx[((long long)(i + 1) * My + j) * Mz + k].x);
    s.add(vx[((long long)i * My + j) * Mz + k].y);
    s.add(vy[((long long)i * (My + 1) + j + 1) * Mz + k].x);
    s.add(vy[((long long)i * (My + 1) + j) * Mz + k].y);
    s.add(vz[((long long)i * My + j) * (Mz + 1) + k + 1].x);
    s.add(vz[((long long)i * My + j) * (Mz + 1) + k].y);
    s.add(fy[((long long)i * (My + 1) + j + 1) * Mz + k].y);
    vol[id] = s.value();
}

// rho'(c) = sum_f s_f [Ft + (Psi0(f) - Psi_c) Ny], compensated
__global__ void k_gather32(PassDesc d, const float2* __restrict__ fx, const float2* __restrict__ fy,
                           const float2* __restrict__ fz, const float2* __restrict__ rx,
                           const float2* __restrict__ ry, const float2* __restrict__ rz,
                           const float2* __restrict__ psi, const float* __restrict__ in, float* __restrict__ out,
                           int mode) {
    const int Mx = d.A.Mx, My = d.A.My, Mz = d.A.Mz;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)Mx * My * Mz) return;
    const int k = (int)(id % Mz);
    const int j = (int)((id / Mz) % My);
    const int i = (int)(id / ((long long)Mz * My));
    const float2 pc = __ldg(psi + psi_node(d.P, i, j, k));
    const float invh = d.invhf;
    auto base_diff = [&](int a, int b, int c) {
        const float2 p = __ldg(psi + psi_node(d.P, a, b, c));
        return ((p.x - pc.x) + (p.y - pc.y)) * invh;
    };
    // lower faces (anchor = the cell itself): base difference 0
    const float2 lx = rx[((long long)i * My + j) * Mz + k];
    const float2 ly = ry[((long long)i * (My + 1) + j) * Mz + k];
    const float2 lz = rz[((long long)i * My + j) * (Mz + 1) + k];
    const float2 ux = fx[((long long)(i + 1) * My + j) * Mz + k];
    const float2 uy = fy[((long long)i * (My + 1) + j + 1) * Mz + k];
    const float2 uz = fz[((long long)i * My + j) * (Mz + 1) + k + 1];
    Kahan s;
    s.add(lx.x); s.add(ly.x); s.add(lz.x);
    s.add(ux.x); s.add(uy.x); s.add(uz.x);
    s.add(base_diff(i + 1, j, k) * ux.y);
    s.add(base_diff(i, j + 1, k) * uy.y);
    s.add(base_diff(i, j, k + 1) * uz.y);
    const float val = s.value();
    if (mode == 0) out[id] = val;
    else if (mode == 1) out[id] = in[id] - val;
    else out[id] = out[id] + val;
}

}  // namespace

// One face stage of the FP32 pipeline: clip (growing the piece store and clipping again when
// it is too small), per-piece quadrature, per-face sums weighted into the face fluxes.
static cudaError_t face_stage32(const PassDesc& d, const float* a, const float2* psi, const float* disp,
                                const PassWork<float>& w, float wgt, int acc, cudaStream_t s) {
    PieceStore& ps = *w.pieces;
    long long nface[3];
    for (int fam = 0; fam < 3; ++fam)
        nface[fam] = (long long)(d.A.Mx + (fam == 0)) * (d.A.My + (fam == 1)) * (d.A.Mz + (fam == 2));
    if (std::max(nface[0], std::max(nface[1], nface[2])) >= (1LL << 29)) return cudaErrorInvalidValue;
    // Faces at rest (the zero-velocity pass, the MacCormack face at rest): an x- or z-face keeps
    // its four corners at one x (z), so every piece's y-normal is exactly zero and the face
    // emits no piece; its flux, normal and volume sums are zero and only the y-faces are clipped.
    const bool rest = d.zero_velocity != 0;
    if (rest && !acc) {
        for (int fam = 0; fam < 3; fam += 2) {
            cudaMemsetAsync(w.flux[fam], 0, nface[fam] * sizeof(float2), s);
            cudaMemsetAsync(w.flux_rev[fam], 0, nface[fam] * sizeof(float2), s);
            if (d.volumes) cudaMemsetAsync(w.fvol[fam], 0, nface[fam] * sizeof(float2), s);
        }
    }
    // At rest at most one line of each colour crosses the unit square: four pieces.  With room for that
    // many the host does not wait for the count.
    constexpr long long kRestPieces = 4;
    const bool fits = rest && ps.clip_fast && ps.cap >= kRestPieces * nface[1];
    unsigned npc = 0;
    cudaError_t ea = cudaFuncSetAttribute(k_clip32, cudaFuncAttributeMaxDynamicSharedMemorySize, kClipSmem);
    if (ea == cudaSuccess)
        ea = cudaFuncSetAttribute(k_clip32, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (ea != cudaSuccess) return ea;
    // the work counters as they were before the clip: a second attempt starts from them again
    ea = cudaMemcpyAsync(ps.saved, w.counters, 5 * sizeof(unsigned long long), cudaMemcpyDeviceToDevice, s);
    if (ea != cudaSuccess) return ea;
    for (int attempt = 0; attempt < 2; ++attempt) {
        cudaMemsetAsync(ps.count, 0, 3 * sizeof(unsigned), s);
        if (attempt > 0)
            cudaMemcpyAsync(w.counters, ps.saved, 5 * sizeof(unsigned long long), cudaMemcpyDeviceToDevice, s);
        if (rest && ps.clip_fast) {
            k_rest_clip32<<<1, 32, 0, s>>>(d, 1, ps);
            k_rest_fill32<<<nblk(nface[1], 256), 256, 0, s>>>(d, 1, ps, w.status, w.counters);
        } else {
            const FamilyBlocks fb = family_blocks(nface, rest, kClipThreads);
            k_clip32<<<fb.first[3], kClipThreads, kClipSmem, s>>>(d, fb, disp, ps, w.status, w.counters, ps.clip_fast);
            k_clip32_deferred<<<kDeferBlocks, kDeferThreads, 0, s>>>(d, disp, ps, w.status, w.counters, ps.clip_fast);
        }
        if (fits) {
            npc = (unsigned)(kRestPieces * nface[1]);
            break;
        }
        unsigned counts[3];   // pieces, faces listed, faces left
        cudaError_t e = cudaMemcpyAsync(counts, ps.count, sizeof(counts), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e == cudaSuccess && counts[2] > 0) {
            k_clip32_local<<<152 * 8, 128, 0, s>>>(d, disp, ps, w.status, w.counters);
            if (w.launches) ++*w.launches;
            // no second wait where the pieces these faces can have fit at any rate (7 us a pass)
            const long long most = (long long)counts[0] + (long long)counts[2] * kMaxPieces32;
            if (most <= std::min(ps.cap, (long long)INT_MAX)) {
                npc = (unsigned)most;
                break;
            }
            e = cudaMemcpyAsync(counts, ps.count, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        }
        if (e != cudaSuccess) return e;
        npc = counts[0];
        if ((long long)npc <= ps.cap) break;
        // more pieces than the store holds: grow it and clip again
        e = piece_store_reserve(ps, (long long)npc + npc / 4 + 1024, std::max(nface[0], std::max(nface[1], nface[2])),
                                *w.records);
        if (e != cudaSuccess) return e;
    }
    if ((long long)npc > ps.cap) return cudaErrorMemoryAllocation;
    if (npc > 0) {
        const long long ntile = ((long long)npc + kQuadThreads - 1) / kQuadThreads;
        const unsigned grid = (unsigned)std::min<long long>(ntile, 152 * 8);
        const RecordStore& rec = *w.records;   // growing the piece store may have taken them
        prof_mark(w, 0, s);
        if (d.interp == INTERP_LINEAR)
            k_quad32_plain<INTERP_LINEAR><<<grid, kQuadThreads, 0, s>>>(d, a, psi, ps);
        else if (d.interp != INTERP_WENO6)
            k_quad32_plain<INTERP_1DY_LINEAR><<<grid, kQuadThreads, 0, s>>>(d, a, psi, ps);
        else if (!rec.field && d.comp < 0)
            k_quad32<FromField<WenoNewton>><<<grid, kQuadThreads, 0, s>>>(d, {FieldRows{a, d.A.Mz}}, nullptr, psi, ps, w.counters);
        else if (!rec.field)
            k_quad32<FromField<WenoSamples>><<<grid, kQuadThreads, 0, s>>>(d, {FieldRows{a, d.A.Mz}}, nullptr, psi, ps, w.counters);
        else if (d.comp < 0)
            k_quad32<WenoNewton><<<grid, kQuadThreads, 0, s>>>(d, newton_records(d.A, rec.field), (const float4*)rec.psi, psi,
                                                               ps, w.counters);
        else
            k_quad32<WenoSamples><<<grid, kQuadThreads, 0, s>>>(d, sample_records(d.A, rec.field), nullptr, psi, ps,
                                                                w.counters);
        prof_mark(w, 1, s);
    }
    FaceSums fs;
    for (int fam = 0; fam < 3; ++fam) {
        fs.flux[fam] = (float2*)w.flux[fam];
        fs.flux_rev[fam] = (float2*)w.flux_rev[fam];
        fs.fvol[fam] = d.volumes ? (float2*)w.fvol[fam] : nullptr;
    }
    const FamilyBlocks fb = family_blocks(nface, rest, 256);
    k_facesum32<<<fb.first[3], 256, 0, s>>>(d, fb, ps, fs, w.status, wgt, acc);
    return cudaGetLastError();
}

template <>
cudaError_t run_pass<float>(const PassDesc& d64, const VelocityFields& vel64, const float* a, const PassWork<float>& w,
                            const float* in, float* out, int mode, cudaStream_t s) {
    const PassDesc d = desc32(d64);
    VelocityFields vel = vel64;
    vel.fu = field32(vel64.fu); vel.fv = field32(vel64.fv); vel.fw = field32(vel64.fw);
    float2* psi = (float2*)w.psi;
    psi32(d, a, psi, s);
    if (d.interp == INTERP_WENO6 && w.records->field) {
        // without the y-integral no point of the field itself is interpolated
        if (d.comp >= 0) {
            const WenoSamples::Records r = sample_records(d.A, w.records->field);
            if (d.use_integral)
                k_records_samples<<<nblk(weno_rec_count(d.A), 256), 256, 0, s>>>(d.A, a, const_cast<float4*>(r.r),
                                                                                 const_cast<float*>(r.r2));
        } else {
            if (d.use_integral)
                k_records_newton<false><<<nblk(weno_rec_count(d.A), 256), 256, 0, s>>>(d.A, a, (float4*)w.records->field);
            k_records_newton<true><<<nblk(weno_rec_count(d.P), 256), 256, 0, s>>>(d.P, psi,
                                                                                   (float4*)w.records->psi);
        }
    }
    const long long nv = (long long)(d.A.Mx + 1) * (d.A.My + 1) * (d.A.Mz + 1);
    if (!d.zero_velocity)
        backtrace32(d, vel, w.verts, s);
    cudaError_t e;
    if (!d.maccormack || d.zero_velocity) {
        // one face per face slot; with zero velocity the MacCormack faces coincide and their
        // weights sum to one
        e = face_stage32(d, a, psi, w.verts, w, 1.f, 0, s);
    } else {
        if (!w.verts2) return cudaErrorInvalidValue;
        k_forward32<<<nblk(nv, 128), 128, 0, s>>>(d, (const float*)vel.u, (const float*)vel.v, (const float*)vel.w,
                                                 vel.fu, vel.fv, vel.fw, w.verts, w.verts2);
        PassDesc rest = d;
        rest.zero_velocity = 1;
        e = face_stage32(rest, a, psi, w.verts, w, 0.5f, 0, s);                       // the face at rest
        if (e == cudaSuccess) e = face_stage32(d, a, psi, w.verts, w, 1.f, 1, s);     // backtraced
        if (e == cudaSuccess) e = face_stage32(d, a, psi, w.verts2, w, -0.5f, 1, s);  // traced back
    }
    if (e != cudaSuccess) return e;
    const long long nc = (long long)d.A.Mx * d.A.My * d.A.Mz;
    if (d.volumes) {
        if (!w.vol || !w.fvol[0] || d.comp >= 0) return cudaErrorInvalidValue;
        k_volume_gather32<<<nblk(nc, 256), 256, 0, s>>>(d, (const float2*)w.fvol[0], (const float2*)w.fvol[1],
                                                        (const float2*)w.fvol[2], (const float2*)w.flux[1], w.vol);
    }
    k_gather32<<<nblk(nc, 256), 256, 0, s>>>(d, (const float2*)w.flux[0], (const float2*)w.flux[1],
                                             (const float2*)w.flux[2], (const float2*)w.flux_rev[0],
                                             (const float2*)w.flux_rev[1], (const float2*)w.flux_rev[2], psi, in, out,
                                             mode);
    return cudaGetLastError();
}

cudaError_t piece_store_reserve(PieceStore& p, long long pieces, long long faces_per_family, RecordStore& mem) {
    cudaDeviceSynchronize();
    if (pieces > p.cap) {
        cudaFree(p.rec); cudaFree(p.face);
        p.rec = nullptr; p.face = nullptr; p.cap = 0;
        cudaError_t e = mem.alloc((void**)&p.rec, pieces * sizeof(float4));
        if (e == cudaSuccess) e = mem.alloc((void**)&p.face, pieces * sizeof(int));
        if (e != cudaSuccess) return e;
        p.cap = pieces;
    }
    if (!p.block) {
        // what does not grow, in one allocation
        auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
        const size_t nf = (size_t)faces_per_family;
        const size_t rb = up(nf * sizeof(int2)), nb = up(nf * sizeof(float2)), db = up(3 * nf * sizeof(int));
        const size_t eb = up((2 + kMaxPieces32) * sizeof(float4)), cb = 256;
        cudaError_t e = mem.alloc(&p.block, 3 * rb + 3 * nb + db + eb + 2 * cb);
        if (e != cudaSuccess) { p.block = nullptr; return e; }
        char* q = (char*)p.block;
        auto take = [&](size_t b) { char* r = q; q += b; return r; };
        p.count = (unsigned*)take(cb);
        p.saved = (unsigned long long*)take(cb);
        for (int f = 0; f < 3; ++f) { p.range[f] = (int2*)take(rb); p.normal[f] = (float2*)take(nb); }
        p.deferred = (int*)take(db);
        p.listcap = 3 * faces_per_family;
        p.rest = (float4*)take(eb);
    }
    return cudaSuccess;
}

void piece_store_free(PieceStore& p) {
    cudaFree(p.rec); cudaFree(p.face); cudaFree(p.block);
    p = PieceStore();
}

template <>
cudaError_t launch_psi<float>(const PassDesc& d64, const float* a, float* psi, cudaStream_t s) {
    const PassDesc d = desc32(d64);
    psi32(d, a, (float2*)psi, s);
    return cudaGetLastError();
}

template <>
cudaError_t launch_backtrace<float>(const PassDesc& d64, const VelocityFields& vel, float* verts, cudaStream_t s) {
    const PassDesc d = desc32(d64);
    VelocityFields v32 = vel;
    v32.fu = field32(vel.fu); v32.fv = field32(vel.fv); v32.fw = field32(vel.fw);
    backtrace32(d, v32, verts, s);
    return cudaGetLastError();
}

}  // namespace fia
