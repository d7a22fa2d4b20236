// fia_pressure.cu -- pressure projection (calc_pressure_3d.cpp:18-270) on the GPU.
//
// The reference assembles a CSR 7-point Laplacian over all cells but the last one (pinned
// to p = 0), right-hand side b = div(u) h, and solves it with amgcl (SA-AMG + CG).  Here
// the same operator is applied matrix-free and solved with CG on B = -A (symmetric positive
// definite on the free cells): Jacobi-preconditioned, or flexible CG around a preconditioner
// supplied by the caller (the learned one).  Solid cells are excluded like walls.
//
// Element arithmetic is in the field's own type; every dot product and norm is accumulated
// to FP64 accuracy: per thread exactly in double (FP64 form) or as an unevaluated float
// pair with FMA-exact products (FP32 form), across threads and blocks in double, with
// fixed per-block partials summed in block order by the last block of each kernel (no
// atomics on values, so the result does not depend on scheduling).
#include "fia_pressure.cuh"

#include <algorithm>
#include <type_traits>
#include <cmath>
#include <cstdint>

namespace fia {

constexpr int kRedBlocks = 152 * 6;
constexpr int kRedThreads = 256;
constexpr int kCgBatch = 16;

// scal layout
enum : int {
    S_ALPHA = 0, S_BETA = 1, S_RZ = 2, S_RR = 3, S_THRESH = 4, S_DONE = 5, S_ITERS = 6, S_DQ = 7,
    S_BETAJ = 8,                        // flexible CG: beta of direction slot j
    S_DQJ = S_BETAJ + kFcgMaxDirs + 1   // flexible CG: d.q of direction slot j
};
static_assert(S_DQJ + kFcgMaxDirs + 1 <= kScalDoubles, "scalar block too small for the FCG direction ring");

// ---------------------------------------------------------------------------------
// per-thread dot accumulators
// ---------------------------------------------------------------------------------
template <typename T>
struct DotAcc;

template <>
struct DotAcc<double> {
    double s = 0.0;
    __device__ __forceinline__ void add(double a, double b) { s = fma(a, b, s); }
    __device__ __forceinline__ double value() const { return s; }
};

template <>
struct DotAcc<float> {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(float a, float b) {
        const float p = __fmul_rn(a, b);
        const float pe = __fmaf_rn(a, b, -p);          // exact product error
        const float s = __fadd_rn(hi, p);
        const float bb = __fsub_rn(s, hi);
        const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(p, bb));
        hi = s;
        lo = __fadd_rn(lo, __fadd_rn(e, pe));
    }
    __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Block-level sums of NV values written to part[b + nb*q].
template <int NV>
__device__ __forceinline__ void block_sums(const double (&v)[NV], double* part) {
    __shared__ double sh[NV][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        const double s = warp_sum(v[q]);
        if (lane == 0) sh[q][wid] = s;
    }
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            double s = lane < nw ? sh[q][lane] : 0.0;
            s = warp_sum(s);
            if (lane == 0) part[blockIdx.x + gridDim.x * q] = s;
        }
    }
}

__device__ __forceinline__ bool last_block(unsigned* ticket) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
    __syncthreads();
    return last;
}

// sum of one partial row by the last block, in block order
__device__ double block_total(const double* part, int nblocks, int q) {
    __shared__ double sh[32];
    __shared__ double tot;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double s = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) s += __ldcg(part + b + nblocks * q);
    s = warp_sum(s);
    if (lane == 0) sh[wid] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[w];
        tot = t;
    }
    __syncthreads();
    return tot;
}

// The same for NV rows at once (each in block_total's order): row after row, the last block's loads,
// shuffles and barriers are waited for NV times.
template <int NV>
__device__ __forceinline__ void block_totals(const double* part, int nblocks, double (&tot)[NV]) {
    __shared__ double sh[NV][33];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double s[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) s[q] = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
#pragma unroll
        for (int q = 0; q < NV; ++q) s[q] += __ldcg(part + b + nblocks * q);
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        s[q] = warp_sum(s[q]);
        if (lane == 0) sh[q][wid] = s[q];
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[threadIdx.x][w];
        sh[threadIdx.x][32] = t;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; ++q) tot[q] = sh[q][32];
}

// ---------------------------------------------------------------------------------
// the operator
// ---------------------------------------------------------------------------------
struct Cell {
    int ix, iy, iz;
};
__device__ __forceinline__ Cell decode(unsigned c, int ny, int nz) {
    Cell r;
    r.iz = (int)(c % (unsigned)nz);
    const unsigned t = c / (unsigned)nz;
    r.iy = (int)(t % (unsigned)ny);
    r.ix = (int)(t / (unsigned)ny);
    return r;
}

__device__ __forceinline__ bool excluded(const PoissonGrid& g, unsigned c) {
    return (int)c == g.pin || (g.solid && g.solid[c]);
}

// Visits the six neighbours of free cell c: f(o) for coupled neighbours (fluid, not the
// pinned cell); returns the diagonal of B (coupled neighbours + the pinned one).
template <typename F>
__device__ __forceinline__ int for_neighbours(const PoissonGrid& g, unsigned c, Cell k, F&& f) {
    const unsigned sx = (unsigned)g.ny * g.nz, sy = (unsigned)g.nz;
    int diag = 0;
    auto nb = [&](unsigned o) {
        if (g.solid && g.solid[o]) return;          // zero-flux face, like a wall
        ++diag;
        if ((int)o != g.pin) f(o);                  // the pinned cell holds p = 0
    };
    if (k.ix > 0) nb(c - sx);
    if (k.ix < g.nx - 1) nb(c + sx);
    if (k.iy > 0) nb(c - sy);
    if (k.iy < g.ny - 1) nb(c + sy);
    if (k.iz > 0) nb(c - 1);
    if (k.iz < g.nz - 1) nb(c + 1);
    return diag;
}

// Net outflow of free cell c, summed over its six faces in the accumulation type A.  A face
// shared with a solid cell carries the solid's zero velocity whatever the array holds there
// (advection and buoyancy write every face), so the right-hand side matches the operator,
// whose rows drop solid neighbours, and the projected field is divergence-free next to solids.
template <typename A, typename T>
__device__ __forceinline__ A net_outflow(const PoissonGrid& g, unsigned c, Cell k, const T* __restrict__ u,
                                         const T* __restrict__ v, const T* __restrict__ w) {
    const int ny = g.ny, nz = g.nz;
    const unsigned sx = (unsigned)ny * nz;
    const unsigned u0 = c, u1 = c + sx;
    const unsigned v0 = ((unsigned)k.ix * (ny + 1) + k.iy) * nz + k.iz, v1 = v0 + nz;
    const unsigned w0 = ((unsigned)k.ix * ny + k.iy) * (nz + 1) + k.iz, w1 = w0 + 1;
    A fu0 = (A)u[u0], fu1 = (A)u[u1], fv0 = (A)v[v0], fv1 = (A)v[v1], fw0 = (A)w[w0], fw1 = (A)w[w1];
    if (g.solid) {
        if (k.ix > 0 && g.solid[c - sx]) fu0 = A(0);
        if (k.ix < g.nx - 1 && g.solid[c + sx]) fu1 = A(0);
        if (k.iy > 0 && g.solid[c - nz]) fv0 = A(0);
        if (k.iy < ny - 1 && g.solid[c + nz]) fv1 = A(0);
        if (k.iz > 0 && g.solid[c - 1]) fw0 = A(0);
        if (k.iz < nz - 1 && g.solid[c + 1]) fw1 = A(0);
    }
    return (fu1 - fu0) + (fv1 - fv0) + (fw1 - fw0);
}

template <typename T>
__device__ __forceinline__ T inv_count(int d) {
    return d > 0 ? T(1) / T(d) : T(0);
}

// ---------------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------------

// r = -b - B p (warm) or r = -b, p = 0; partials |b|^2 and |r|^2
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_rhs(PoissonGrid g, T h, const T* __restrict__ u,
                                                      const T* __restrict__ v, const T* __restrict__ w,
                                                      T* __restrict__ r, T* __restrict__ p, int warm, double* part) {
    const unsigned n = (unsigned)g.nx * g.ny * g.nz;
    const int ny = g.ny, nz = g.nz;
    DotAcc<T> bb, rr;
    for (unsigned c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        const Cell k = decode(c, ny, nz);
        T b = T(0), rc = T(0);
        if (!excluded(g, c)) {
            b = net_outflow<T>(g, c, k, u, v, w) * h;
            rc = -b;
            if (warm) {
                T s = T(0);
                const int diag = for_neighbours(g, c, k, [&](unsigned o) { s += p[o]; });
                rc -= T(diag) * p[c] - s;
            }
        }
        if (!warm) p[c] = T(0);
        r[c] = rc;
        bb.add(b, b);
        rr.add(rc, rc);
    }
    const double acc[2] = {bb.value(), rr.value()};
    block_sums<2>(acc, part);
}

// Final sums of nv partial rows into sums[0..nv).
__global__ void k_finish(const double* part, int nblocks, int nv, double* sums) {
    __shared__ double sh[4][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int q = 0; q < nv; ++q) {
        double s = 0.0;
        for (int b = threadIdx.x; b < nblocks; b += blockDim.x) s += part[b + nblocks * q];
        s = warp_sum(s);
        if (lane == 0) sh[q][wid] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 0; q < nv; ++q) {
            double t = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[q][w];
            sums[q] = t;
        }
    }
}

// z = r / diag(B); rz; solver scalars initialised by the last block
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_pcg_init(PoissonGrid g, const T* __restrict__ r, T* __restrict__ z,
                                                           double* scal, double threshold, double rr0, double* part,
                                                           unsigned* ticket) {
    const unsigned n = (unsigned)g.nx * g.ny * g.nz;
    DotAcc<T> rz;
    for (unsigned c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        T zc = T(0);
        if (!excluded(g, c)) {
            const int diag = for_neighbours(g, c, decode(c, g.ny, g.nz), [](unsigned) {});
            zc = r[c] * inv_count<T>(diag);
        }
        z[c] = zc;
        rz.add(r[c], zc);
    }
    const double acc[1] = {rz.value()};
    block_sums<1>(acc, part);
    if (last_block(ticket)) {
        const double t = block_total(part, gridDim.x, 0);
        if (threadIdx.x == 0) {
            scal[S_ALPHA] = 0.0; scal[S_BETA] = 0.0; scal[S_RZ] = t; scal[S_RR] = rr0;
            scal[S_THRESH] = threshold; scal[S_DONE] = rr0 <= threshold ? 1.0 : 0.0; scal[S_ITERS] = 0.0;
            scal[S_DQ] = 0.0;
            *ticket = 0;
        }
    }
}

// ---------------------------------------------------------------------------------
// per-iteration kernels, W consecutive cells of a z-line per thread and loop trip
// (float4 / double2 loads when nz is a multiple of W; W = 1 otherwise)
// ---------------------------------------------------------------------------------
template <typename T, int W>
__device__ __forceinline__ void ldv(const T* __restrict__ p, T (&v)[W]) {
    if constexpr (W == 4) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else if constexpr (W == 2) {
        const double2 t = *reinterpret_cast<const double2*>(p);
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = p[0];
    }
}
template <typename T, int W>
__device__ __forceinline__ void stv(T* __restrict__ p, const T (&v)[W]) {
    if constexpr (W == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else if constexpr (W == 2) *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
    else p[0] = v[0];
}

// warp sum of an accumulator, as one; lane 0 holds the total
__device__ __forceinline__ DotAcc<float> acc_warp(DotAcc<float> a) {
    for (int o = 16; o > 0; o >>= 1) {
        const float h2 = __shfl_down_sync(0xffffffffu, a.hi, o), l2 = __shfl_down_sync(0xffffffffu, a.lo, o);
        const float s = __fadd_rn(a.hi, h2);
        const float bb = __fsub_rn(s, a.hi);
        const float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(h2, bb));
        a.hi = s;
        a.lo = __fadd_rn(__fadd_rn(a.lo, l2), e);
    }
    return a;
}
__device__ __forceinline__ DotAcc<double> acc_warp(DotAcc<double> a) {
    a.s = warp_sum(a.s);
    return a;
}
template <typename T>
__device__ __forceinline__ double warp_total(const DotAcc<T>& a) { return acc_warp(a).value(); }

// block sums of NV accumulators into part[b + nb*q] (FP64 conversions only per warp)
template <typename T, int NV>
__device__ __forceinline__ void block_dots(const DotAcc<T> (&acc)[NV], double* part) {
    __shared__ double sh[NV][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        const double t = warp_total(acc[q]);
        if (lane == 0) sh[q][wid] = t;
    }
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            double v = lane < nw ? sh[q][lane] : 0.0;
            v = warp_sum(v);
            if (lane == 0) part[blockIdx.x + gridDim.x * q] = v;
        }
    }
}

// diagonal of B at cell c0 + e of a group (walls and solid neighbours removed)
template <int W>
__device__ __forceinline__ int diag_at(const PoissonGrid& g, unsigned c0, const Cell& k, int e) {
    const unsigned sx = (unsigned)g.ny * g.nz, sy = (unsigned)g.nz, c = c0 + e;
    int d = 0;
    auto nb = [&](bool ok, unsigned o) { if (ok && !(g.solid && g.solid[o])) ++d; };
    nb(k.ix > 0, c - sx);
    nb(k.ix < g.nx - 1, c + sx);
    nb(k.iy > 0, c - sy);
    nb(k.iy < g.ny - 1, c + sy);
    nb(e > 0 || k.iz > 0, c - 1);
    nb(e < W - 1 || k.iz + W < g.nz, c + 1);
    return d;
}

// d_new = z + beta d_old (d_new = z on the first iteration);  q = B d_new;
// alpha = rz / (d_new.q), or (d_new.r) / (d_new.q) when r is given (flexible CG: exact line
// search along d whatever the preconditioner did)
template <typename T, int W>
__global__ void __launch_bounds__(kRedThreads) k_cg_direction_apply(PoissonGrid g, double* __restrict__ scal,
                                                                     const T* __restrict__ z, const T* __restrict__ dold,
                                                                     T* __restrict__ dnew, T* __restrict__ q, int first,
                                                                     const T* __restrict__ rres, double* part,
                                                                     unsigned* ticket) {
    if (scal[S_DONE] != 0.0) return;
    const unsigned n = (unsigned)g.nx * g.ny * g.nz, ngr = n / W;
    const unsigned sx = (unsigned)g.ny * g.nz, sy = (unsigned)g.nz;
    const T beta = (T)scal[S_BETA];
    auto dvec = [&](unsigned o0, T (&o)[W]) {
        ldv<T, W>(z + o0, o);
        if (!first) {
            T b[W];
            ldv<T, W>(dold + o0, b);
#pragma unroll
            for (int e = 0; e < W; ++e) o[e] += beta * b[e];
        }
    };
    auto d1 = [&](unsigned o) -> T { return first ? z[o] : z[o] + beta * dold[o]; };
    DotAcc<T> acc[2];
    for (unsigned gi = blockIdx.x * blockDim.x + threadIdx.x; gi < ngr; gi += gridDim.x * blockDim.x) {
        const unsigned c0 = gi * W;
        const Cell k = decode(c0, g.ny, g.nz);
        T dc[W], s[W];
        int dg[W];
        dvec(c0, dc);
#pragma unroll
        for (int e = 0; e < W; ++e) { s[e] = T(0); dg[e] = 0; }
        auto side = [&](bool ok, unsigned o0) {
            if (!ok) return;
            T nv[W];
            dvec(o0, nv);
#pragma unroll
            for (int e = 0; e < W; ++e) {
                const unsigned o = o0 + e;
                if (g.solid && g.solid[o]) continue;
                ++dg[e];
                if ((int)o != g.pin) s[e] += nv[e];
            }
        };
        side(k.ix > 0, c0 - sx);
        side(k.ix < g.nx - 1, c0 + sx);
        side(k.iy > 0, c0 - sy);
        side(k.iy < g.ny - 1, c0 + sy);
#pragma unroll
        for (int e = 0; e < W; ++e) {
            const unsigned c = c0 + e;
            if (e > 0 || k.iz > 0) {
                const unsigned o = c - 1;
                if (!(g.solid && g.solid[o])) { ++dg[e]; if ((int)o != g.pin) s[e] += e > 0 ? dc[e - 1] : d1(o); }
            }
            if (e < W - 1 || k.iz + W < g.nz) {
                const unsigned o = c + 1;
                if (!(g.solid && g.solid[o])) { ++dg[e]; if ((int)o != g.pin) s[e] += e < W - 1 ? dc[e + 1] : d1(o); }
            }
        }
        T qv[W];
#pragma unroll
        for (int e = 0; e < W; ++e) {
            qv[e] = excluded(g, c0 + e) ? T(0) : T(dg[e]) * dc[e] - s[e];
            acc[0].add(dc[e], qv[e]);
        }
        stv<T, W>(dnew + c0, dc);
        stv<T, W>(q + c0, qv);
        if (rres) {
            T rv[W];
            ldv<T, W>(rres + c0, rv);
#pragma unroll
            for (int e = 0; e < W; ++e) acc[1].add(dc[e], rv[e]);
        }
    }
    block_dots<T, 2>(acc, part);
    if (last_block(ticket)) {
        double t[2] = {0.0, 0.0};
        if (rres) block_totals<2>(part, gridDim.x, t);
        else block_totals<1>(part, gridDim.x, reinterpret_cast<double (&)[1]>(t));
        if (threadIdx.x == 0) {
            const double num = rres ? t[1] : scal[S_RZ];
            scal[S_ALPHA] = t[0] != 0.0 ? num / t[0] : 0.0;
            scal[S_DQ] = t[0];
            *ticket = 0;
        }
    }
}

// r = rhs - B p on the free cells; partials |r|^2
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_residual(PoissonGrid g, const T* __restrict__ rhs,
                                                           const T* __restrict__ p, T* __restrict__ r, double* part) {
    const unsigned n = (unsigned)g.nx * g.ny * g.nz;
    DotAcc<T> rr;
    for (unsigned c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        T rc = T(0);
        if (!excluded(g, c)) {
            T s = T(0);
            const int diag = for_neighbours(g, c, decode(c, g.ny, g.nz), [&](unsigned o) { s += p[o]; });
            rc = rhs[c] - (T(diag) * p[c] - s);
        }
        r[c] = rc;
        rr.add(rc, rc);
    }
    const double acc[1] = {rr.value()};
    block_sums<1>(acc, part);
}

// x += alpha d; r -= alpha q; rr; with jacobi: z = r / diag, rz, beta = rz_new / rz_old.
template <typename T, int W>
__global__ void __launch_bounds__(kRedThreads) k_cg_update(PoissonGrid g, double* __restrict__ scal, T* __restrict__ x,
                                                            T* __restrict__ r, const T* __restrict__ d,
                                                            const T* __restrict__ q, T* __restrict__ z, int jacobi,
                                                            double* part, unsigned* ticket) {
    if (scal[S_DONE] != 0.0) return;
    const unsigned n = (unsigned)g.nx * g.ny * g.nz, ngr = n / W;
    const T a = (T)scal[S_ALPHA];
    DotAcc<T> acc[2];   // rz, rr
    for (unsigned gi = blockIdx.x * blockDim.x + threadIdx.x; gi < ngr; gi += gridDim.x * blockDim.x) {
        const unsigned c0 = gi * W;
        T xv[W], dv[W], rv[W], qv[W];
        ldv<T, W>(x + c0, xv); ldv<T, W>(d + c0, dv); ldv<T, W>(r + c0, rv); ldv<T, W>(q + c0, qv);
#pragma unroll
        for (int e = 0; e < W; ++e) {
            xv[e] += a * dv[e];
            rv[e] -= a * qv[e];
            acc[1].add(rv[e], rv[e]);
        }
        stv<T, W>(x + c0, xv);
        stv<T, W>(r + c0, rv);
        if (jacobi) {
            const Cell k = decode(c0, g.ny, g.nz);
            T zv[W];
#pragma unroll
            for (int e = 0; e < W; ++e) {
                zv[e] = excluded(g, c0 + e) ? T(0) : rv[e] * inv_count<T>(diag_at<W>(g, c0, k, e));
                acc[0].add(rv[e], zv[e]);
            }
            stv<T, W>(z + c0, zv);
        }
    }
    block_dots<T, 2>(acc, part);
    if (last_block(ticket)) {
        double t[2];
        block_totals<2>(part, gridDim.x, t);
        if (threadIdx.x == 0) {
            if (jacobi) {
                scal[S_BETA] = scal[S_RZ] != 0.0 ? t[0] / scal[S_RZ] : 0.0;
                scal[S_RZ] = t[0];
            }
            scal[S_RR] = t[1];
            scal[S_ITERS] += 1.0;
            if (t[1] <= scal[S_THRESH]) scal[S_DONE] = 1.0;
            *ticket = 0;
        }
    }
}

// ---------------------------------------------------------------------------------
// Jacobi-PCG as one kernel
// ---------------------------------------------------------------------------------
// Many iterations per launch (cooperative; the blocks meet twice an iteration).  Block b owns the
// cells [b chunk, (b + 1) chunk) in linear order and keeps d of them, and of one z-line on either
// side, in shared memory; q, r and x of them too as far as they fit (NS arrays of the four).
// Along y and z the operator reads shared memory; along x the neighbour's d = z + beta d_old is
// formed from the z and d_old that its block stored before the last meeting, as in
// k_cg_direction_apply.  The arithmetic on the vectors is that of the two kernels above, cell by
// cell, and its dots are float pairs within a warp and FP64 from there on, as theirs; only their order
// differs.
//
// What an iteration costs is latency: FP64 operations run in one thread or one warp (one of every
// thread of a block takes a quarter of a microsecond), the neighbours' loads are issued before the
// block's own cells are updated, and what a group of cells needs of its place in the grid is one word,
// made once.  Microseconds an iteration, with the two kernels above and with this one: FP32 16^3 18 ->
// 7.1, 64^3 23 -> 10.2, 128^3 36 -> 18.2, 160^3 53 -> 48; FP64 64^3 46 -> 17.7, 128^3 134 -> 81.  (Slots
// polled by every block, with the meeting's number beside the value instead of a counter, were slower:
// 19.8 against 14 us at 64^3.)
// Rows that are no whole groups take one cell a step, and from 4096 cells a block on their places are formed
// at each visit: 127^3 49 -> 41, 141^3 61 -> 55; FP64 127^3 133 -> 82.  In FP32 they need three shared
// arrays: with two the two kernels are as fast (143^3 to 161^3 within 2%).
// Larger grids, whose chunks leave no room for two shared arrays, keep the two kernels: there the
// vectors' traffic is the time (256^3: 152 us for 11 vectors of 67 MB, 108 us at the copy rate).
constexpr int kPcgThreadsMax = 1024;
constexpr int kPcgIters = 256;           // iterations per launch
constexpr int kPcgSpinLimit = 1 << 21;   // polls of a meeting before the kernel gives up
constexpr unsigned kPcgStuck = 1u << 30; // set in the counter when one did
constexpr size_t kPcgSmem = 224 * 1024;  // dynamic shared memory of a block (227 KB less the static part)
constexpr int kPcgPartWords = 3;         // doubles a block: one sum, then two
constexpr int kPcgBlocksMax = 1024;
// SMs left to other kernels.  A cooperative launch starts when all of its blocks find room, and a block of
// this kernel shares an SM with nothing that runs there already (its shared memory is another split of
// L1).  With blocks on all 152 SMs one small kernel of another stream, however long it ran, held the
// call up: 1.2 s beside a one-thread kernel of 1.2 s.  Costs 1 to 2% from 128^3 on (128^3 17.8 -> 18.1 us,
// FP64 79.8 -> 81.7).
constexpr int kPcgLeave = 4;
constexpr unsigned kPcgOneBlock = 1024;  // groups that one block takes alone

template <typename T>
struct PcgArgs {
    PoissonGrid g;
    T *x, *r, *z, *d0, *d1;
    double* scal;
    double* parts;               // kPcgPartWords * gridDim.x
    unsigned* bar;               // arrivals, zero at launch
    unsigned chunk;              // cells per block, a multiple of W
    int iters;                   // at most this many iterations
    int first;                   // no direction yet
};

template <typename T, int W>
__device__ __forceinline__ void ldcgv(const T* p, T (&v)[W]) {
    if constexpr (W == 4) {
        const float4 t = __ldcg(reinterpret_cast<const float4*>(p));
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else if constexpr (W == 2) {
        const double2 t = __ldcg(reinterpret_cast<const double2*>(p));
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = __ldcg(p);
    }
}

// Place of a group of W cells: bits 0-5 the neighbours inside the grid (x-, x+, y-, y+, z- of the
// first cell, z+ of the last), then 3 bits a cell: the diagonal of B, 7 where the cell is
// excluded.  Excluded cells need no further care: their z and d are zero.
template <int W>
__device__ __forceinline__ unsigned pcg_place(const PoissonGrid& g, unsigned c) {
    const Cell k = decode(c, g.ny, g.nz);
    unsigned p = (k.ix > 0) | (k.ix < g.nx - 1) << 1 | (k.iy > 0) << 2 | (k.iy < g.ny - 1) << 3 | (k.iz > 0) << 4 |
                 (k.iz + W < g.nz) << 5;
#pragma unroll
    for (int e = 0; e < W; ++e) p |= (excluded(g, c + e) ? 7u : (unsigned)diag_at<W>(g, c, k, e)) << (6 + 3 * e);
    return p;
}

// All blocks meet: publishes the block's NV sums of its threads' accumulators and returns their
// sums over the blocks in tot[] (thread 0; every block adds them up in the same order).  What the
// block's threads stored to global memory before is visible to every block after (loads past L1).
// FP64 from the warps' sums on, as block_dots; by one warp a sum, which has the blocks' sums in flight
// together.  parts: NV doubles a block, not those of the meeting before.  False when the wait ran out.
template <typename T, int NV>
__device__ __forceinline__ bool pcg_meet(const DotAcc<T> (&acc)[NV], double* parts, unsigned* bar, unsigned target,
                                         double* tot) {
    __shared__ DotAcc<T> sh[NV][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, nb = gridDim.x;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        const DotAcc<T> t = acc_warp(acc[q]);
        if (lane == 0) sh[q][warp] = t;
    }
    __syncthreads();
    bool ok = true;
    if (warp == 0) {
        double t[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) t[q] = lane < nw ? sh[q][lane].value() : 0.0;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            if (nw > 16) t[q] += __shfl_down_sync(0xffffffffu, t[q], 16);
            for (int o = 8; o > 0; o >>= 1) t[q] += __shfl_down_sync(0xffffffffu, t[q], o);
        }
        if (lane == 0) {
            if (nb == 1) {
#pragma unroll
                for (int q = 0; q < NV; ++q) tot[q] = t[q];
            } else {
#pragma unroll
                for (int q = 0; q < NV; ++q) __stcg(parts + (size_t)q * nb + blockIdx.x, t[q]);
                unsigned seen;
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
                int it = 0;
                do {
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
                } while (seen < target && ++it < kPcgSpinLimit);
                ok = seen >= target && seen < kPcgStuck;
                if (!ok) atomicOr(bar, kPcgStuck);   // the others leave at once
            }
        }
    }
    if (nb == 1) return true;
    if (!__syncthreads_and(ok)) return false;
    if (warp < NV) {
        constexpr int kAhead = 5;   // loads in flight: all of 152 blocks
        double t = 0.0;
        for (int b0 = lane; b0 < nb; b0 += 32 * kAhead) {
            double v[kAhead];
#pragma unroll
            for (int j = 0; j < kAhead; ++j) v[j] = b0 + 32 * j < nb ? __ldcg(parts + (size_t)warp * nb + b0 + 32 * j) : 0.0;
#pragma unroll
            for (int j = 0; j < kAhead; ++j) t += v[j];
        }
        t = warp_sum(t);
        if (lane == 0) tot[warp] = t;
    }
    __syncthreads();
    return true;
}

// G > 0: at most G groups a thread, their places in registers; 0: any number, placed as visited
template <typename T, int W, int NS, int G>
__global__ void __launch_bounds__(kPcgThreadsMax) k_pcg(PcgArgs<T> A) {
    extern __shared__ __align__(16) unsigned char pcg_smem[];
    __shared__ double tot[2];
    __shared__ T step;      // alpha, then beta
    __shared__ int done;
    __shared__ T inv[8];    // 1 / diagonal, 0 for excluded cells
    const PoissonGrid g = A.g;
    const unsigned n = (unsigned)g.nx * g.ny * g.nz, sx = (unsigned)g.ny * g.nz, sy = (unsigned)g.nz;
    const unsigned c0 = blockIdx.x * A.chunk, c1 = min(n, c0 + A.chunk);
    // shared cells [lo, hi): the chunk and a z-line either side (nz is a multiple of W)
    const unsigned lo = c0 > sy ? c0 - sy : 0u, hi = min(n, c1 + sy);
    T* sd = reinterpret_cast<T*>(pcg_smem);
    T* own = sd + A.chunk + 2 * sy;
    T* const sq = own;
    T* const r = NS >= 3 ? own + A.chunk : A.r + c0;
    T* const x = NS >= 4 ? own + 2 * (size_t)A.chunk : A.x + c0;
    if (A.scal[S_DONE] != 0.0) return;
    double rz = 0.0, beta_d = 0.0, rr = 0.0, its = 0.0, threshold = 0.0;   // thread 0
    if (threadIdx.x == 0) {
        rz = A.scal[S_RZ]; beta_d = A.scal[S_BETA]; rr = A.scal[S_RR]; its = A.scal[S_ITERS];
        threshold = A.scal[S_THRESH];
        step = (T)beta_d;
        done = 0;
    }
    if (threadIdx.x < 8) inv[threadIdx.x] = threadIdx.x < 7 ? inv_count<T>((int)threadIdx.x) : T(0);
    T* dold = A.d0;
    T* dnew = A.d1;
    const unsigned cstep = blockDim.x * W, cfirst = c0 + threadIdx.x * W;
    unsigned places[G > 0 ? G : 1];
    // f(cell, place) for every group of this thread
    auto each = [&](auto&& f) {
        if constexpr (G > 0) {
#pragma unroll
            for (int i = 0; i < G; ++i) {
                const unsigned c = cfirst + i * cstep;
                if (c < c1) f(c, places[i]);
            }
        } else {
            for (unsigned c = cfirst; c < c1; c += cstep) f(c, pcg_place<W>(g, c));
        }
    };
    if constexpr (G > 0) {
#pragma unroll
        for (int i = 0; i < G; ++i) {
            const unsigned c = cfirst + i * cstep;
            places[i] = c < c1 ? pcg_place<W>(g, c) : 0u;
        }
    }
    for (unsigned c = cfirst; c < c1; c += cstep) {
        T v[W];
        if (NS >= 3) { ldv<T, W>(A.r + c, v); stv<T, W>(r + (c - c0), v); }
        if (NS >= 4) { ldv<T, W>(A.x + c, v); stv<T, W>(x + (c - c0), v); }
        if (!A.first) { ldv<T, W>(dold + c, v); stv<T, W>(sd + (c - lo), v); }
    }
    __syncthreads();
    bool first = A.first != 0;
    unsigned target = 0;
    for (int it = 0; it < A.iters && !done; ++it) {
        const T beta = step;
        // d of another block's group
        auto far = [&](unsigned o, T (&v)[W]) {
            ldcgv<T, W>(A.z + o, v);
            if (!first) {
                T b[W];
                ldcgv<T, W>(dold + o, b);
#pragma unroll
                for (int e = 0; e < W; ++e) v[e] = fma(beta, b[e], v[e]);
            }
        };
        auto near = [&](unsigned o) { return o >= lo && o < hi; };
        // x-neighbours' part of the operator's sum; `late`: taken after the block's d are in place
        auto xsum = [&](unsigned c, unsigned p, bool late, T (&s)[W]) {
            const bool xm = p & 1u, xp = p & 2u;
            const bool wait = (xm && near(c - sx)) || (xp && near(c + sx));
            if (wait != late) return wait;
            T a[W], b[W];
#pragma unroll
            for (int e = 0; e < W; ++e) { a[e] = T(0); b[e] = T(0); }
            if (xm) { if (near(c - sx)) ldv<T, W>(sd + (c - sx - lo), a); else far(c - sx, a); }
            if (xp) { if (near(c + sx)) ldv<T, W>(sd + (c + sx - lo), b); else far(c + sx, b); }
#pragma unroll
            for (int e = 0; e < W; ++e) s[e] = a[e] + b[e];
            return wait;
        };
        // the z-lines either side
        for (unsigned i = threadIdx.x * W; i < (c0 - lo) + (hi - c1); i += cstep) {
            const unsigned c = i < c0 - lo ? lo + i : c1 + (i - (c0 - lo));
            T v[W];
            far(c, v);
            stv<T, W>(sd + (c - lo), v);
        }
        // d = z + beta d_old, with z = r / diag as it was stored
        each([&](unsigned c, unsigned p) {
            T v[W], o[W], s[W];
            if (!xsum(c, p, false, s)) stv<T, W>(sq + (c - c0), s);
            ldv<T, W>(r + (c - c0), v);
            if (!first) ldv<T, W>(sd + (c - lo), o);
#pragma unroll
            for (int e = 0; e < W; ++e) {
                v[e] *= inv[(p >> (6 + 3 * e)) & 7u];
                if (!first) v[e] = fma(beta, o[e], v[e]);
            }
            stv<T, W>(sd + (c - lo), v);
            stv<T, W>(dnew + c, v);
        });
        __syncthreads();
        // q = B d
        DotAcc<T> dq[1];
        each([&](unsigned c, unsigned p) {
            T dc[W], s[W], a[W], b[W], q[W];
            if (!xsum(c, p, true, s)) ldv<T, W>(sq + (c - c0), s);
            ldv<T, W>(sd + (c - lo), dc);
#pragma unroll
            for (int e = 0; e < W; ++e) { a[e] = T(0); b[e] = T(0); }
            if (p & 4u) ldv<T, W>(sd + (c - sy - lo), a);
            if (p & 8u) ldv<T, W>(sd + (c + sy - lo), b);
            const T zm = p & 16u ? sd[c - 1 - lo] : T(0), zp = p & 32u ? sd[c + W - lo] : T(0);
#pragma unroll
            for (int e = 0; e < W; ++e) {
                s[e] += a[e];
                s[e] += b[e];
                s[e] += e > 0 ? dc[e > 0 ? e - 1 : 0] : zm;
                s[e] += e < W - 1 ? dc[e < W - 1 ? e + 1 : 0] : zp;
                const unsigned dg = (p >> (6 + 3 * e)) & 7u;
                q[e] = dg == 7u ? T(0) : fma(T((int)dg), dc[e], -s[e]);
                dq[0].add(dc[e], q[e]);
            }
            stv<T, W>(sq + (c - c0), q);
        });
        if (!pcg_meet<T, 1>(dq, A.parts, A.bar, target += gridDim.x, tot)) break;
        if (threadIdx.x == 0) step = (T)(tot[0] != 0.0 ? rz / tot[0] : 0.0);
        __syncthreads();
        const T al = step;
        DotAcc<T> acc[2];   // r.z, r.r
        each([&](unsigned c, unsigned p) {
            T xv[W], dv[W], rv[W], qv[W], zv[W];
            ldv<T, W>(x + (c - c0), xv); ldv<T, W>(sd + (c - lo), dv);
            ldv<T, W>(r + (c - c0), rv); ldv<T, W>(sq + (c - c0), qv);
#pragma unroll
            for (int e = 0; e < W; ++e) {
                xv[e] = fma(al, dv[e], xv[e]);
                rv[e] = fma(-al, qv[e], rv[e]);
                zv[e] = rv[e] * inv[(p >> (6 + 3 * e)) & 7u];
            }
            stv<T, W>(A.z + c, zv);
            stv<T, W>(x + (c - c0), xv);
            stv<T, W>(r + (c - c0), rv);
#pragma unroll
            for (int e = 0; e < W; ++e) {
                acc[1].add(rv[e], rv[e]);
                acc[0].add(rv[e], zv[e]);
            }
        });
        if (!pcg_meet<T, 2>(acc, A.parts + gridDim.x, A.bar, target += gridDim.x, tot)) break;
        if (threadIdx.x == 0) {
            beta_d = rz != 0.0 ? tot[0] / rz : 0.0;
            rz = tot[0];
            rr = tot[1];
            its += 1.0;
            step = (T)beta_d;
            done = rr <= threshold;
        }
        __syncthreads();
        T* t = dold; dold = dnew; dnew = t;
        first = false;
    }
    for (unsigned c = cfirst; c < c1; c += cstep) {
        T v[W];
        if (NS >= 3) { ldv<T, W>(r + (c - c0), v); stv<T, W>(A.r + c, v); }
        if (NS >= 4) { ldv<T, W>(x + (c - c0), v); stv<T, W>(A.x + c, v); }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        A.scal[S_BETA] = beta_d; A.scal[S_RZ] = rz; A.scal[S_RR] = rr; A.scal[S_ITERS] = its;
        if (done) A.scal[S_DONE] = 1.0;
    }
}

// flexible CG with m kept directions (Notay's FCG(m)):
//   beta_j = -(z.q_j)/(d_j.q_j) for the kept directions j;  d = z + sum_j beta_j d_j;
//   q = B d;  alpha = (d.r)/(d.q)
template <typename T>
struct DirSet {
    const T* v[kFcgMaxDirs];
    int slot[kFcgMaxDirs];
    int n;
};

// The number NQ of kept directions is a template argument: tested inside the loop it keeps each
// vector's load behind the test.  Bound by HBM: 67 MB a vector at 256^3, ten vectors with eight
// directions (floor 99 us).  Copied to the thread's own shared slots, two groups of all vectors are in
// flight (kDotsSmem; 2 CTAs per SM): 134 us, 139 with the loads in registers, a few at a time.
constexpr int kDotsStages = 2;
template <typename T, int W, int NQ>
constexpr int kDotsSmem = W * sizeof(T) == 16 ? kDotsStages * (NQ + 2) * kRedThreads * 16 : 0;
template <typename T, int W, int NQ>
__global__ void __launch_bounds__(kRedThreads) k_fcgm_dots(unsigned n, double* __restrict__ scal, const T* __restrict__ z,
                                                            const T* __restrict__ r, DirSet<T> qs, double* part,
                                                            unsigned* ticket) {
    if (scal[S_DONE] != 0.0) return;
    const unsigned ngr = n / W, step = gridDim.x * blockDim.x, g0 = blockIdx.x * blockDim.x + threadIdx.x;
    DotAcc<T> acc[NQ + 1];   // z.q_j, then z.r
    auto vec = [&](int v) { return v == 0 ? z : (v == 1 ? r : qs.v[v < 2 ? 0 : v - 2]); };
    auto add = [&](const T (&zv)[W], const T (&v)[W], int j) {
#pragma unroll
        for (int e = 0; e < W; ++e) acc[j].add(zv[e], v[e]);
    };
    if constexpr (W * sizeof(T) == 16) {
        extern __shared__ __align__(16) unsigned char dots_smem[];
        unsigned char* mine = dots_smem + threadIdx.x * 16;
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(mine);
        auto slot = [](int stage, int v) { return (stage * (NQ + 2) + v) * (kRedThreads * 16); };
        auto issue = [&](unsigned gi, int stage) {
            if (gi < ngr)
#pragma unroll
                for (int v = 0; v < NQ + 2; ++v)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(base + slot(stage, v)),
                                 "l"(vec(v) + (size_t)gi * W)
                                 : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int k = 0; k < kDotsStages; ++k) issue(g0 + k * step, k);
        int stage = 0;
        for (unsigned gi = g0; gi < ngr; gi += step) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kDotsStages - 1) : "memory");
            T zv[W], v[W];
            ldv<T, W>(reinterpret_cast<const T*>(mine + slot(stage, 0)), zv);
#pragma unroll
            for (int j = 0; j < NQ; ++j) {
                ldv<T, W>(reinterpret_cast<const T*>(mine + slot(stage, 2 + j)), v);
                add(zv, v, j);
            }
            ldv<T, W>(reinterpret_cast<const T*>(mine + slot(stage, 1)), v);
            add(zv, v, NQ);
            issue(gi + kDotsStages * step, stage);
            stage = stage + 1 == kDotsStages ? 0 : stage + 1;
        }
    } else {
        for (unsigned gi = g0; gi < ngr; gi += step) {
            T zv[W], v[W];
            ldv<T, W>(z + gi * W, zv);
#pragma unroll
            for (int j = 0; j <= NQ; ++j) {
                ldv<T, W>((j < NQ ? qs.v[j < NQ ? j : 0] : r) + gi * W, v);
                add(zv, v, j);
            }
        }
    }
    block_dots<T, NQ + 1>(acc, part);
    if (last_block(ticket)) {
        double t[NQ + 1];
        block_totals<NQ + 1>(part, gridDim.x, t);
        if (threadIdx.x == 0) {
#pragma unroll
            for (int j = 0; j < NQ; ++j) {
                const double dq = scal[S_DQJ + qs.slot[j]];
                scal[S_BETAJ + qs.slot[j]] = dq != 0.0 ? -t[j] / dq : 0.0;
            }
            scal[S_RZ] = t[NQ];
            *ticket = 0;
        }
    }
}

// d_new = z + sum_j beta_j d_j (streamed once; the stencil kernel below then reads d_new
// instead of recomputing it for each neighbour)
template <typename T, int W, int NQ>
__global__ void __launch_bounds__(kRedThreads) k_fcgm_combine(unsigned n, const double* __restrict__ scal,
                                                               const T* __restrict__ z, DirSet<T> ds,
                                                               T* __restrict__ dnew) {
    if (scal[S_DONE] != 0.0) return;
    const unsigned ngr = n / W;
    T beta[NQ + 1];
#pragma unroll
    for (int j = 0; j < NQ; ++j) beta[j] = (T)scal[S_BETAJ + ds.slot[j]];
    for (unsigned gi = blockIdx.x * blockDim.x + threadIdx.x; gi < ngr; gi += gridDim.x * blockDim.x) {
        const unsigned c0 = gi * W;
        T o[W], b[NQ + 1][W];
        ldv<T, W>(z + c0, o);
#pragma unroll
        for (int j = 0; j < NQ; ++j) ldv<T, W>(ds.v[j] + c0, b[j]);
#pragma unroll
        for (int j = 0; j < NQ; ++j)
#pragma unroll
            for (int e = 0; e < W; ++e) o[e] += beta[j] * b[j][e];
        stv<T, W>(dnew + c0, o);
    }
}

// q = B d;  d.q and d.r; the last block sets alpha = d.r / d.q.  The neighbours outside the grid
// are read at the cell itself and not added, so that a group's loads wait for no test: 55 us at 256^3,
// 117 with each behind its test (floor 30: d, r and q).
template <typename T, int W, bool SOLID>
__global__ void __launch_bounds__(kRedThreads) k_fcgm_apply(PoissonGrid g, double* __restrict__ scal,
                                                             const T* __restrict__ d, T* __restrict__ qnew, int newslot,
                                                             const T* __restrict__ rres, double* part, unsigned* ticket) {
    if (scal[S_DONE] != 0.0) return;
    const unsigned n = (unsigned)g.nx * g.ny * g.nz, ngr = n / W;
    const unsigned sx = (unsigned)g.ny * g.nz, sy = (unsigned)g.nz;
    const int pin = g.pin;
    auto solid = [&](unsigned o) { return SOLID && g.solid[o] != 0; };
    DotAcc<T> acc[2];
    for (unsigned gi = blockIdx.x * blockDim.x + threadIdx.x; gi < ngr; gi += gridDim.x * blockDim.x) {
        const unsigned c0 = gi * W;
        const Cell k = decode(c0, g.ny, g.nz);
        const bool in[6] = {k.ix > 0, k.ix < g.nx - 1, k.iy > 0, k.iy < g.ny - 1, k.iz > 0, k.iz + W < g.nz};
        const unsigned at[4] = {in[0] ? c0 - sx : c0, in[1] ? c0 + sx : c0, in[2] ? c0 - sy : c0, in[3] ? c0 + sy : c0};
        T dc[W], rv[W], nv[4][W], s[W];
        int dg[W];
        ldv<T, W>(d + c0, dc);
#pragma unroll
        for (int m = 0; m < 4; ++m) ldv<T, W>(d + at[m], nv[m]);
        const T zl = d[in[4] ? c0 - 1 : c0], zr = d[in[5] ? c0 + W : c0];
        ldv<T, W>(rres + c0, rv);
#pragma unroll
        for (int e = 0; e < W; ++e) { s[e] = T(0); dg[e] = 0; }
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int e = 0; e < W; ++e)
                if (in[m] && !solid(at[m] + e)) {
                    ++dg[e];
                    if ((int)(at[m] + e) != pin) s[e] += nv[m][e];
                }
        T qv[W];
#pragma unroll
        for (int e = 0; e < W; ++e) {
            const unsigned c = c0 + e;
            if ((e > 0 || in[4]) && !solid(c - 1)) {
                ++dg[e];
                if ((int)(c - 1) != pin) s[e] += e > 0 ? dc[e > 0 ? e - 1 : 0] : zl;
            }
            if ((e < W - 1 || in[5]) && !solid(c + 1)) {
                ++dg[e];
                if ((int)(c + 1) != pin) s[e] += e < W - 1 ? dc[e < W - 1 ? e + 1 : 0] : zr;
            }
            qv[e] = (int)c == pin || solid(c) ? T(0) : T(dg[e]) * dc[e] - s[e];
            acc[0].add(dc[e], qv[e]);
            acc[1].add(dc[e], rv[e]);
        }
        stv<T, W>(qnew + c0, qv);
    }
    block_dots<T, 2>(acc, part);
    if (last_block(ticket)) {
        double t[2];
        block_totals<2>(part, gridDim.x, t);
        if (threadIdx.x == 0) {
            scal[S_ALPHA] = t[0] != 0.0 ? t[1] / t[0] : 0.0;
            scal[S_DQJ + newslot] = t[0];
            *ticket = 0;
        }
    }
}

__global__ void k_fcg_begin(double* scal, double threshold, double rr0) {
    scal[S_ALPHA] = 0.0; scal[S_BETA] = 0.0; scal[S_RZ] = 0.0; scal[S_RR] = rr0;
    scal[S_THRESH] = threshold; scal[S_DONE] = rr0 <= threshold ? 1.0 : 0.0; scal[S_ITERS] = 0.0; scal[S_DQ] = 0.0;
}

// u -= (p_i - p_{i-1}) / h on faces between two fluid cells (calc_pressure_3d.cpp:196-232);
// faces touching a solid cell are set to the solid's (zero) velocity.
template <typename T, typename P>
__global__ void k_subtract_gradient(PoissonGrid g, P invh, const P* __restrict__ p, T* __restrict__ u,
                                    T* __restrict__ v, T* __restrict__ w) {
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const unsigned nu = (unsigned)(nx + 1) * ny * nz, nv = (unsigned)nx * (ny + 1) * nz;
    const unsigned nw = (unsigned)nx * ny * (nz + 1);
    const unsigned tot = nu + nv + nw;
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += gridDim.x * blockDim.x) {
        T* f; unsigned i, c, cm; bool interior;
        if (t < nu) {
            i = t; f = u;
            const Cell k = decode(i, ny, nz);
            interior = k.ix >= 1 && k.ix < nx;
            c = ((unsigned)k.ix * ny + k.iy) * nz + k.iz; cm = c - (unsigned)ny * nz;
        } else if (t < nu + nv) {
            i = t - nu; f = v;
            const Cell k = decode(i, ny + 1, nz);
            interior = k.iy >= 1 && k.iy < ny;
            c = ((unsigned)k.ix * ny + k.iy) * nz + k.iz; cm = c - nz;
        } else {
            i = t - nu - nv; f = w;
            const Cell k = decode(i, ny, nz + 1);
            interior = k.iz >= 1 && k.iz < nz;
            c = ((unsigned)k.ix * ny + k.iy) * nz + k.iz; cm = c - 1;
        }
        if (!interior) continue;
        if (g.solid && (g.solid[c] || g.solid[cm])) f[i] = T(0);
        else f[i] = (T)((P)f[i] - (p[c] - p[cm]) * invh);
    }
}

// wall momentum loss tallies (calc_pressure_3d.cpp:235-268)
template <typename T>
__global__ void k_wall_loss(int nx, int ny, int nz, double h, const T* __restrict__ p, double* part) {
    double acc[3] = {0.0, 0.0, 0.0};
    const long long nyz = (long long)ny * nz, nxz = (long long)nx * nz, nxy = (long long)nx * ny;
    const long long tot = nyz + nxz + nxy;
    const double h2 = h * h;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += (long long)gridDim.x * blockDim.x) {
        if (t < nyz) {
            const int iy = (int)(t / nz), iz = (int)(t % nz);
            acc[0] += -(double)p[((long long)0 * ny + iy) * nz + iz] * h2 + (double)p[((long long)(nx - 1) * ny + iy) * nz + iz] * h2;
        } else if (t < nyz + nxz) {
            const long long s = t - nyz;
            const int ix = (int)(s / nz), iz = (int)(s % nz);
            acc[1] += -(double)p[((long long)ix * ny + 0) * nz + iz] * h2 + (double)p[((long long)ix * ny + ny - 1) * nz + iz] * h2;
        } else {
            const long long s = t - nyz - nxz;
            const int ix = (int)(s / ny), iy = (int)(s % ny);
            acc[2] += -(double)p[((long long)ix * ny + iy) * nz + 0] * h2 + (double)p[((long long)ix * ny + iy) * nz + nz - 1] * h2;
        }
    }
    block_sums<3>(acc, part);
}

// ---------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------
template <typename T> struct VecW;
template <> struct VecW<float> { static constexpr int W = 4; };
template <> struct VecW<double> { static constexpr int W = 2; };

template <typename T>
void launch_direction(const PressureWork<T>& W, const PoissonGrid& g, const T* dold, T* dnew, bool first, const T* rres,
                      double* part, unsigned* ticket, cudaStream_t s) {
    constexpr int V = VecW<T>::W;
    if (g.nz % V == 0)
        k_cg_direction_apply<T, V><<<kRedBlocks, kRedThreads, 0, s>>>(g, W.scal, W.z, dold, dnew, W.q, first ? 1 : 0,
                                                                       rres, part, ticket);
    else
        k_cg_direction_apply<T, 1><<<kRedBlocks, kRedThreads, 0, s>>>(g, W.scal, W.z, dold, dnew, W.q, first ? 1 : 0,
                                                                       rres, part, ticket);
}

template <typename T>
void launch_update(const PressureWork<T>& W, const PoissonGrid& g, const T* d, bool jacobi, double* part,
                   unsigned* ticket, cudaStream_t s, const T* q = nullptr) {
    constexpr int V = VecW<T>::W;
    if (!q) q = W.q;
    if (g.nz % V == 0)
        k_cg_update<T, V><<<kRedBlocks, kRedThreads, 0, s>>>(g, W.scal, W.p, W.r, d, q, W.z, jacobi ? 1 : 0, part,
                                                              ticket);
    else
        k_cg_update<T, 1><<<kRedBlocks, kRedThreads, 0, s>>>(g, W.scal, W.p, W.r, d, q, W.z, jacobi ? 1 : 0, part,
                                                              ticket);
}
template <typename T>
cudaError_t pressure_rhs(const PressureWork<T>& W, const PoissonGrid& g, double h, const T* u, const T* v,
                         const T* w, bool warm, double* bb_rr_host, cudaStream_t s) {
    k_rhs<T><<<kRedBlocks, kRedThreads, 0, s>>>(g, (T)h, u, v, w, W.r, W.p, warm ? 1 : 0, W.part);
    k_finish<<<1, 256, 0, s>>>(W.part, kRedBlocks, 2, W.sums);
    cudaMemcpyAsync(bb_rr_host, W.sums, 2 * sizeof(double), cudaMemcpyDeviceToHost, s);
    return cudaStreamSynchronize(s);
}

// Blocks, threads and shared arrays of k_pcg for a grid, or none (blocks 0: too large a chunk for
// two shared arrays, or no cooperative launch).
struct PcgPlan {
    int blocks = 0, threads = 0, arrays = 0;
    bool placed = false;    // groups' places in registers
    unsigned chunk = 0;
    size_t smem = 0;
};
template <typename T>
constexpr int pcg_least_arrays(int W) { return sizeof(T) == 4 && W == 1 ? 3 : 2; }
template <typename T>
PcgPlan pcg_plan(const PoissonGrid& g) {
    PcgPlan p;
    int dev = 0, sms = 0, coop = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
        return p;
    sms = std::min(std::max(1, sms - kPcgLeave), kPcgBlocksMax);
    const unsigned n = (unsigned)g.nx * g.ny * g.nz, W = g.nz % VecW<T>::W == 0 ? VecW<T>::W : 1, groups = n / W;
    // 512 groups a block in FP32, 256 in FP64 (64^3 FP32 10.7 against 11.2 us an iteration with 256;
    // 20^3 FP64 11.6 against 13.9 with 512)
    const unsigned least = sizeof(T) == 4 ? 512 : 256;
    unsigned blocks = groups <= kPcgOneBlock ? 1u : std::min<unsigned>((unsigned)sms, (groups + least - 1) / least);
    const unsigned chunk = (groups + blocks - 1) / blocks * W;
    blocks = (n + chunk - 1) / chunk;
    for (int a = 4; a >= pcg_least_arrays<T>(W); --a) {
        const size_t smem = ((size_t)a * chunk + 2 * (size_t)g.nz) * sizeof(T);
        if (smem > kPcgSmem) continue;
        p.blocks = (int)blocks;
        // a thread a group; two where there are many in FP64, whose sums across a warp cost most
        // (64^3 18.4 against 20.2 us an iteration), and in one block (16^3 FP32 4.8 against 5.1)
        const unsigned per = (sizeof(T) == 8 || blocks == 1) && chunk / W > 512 ? 2 : 1;
        p.threads = (int)std::min<unsigned>(kPcgThreadsMax, std::max<unsigned>(128u, (chunk / W / per + 31) / 32 * 32));
        p.placed = chunk / W <= 4u * p.threads;
        p.arrays = a; p.chunk = chunk; p.smem = smem;
        return p;
    }
    return p;
}

template <typename T, int W, int NS, int G>
cudaError_t launch_pcg_t(const PcgPlan& p, PcgArgs<T> A, cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute(k_pcg<T, W, NS, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPcgSmem);
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pcg<T, W, NS, G>, p.threads, p.smem);
    if (e == cudaSuccess && per_sm < 1) e = cudaErrorCooperativeLaunchTooLarge;
    if (e != cudaSuccess) return e;
    void* args[] = {&A};
    return cudaLaunchCooperativeKernel((const void*)k_pcg<T, W, NS, G>, dim3(p.blocks), dim3(p.threads), args, p.smem, s);
}
template <typename T, int W>
cudaError_t launch_pcg_w(const PcgPlan& p, const PcgArgs<T>& A, cudaStream_t s) {
    switch (p.arrays) {
        case 4: return p.placed ? launch_pcg_t<T, W, 4, 4>(p, A, s) : launch_pcg_t<T, W, 4, 0>(p, A, s);
        case 3: return p.placed ? launch_pcg_t<T, W, 3, 4>(p, A, s) : launch_pcg_t<T, W, 3, 0>(p, A, s);
        default:
            if constexpr (pcg_least_arrays<T>(W) == 2) return launch_pcg_t<T, W, 2, 0>(p, A, s);
            else return cudaErrorInvalidValue;
    }
}
template <typename T>
cudaError_t launch_pcg(const PcgPlan& p, const PcgArgs<T>& A, cudaStream_t s) {
    constexpr int V = VecW<T>::W;
    return A.g.nz % V == 0 ? launch_pcg_w<T, V>(p, A, s) : launch_pcg_w<T, 1>(p, A, s);
}

template <typename T>
cudaError_t pressure_pcg(const PressureWork<T>& W, const PoissonGrid& g, double bb, double rr0, double tol,
                         int max_iter, PressureReport* rep, cudaStream_t s) {
    const int nb = kRedBlocks, nt = kRedThreads;
    rep->launches = 1;
    k_pcg_init<T><<<nb, nt, 0, s>>>(g, W.r, W.z, W.scal, tol * tol * bb, rr0, W.part, W.ticket);
    // iterations are enqueued in batches; the device flag turns the rest of a batch into
    // empty launches once the residual is below tolerance
    PcgPlan plan = pcg_plan<T>(g);
    T* dold = W.d;
    T* dnew = W.d2;
    int launched = 0;
    double st[3] = {rr0 <= tol * tol * bb ? 1.0 : 0.0, 0.0, rr0};   // done, iterations, rr
    while (launched < max_iter && st[0] == 0.0) {
        const int batch = std::min(plan.blocks ? kPcgIters : kCgBatch, max_iter - launched);
        if (plan.blocks) {
            static_assert(0x40404040u >= kPcgStuck && 0x40404040u < 2 * kPcgStuck, "a counter in which a wait ran out");
            cudaError_t e = cudaMemsetAsync(W.slots, W.stuck ? 0x40 : 0, sizeof(unsigned long long), s);
            const PcgArgs<T> A{g, W.p, W.r, W.z, dold, dnew, W.scal, (double*)(W.slots + 1), (unsigned*)W.slots, plan.chunk, batch, launched == 0};
            if (e == cudaSuccess) e = launch_pcg<T>(plan, A, s);
            if (e == cudaErrorCooperativeLaunchTooLarge) {   // not all blocks fit at once: launch by launch
                cudaGetLastError();
                plan.blocks = 0;
                continue;
            }
            if (e != cudaSuccess) return e;
            if (batch & 1) std::swap(dold, dnew);
            rep->launches += 1;
        } else {
            for (int b = 0; b < batch; ++b) {
                launch_direction<T>(W, g, dold, dnew, launched + b == 0, nullptr, W.part, W.ticket, s);
                launch_update<T>(W, g, dnew, true, W.part + 2 * nb, W.ticket + 1, s);
                std::swap(dold, dnew);
            }
            rep->launches += 2 * batch;
        }
        launched += batch;
        double tail[4];
        unsigned stuck = 0;
        cudaMemcpyAsync(tail, W.scal + S_RR, 4 * sizeof(double), cudaMemcpyDeviceToHost, s);
        if (plan.blocks) cudaMemcpyAsync(&stuck, W.slots, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
        const cudaError_t e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return e;
        if (stuck >= kPcgStuck) return cudaErrorLaunchTimeout;   // a meeting of k_pcg ran out
        st[0] = tail[S_DONE - S_RR]; st[1] = tail[S_ITERS - S_RR]; st[2] = tail[0];
    }
    rep->iterations = (int)st[1];
    rep->rel_residual = bb > 0.0 ? std::sqrt(st[2] / bb) : 0.0;
    rep->status = st[0] == 0.0 ? 1 : 0;
    return cudaGetLastError();
}

template <typename T>
cudaError_t pressure_solve(const PressureWork<T>& W, const PoissonGrid& g, double h, const T* u, const T* v,
                           const T* w, double tol, int max_iter, PressureReport* rep, cudaStream_t s) {
    double br[2];
    cudaError_t e = pressure_rhs<T>(W, g, h, u, v, w, false, br, s);
    if (e != cudaSuccess) return e;
    rep->iterations = 0; rep->rel_residual = 0.0; rep->status = 0; rep->launches = 2; rep->bb = br[0];
    if (br[0] == 0.0) return cudaGetLastError();
    PressureReport r2;
    e = pressure_pcg<T>(W, g, br[0], br[1], tol, max_iter, &r2, s);
    r2.launches += 2;
    r2.bb = br[0];
    *rep = r2;
    return e;
}

template <typename T>
cudaError_t pressure_residual(const PressureWork<T>& W, const PoissonGrid& g, const T* rhs, double* rr_host,
                              cudaStream_t s) {
    k_residual<T><<<kRedBlocks, kRedThreads, 0, s>>>(g, rhs, W.p, W.r, W.part);
    k_finish<<<1, 256, 0, s>>>(W.part, kRedBlocks, 1, W.sums);
    cudaMemcpyAsync(rr_host, W.sums, sizeof(double), cudaMemcpyDeviceToHost, s);
    return cudaStreamSynchronize(s);
}

template <typename T>
cudaError_t fcg_begin(const PressureWork<T>& W, double bb, double rr0, double tol, cudaStream_t s) {
    k_fcg_begin<<<1, 1, 0, s>>>(W.scal, tol * tol * bb, rr0);
    return cudaGetLastError();
}

template <typename T>
cudaError_t fcg_iteration(const PressureWork<T>& W, const PoissonGrid& g, const FcgBuffers<T>& B, int it, int m,
                          cudaStream_t s) {
    const unsigned n = (unsigned)g.nx * g.ny * g.nz;
    m = std::max(1, std::min(m, kFcgMaxDirs));
    const int ring = m + 1, newslot = it % ring;
    DirSet<T> qs, ds;
    qs.n = ds.n = std::min(it, m);
    for (int j = 0; j < qs.n; ++j) {
        const int sl = (it - 1 - j) % ring;
        qs.v[j] = B.q[sl]; qs.slot[j] = sl;
        ds.v[j] = B.d[sl]; ds.slot[j] = sl;
    }
    const int nb = kRedBlocks, nt = kRedThreads;
    const T* dn = B.d[newslot];
    T* qn = B.q[newslot];
    double* part = W.part + (kFcgMaxDirs + 1) * nb;
    cudaError_t err = cudaSuccess;
    auto run = [&](auto w, auto nq) {
        constexpr int V = decltype(w)::value, NQ = decltype(nq)::value;
        constexpr int sm = kDotsSmem<T, V, NQ>;
        if (sm > 0 && err == cudaSuccess)
            err = cudaFuncSetAttribute(k_fcgm_dots<T, V, NQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
        if (err != cudaSuccess) return;
        k_fcgm_dots<T, V, NQ><<<nb, nt, sm, s>>>(n, W.scal, W.z, W.r, qs, W.part, W.ticket);
        k_fcgm_combine<T, V, NQ><<<nb, nt, 0, s>>>(n, W.scal, W.z, ds, B.d[newslot]);
        if (g.solid) k_fcgm_apply<T, V, true><<<nb, nt, 0, s>>>(g, W.scal, dn, qn, newslot, W.r, part, W.ticket + 1);
        else k_fcgm_apply<T, V, false><<<nb, nt, 0, s>>>(g, W.scal, dn, qn, newslot, W.r, part, W.ticket + 1);
    };
    auto dirs = [&](auto w) {
        static_assert(kFcgMaxDirs == 8, "one case a count");
        switch (qs.n) {
            case 0: run(w, std::integral_constant<int, 0>()); break;
            case 1: run(w, std::integral_constant<int, 1>()); break;
            case 2: run(w, std::integral_constant<int, 2>()); break;
            case 3: run(w, std::integral_constant<int, 3>()); break;
            case 4: run(w, std::integral_constant<int, 4>()); break;
            case 5: run(w, std::integral_constant<int, 5>()); break;
            case 6: run(w, std::integral_constant<int, 6>()); break;
            case 7: run(w, std::integral_constant<int, 7>()); break;
            default: run(w, std::integral_constant<int, 8>());
        }
    };
    if (g.nz % VecW<T>::W == 0) dirs(std::integral_constant<int, VecW<T>::W>());
    else dirs(std::integral_constant<int, 1>());
    if (err != cudaSuccess) return err;
    launch_update<T>(W, g, B.d[newslot], false, W.part, W.ticket + 2, s, B.q[newslot]);
    return cudaGetLastError();
}

cudaError_t solver_state(const double* scal, double out[3], cudaStream_t s) {
    double tail[4];
    cudaMemcpyAsync(tail, scal + S_RR, 4 * sizeof(double), cudaMemcpyDeviceToHost, s);
    const cudaError_t e = cudaStreamSynchronize(s);
    out[0] = tail[0]; out[1] = tail[S_DONE - S_RR]; out[2] = tail[S_ITERS - S_RR];
    return e;
}

template <typename T>
cudaError_t subtract_gradient(const T* p, T* u, T* v, T* w, const PoissonGrid& g, double h, double* loss_part,
                              double* loss_sums, cudaStream_t s) {
    k_subtract_gradient<T, T><<<kRedBlocks, kRedThreads, 0, s>>>(g, (T)(1.0 / h), p, u, v, w);
    k_wall_loss<T><<<kRedBlocks, kRedThreads, 0, s>>>(g.nx, g.ny, g.nz, h, p, loss_part);
    k_finish<<<1, 256, 0, s>>>(loss_part, kRedBlocks, 3, loss_sums);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------
// FP64 residual refinement of the FP32 form
// ---------------------------------------------------------------------------------
// r = -b - B p64 in FP64 arithmetic (b = div(u) h from the FP32 velocities), stored as FP32
// for the next correction solve; partial |r|^2
__global__ void __launch_bounds__(kRedThreads) k_true_residual(PoissonGrid g, double h, const float* __restrict__ u,
                                                                const float* __restrict__ v, const float* __restrict__ w,
                                                                const double* __restrict__ p, float* __restrict__ r,
                                                                double* part) {
    const unsigned n = (unsigned)g.nx * g.ny * g.nz;
    const int ny = g.ny, nz = g.nz;
    double acc = 0.0;
    for (unsigned c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        double rc = 0.0;
        if (!excluded(g, c)) {
            const Cell k = decode(c, ny, nz);
            const double b = net_outflow<double>(g, c, k, u, v, w) * h;
            double s = 0.0;
            const int diag = for_neighbours(g, c, k, [&](unsigned o) { s += p[o]; });
            rc = -b - ((double)diag * p[c] - s);
        }
        r[c] = (float)rc;
        acc += rc * rc;
    }
    const double a[1] = {acc};
    block_sums<1>(a, part);
}

__global__ void k_to_double(const float* __restrict__ a, double* __restrict__ b, unsigned n, int accumulate) {
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        b[i] = accumulate ? b[i] + (double)a[i] : (double)a[i];
}
__global__ void k_to_float(const double* __restrict__ a, float* __restrict__ b, unsigned n) {
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = (float)a[i];
}

cudaError_t true_residual(const PressureWork<float>& W, const PoissonGrid& g, double h, const float* u,
                          const float* v, const float* w, const double* p64, double* rr_host, cudaStream_t s) {
    k_true_residual<<<kRedBlocks, kRedThreads, 0, s>>>(g, h, u, v, w, p64, W.r, W.part);
    k_finish<<<1, 256, 0, s>>>(W.part, kRedBlocks, 1, W.sums);
    cudaMemcpyAsync(rr_host, W.sums, sizeof(double), cudaMemcpyDeviceToHost, s);
    return cudaStreamSynchronize(s);
}

cudaError_t widen(const float* a, double* b, long long n, bool accumulate, cudaStream_t s) {
    k_to_double<<<kRedBlocks, kRedThreads, 0, s>>>(a, b, (unsigned)n, accumulate ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t narrow(const double* a, float* b, long long n, cudaStream_t s) {
    k_to_float<<<kRedBlocks, kRedThreads, 0, s>>>(a, b, (unsigned)n);
    return cudaGetLastError();
}

cudaError_t subtract_gradient_p64(const double* p64, float* u, float* v, float* w, const PoissonGrid& g, double h,
                                  double* loss_part, double* loss_sums, cudaStream_t s) {
    k_subtract_gradient<float, double><<<kRedBlocks, kRedThreads, 0, s>>>(g, 1.0 / h, p64, u, v, w);
    k_wall_loss<double><<<kRedBlocks, kRedThreads, 0, s>>>(g.nx, g.ny, g.nz, h, p64, loss_part);
    k_finish<<<1, 256, 0, s>>>(loss_part, kRedBlocks, 3, loss_sums);
    return cudaGetLastError();
}

// the arrival counter of k_pcg and its blocks' partial sums
size_t pressure_slots() { return 1 + (size_t)kPcgBlocksMax * kPcgPartWords; }

// partial rows: the FCG dot kernel's kFcgMaxDirs + 1 and the direction kernel's 2 (the CG
// kernels use fewer)
size_t pressure_partials() { return (size_t)kRedBlocks * (kFcgMaxDirs + 4); }

#define FIA_PRESSURE_INST(T)                                                                                       \
    template cudaError_t pressure_rhs<T>(const PressureWork<T>&, const PoissonGrid&, double, const T*, const T*,    \
                                         const T*, bool, double*, cudaStream_t);                                    \
    template cudaError_t pressure_pcg<T>(const PressureWork<T>&, const PoissonGrid&, double, double, double, int,   \
                                         PressureReport*, cudaStream_t);                                            \
    template cudaError_t pressure_solve<T>(const PressureWork<T>&, const PoissonGrid&, double, const T*, const T*,  \
                                           const T*, double, int, PressureReport*, cudaStream_t);                   \
    template cudaError_t fcg_begin<T>(const PressureWork<T>&, double, double, double, cudaStream_t);               \
    template cudaError_t pressure_residual<T>(const PressureWork<T>&, const PoissonGrid&, const T*, double*,         \
                                              cudaStream_t);                                                          \
    template cudaError_t fcg_iteration<T>(const PressureWork<T>&, const PoissonGrid&, const FcgBuffers<T>&, int, int, \
                                          cudaStream_t);                                                              \
    template cudaError_t subtract_gradient<T>(const T*, T*, T*, T*, const PoissonGrid&, double, double*, double*,   \
                                              cudaStream_t);
FIA_PRESSURE_INST(double)
FIA_PRESSURE_INST(float)
#undef FIA_PRESSURE_INST

}  // namespace fia
