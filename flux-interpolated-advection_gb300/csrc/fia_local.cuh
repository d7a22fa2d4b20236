// fia_local.cuh -- FP32 building blocks in local cell coordinates (the chosen form).
//
// Positions are carried as an integer anchor (a cell-lattice index) plus a small FP32
// offset q, both in units of the cell length: X = anchor + q.  Every quantity the FP32
// arithmetic sees is then O(CFL): stencil distances, colours, centroids and normals keep
// FP32's full relative precision regardless of where in a 256^3 or 384^3 grid the face is.
// Absolute FP32 coordinates would lose ~1.5e-5 of a cell at 256^3.
//
// psi is carried as a double-float pair (hi, lo) in cell units (psi / h).  A face
// interpolates psi - Psi0 for a base node Psi0 of its own, formed from the pairs as
// (hi - hi0) + (lo - lo0): WENO6, trilinear and 1Dy-linear interpolation all commute with
// adding a constant (the smoothness indicators are quadratic forms of differences and the
// weights sum to one), so this is the same interpolant without FP32 cancellation.
#pragma once
#include "fia_device.cuh"

namespace fia {

// One 1D WENO6 evaluation as a real call.  Inlined, the face kernel held some sixty copies
// of weno6_eval (the unrolled z-passes of a stencil), more code than the instruction cache
// holds; ncu showed most warps waiting on instruction fetch.  Arguments travel in registers.
static __device__ __noinline__ float weno6_f(float f0, float f1, float f2, float f3, float f4, float f5, WenoCoef<float> w) {
    const float f[6] = {f0, f1, f2, f3, f4, f5};
    return weno6_eval<float, true>(f, w);
}
__device__ __forceinline__ float weno6_call(const float* f, const WenoCoef<float>& w) {
    return weno6_f(f[0], f[1], f[2], f[3], f[4], f[5], w);
}
// Two evaluations with the same coefficients in one call: the two dependency chains (the
// weights end in a serial max / reciprocal / normalise tail) interleave, which a call per
// evaluation prevents, at half the calls.  Each result equals weno6_f's.
static __device__ __noinline__ float2 weno6_f2(float a0, float a1, float a2, float a3, float a4, float a5, float b0, float b1,
                                        float b2, float b3, float b4, float b5, WenoCoef<float> w) {
    const float fa[6] = {a0, a1, a2, a3, a4, a5}, fb[6] = {b0, b1, b2, b3, b4, b5};
    return make_float2(weno6_eval<float, true>(fa, w), weno6_eval<float, true>(fb, w));
}
__device__ __forceinline__ float2 weno6_call2(const float* a, const float* b, const WenoCoef<float>& w) {
    return weno6_f2(a[0], a[1], a[2], a[3], a[4], a[5], b[0], b[1], b[2], b[3], b[4], b[5], w);
}

// error-free sum of two floats (Knuth TwoSum)
__host__ __device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// running sum with a compensation term
struct Kahan {
    float s = 0.f, c = 0.f;
    __host__ __device__ __forceinline__ void add(float x) {
        float t, e;
        two_sum(s, x, t, e);
        s = t;
        c += e;
    }
    __host__ __device__ __forceinline__ float value() const { return s + c; }
};

// Loads node values as floats: plain array, or psi pairs relative to a base pair.
// Node offsets are 32-bit: fia_create admits grids with (nx+2)(ny+2)(nz+2) <= 2^31, which
// bounds every node field of the path.
struct PlainLoad {
    const float* __restrict__ a;
    __device__ __forceinline__ float operator()(int i) const { return __ldg(a + i); }
};
struct PsiLoad {
    const float2* __restrict__ a;
    float hi0, lo0;
    __device__ __forceinline__ float operator()(int i) const {
        const float2 v = __ldg(a + i);
        return (v.x - hi0) + (v.y - lo0);
    }
};

// stencil base and fractional offset of the local position along one axis
__device__ __forceinline__ void locate(int anchor, float q, float off, int& base, float& s) {
    const float r = q - off;
    const float f = floorf(r);
    base = anchor + (int)f;
    s = r - f;
}
// the cell holding the local position along one axis (a discrete decision: snapped)
__device__ __forceinline__ int cell_of(int anchor, float q, float off) {
    return anchor + (int)floorf(snap_int(q - off));
}

template <class L>
__device__ float weno6_3d_loc(const L& load, const NodeField& F, const int* anc, const float* q) {
    int bx, by, bz;
    float sx, sy, sz;
    locate(anc[0], q[0], F.oxf, bx, sx);
    locate(anc[1], q[1], F.oyf, by, sy);
    locate(anc[2], q[2], F.ozf, bz, sz);
    float tx[6], ty[6], tz[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        tx[i] = sx + float(2 - i);
        ty[i] = sy + float(2 - i);
        tz[i] = sz + float(2 - i);
    }
    const WenoCoef<float> cx = weno_coef(tx), cy = weno_coef(ty), cz = weno_coef(tz);
    int kk[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) kk[i] = clampi(bz - 2 + i, F.Mz - 1);
    float yv[6];
#pragma unroll 1
    for (int ix = 0; ix < 6; ++ix) {
        const int ii = clampi(bx - 2 + ix, F.Mx - 1);
        float zv[6];
#pragma unroll
        for (int iy = 0; iy < 6; iy += 2) {
            const int j0 = clampi(by - 2 + iy, F.My - 1), j1 = clampi(by - 1 + iy, F.My - 1);
            const int row0 = F.Mz * (F.My * ii + j0), row1 = F.Mz * (F.My * ii + j1);
            float f0[6], f1[6];
#pragma unroll
            for (int iz = 0; iz < 6; ++iz) { f0[iz] = load(row0 + kk[iz]); f1[iz] = load(row1 + kk[iz]); }
            const float2 v = weno6_call2(f0, f1, cz);
            zv[iy] = v.x; zv[iy + 1] = v.y;
        }
        yv[ix] = weno6_call(zv, cy);
    }
    return weno6_call(yv, cx);
}

template <class L>
__device__ float lin3d_loc(const L& load, const NodeField& F, const int* anc, const float* q) {
    int bx, by, bz;
    float sx, sy, sz;
    locate(anc[0], q[0], F.oxf, bx, sx);
    locate(anc[1], q[1], F.oyf, by, sy);
    locate(anc[2], q[2], F.ozf, bz, sz);
    const int k0 = clampi(bz, F.Mz - 1), k1 = clampi(bz + 1, F.Mz - 1);
    float yv[2];
#pragma unroll
    for (int ix = 0; ix < 2; ++ix) {
        const int ii = clampi(bx + ix, F.Mx - 1);
        float zv[2];
#pragma unroll
        for (int iy = 0; iy < 2; ++iy) {
            const int jj = clampi(by + iy, F.My - 1);
            const int row = F.Mz * (F.My * ii + jj);
            zv[iy] = (1.f - sz) * load(row + k0) + sz * load(row + k1);
        }
        yv[ix] = (1.f - sy) * zv[0] + sy * zv[1];
    }
    return (1.f - sx) * yv[0] + sx * yv[1];
}

template <class L>
__device__ float lin1dy_loc(const L& load, const NodeField& F, const int* anc, const float* q) {
    int by;
    float sy;
    const int ix = clampi(cell_of(anc[0], q[0], F.oxf - 0.5f), F.Mx - 1);
    const int iz = clampi(cell_of(anc[2], q[2], F.ozf - 0.5f), F.Mz - 1);
    locate(anc[1], q[1], F.oyf, by, sy);
    const float f0 = load(F.Mz * (F.My * ix + clampi(by, F.My - 1)) + iz);
    const float f1 = load(F.Mz * (F.My * ix + clampi(by + 1, F.My - 1)) + iz);
    return (1.f - sy) * f0 + sy * f1;
}

template <class L>
__device__ __forceinline__ float interp_loc(int method, const L& load, const NodeField& F, const int* anc,
                                            const float* q) {
    if (method == INTERP_WENO6) return weno6_3d_loc(load, F, anc, q);
    if (method == INTERP_LINEAR) return lin3d_loc(load, F, anc, q);
    return lin1dy_loc(load, F, anc, q);
}

}  // namespace fia
