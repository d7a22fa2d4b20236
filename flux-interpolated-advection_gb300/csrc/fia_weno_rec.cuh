// fia_weno_rec.cuh -- the tensor-product WENO6 of the per-piece quadrature, with what depends on
// the samples alone kept apart from what depends on the position.
//
// Along z, the first pass of the tensor product, the samples are the field's own nodes, so a
// record per node row and stencil base holds that part once for every point interpolated there:
// some 350 evaluations per node in a density pass at three pieces per face.  Along y, the Gauss
// points of one half cell share their stencil, so it is formed once for all of them.
//
// Two arithmetics.
//
// WenoNewton (density, and every field of the FP64 form).  For six samples f0..f5 and a position s in [0, 1) past f2, the three
// cubic candidates in Newton form around f2 share their linear term:
//   P_i = f2 + s D2 + m G_i,   m = s (s - 1) / 6,
//   G_0 = 3 S1 + (s + 1) T0,  G_1 = 3 S1 + (s + 1) (S2 - S1),  G_2 = 3 S2 + (s - 2) T2
// (D first, S second, T third differences: D2 = f3 - f2, S1 = f1 - 2 f2 + f3, S2 = f2 - 2 f3 + f4,
// T0 and T2 over f0..f3 and f2..f5), so the interpolant is f2 + s D2 + m sum a_i G_i / sum a_i with
// a_i = C_i(s) q_i, q_i = 1 / (eps + beta_i)^2.  A G_i holds differences of its own candidate's
// samples only, so a jump outside them does not reach it.  The differences and the q_i are functions of the
// samples only (WENO6_interpolation_3d.cpp:70-123; equal in exact arithmetic, and a little closer
// to it in FP32: 3.1e-7 against 3.8e-7 of a 128^3 density step).  17 arithmetic instructions and
// one 32-byte load from a record, against about 62 and six 4-byte loads from the samples.
//
// WenoSamples (velocity).  weno6_eval's own arithmetic (fia_device.cuh), bit for bit, from
// records that hold the samples and their reciprocal indicators.  The pressure of the projection
// after a velocity step answers to the last bits of the velocities: the sum of their rounding on
// the walls is a net outflow that the pinned cell turns into an offset of the pressure, and the
// path of some thousand FP32 CG iterations up to its tolerance depends on them (the Newton form
// moved the pressure of a 64^3 step by 1.3e-4, and by 1e-5 to 7e-5 with the wall rows kept).
#pragma once
#include "fia_advect.cuh"
#include "fia_local.cuh"

namespace fia {

// 1/x for the weights' quotients.  FP32: the hardware approximation (1 ulp) without the scaling
// of subnormal operands, which weno_indicators keeps away.  FP64: the hardware's seed (20 bits) and
// two Newton steps x += x (1 - a x), correct to about one unit in the last place: four FP64
// instructions, of which an IEEE division takes about ten.  The quotient is off by another rounding, where
// a division has one in all; with the Newton form's fewer roundings before it the psi of a 32^3 field is
// still closer to its 113-bit value than with divisions: rms 2.0e-17 against 4.7e-17 on a smooth field of
// order 1, 2.3e-17 against 5.3e-17 on noise, 4.4e-17 against 9.2e-17 on steps.  Whole density steps (12^3
// to 20^3, CFL 1 to 2.5, MacCormack among them) are 1.8% closer to an 80-bit run on average over 54.
__device__ __forceinline__ float weno_rcp(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ double weno_rcp(double a) {
    double x;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(a));
    x = fma(x, fma(-a, x, 1.0), x);
    return fma(x, fma(-a, x, 1.0), x);
}

// what depends on the position alone
template <typename T>
struct WenoPos {
    T s, sp1t, sm2, m, c0, c1, c2;
};
template <typename T>
__device__ __forceinline__ WenoPos<T> weno_pos(T s) {
    WenoPos<T> p;
    const T sm3 = s - T(3), sp2 = s + T(2), sp1 = s + T(1);
    p.s = s;
    p.sp1t = sp1 * (T(1) / T(3));
    p.sm2 = s - T(2);
    p.m = (s * s - s) * (T(1) / T(6));
    // ideal weights scaled by 20, which the quotient does not see
    p.c0 = p.sm2 * sm3;
    p.c1 = (T(-2) * sm3) * sp2;
    p.c2 = sp1 * sp2;
    return p;
}

// what depends on the samples alone; q up to a common factor
template <typename T>
struct WenoData {
    T f, d, s1, s2, t0, t2, q0, q1, q2;   // f2, D2, 3 S1, 3 S2, 3 T0, T2
};

template <typename T>
__device__ __forceinline__ T weno_at(const WenoData<T>& w, const WenoPos<T>& p) {
    const T a0 = p.c0 * w.q0, a1 = p.c1 * w.q1, a2 = p.c2 * w.q2;
    const T g0 = fma(p.sp1t, w.t0, w.s1), g1 = fma(p.sp1t, w.s2 - w.s1, w.s1), g2 = fma(p.sm2, w.t2, w.s2);
    const T g = fma(a2, g2, fma(a1, g1, a0 * g0)) * weno_rcp((a0 + a1) + a2);
    return fma(p.m, g, fma(p.s, w.d, w.f));
}

// The indicators e_i = 180 K (eps + beta_i) as the quadratic forms of weno6_eval (fia_device.cuh)
// in Horner form; the weights do not see the factors.  In FP32 K = 2^-40 centres the squared
// reciprocals in the type's range: differences up to 1e14 give normal weights.
template <typename T>
__device__ __forceinline__ void weno_indicators(T D0, T D1, T D2, T D3, T D4, T& e0, T& e1, T& e2) {
    constexpr T K = sizeof(T) == 4 ? T(1) / T(1099511627776.0) : T(1);
    const T eps = T(0.00018) * K;
    const T w2 = (T(814) * K) * D2;
    e0 = fma(D0, (T(244) * K) * D0 - (T(1171) * K) * D1 + (T(683) * K) * D2,
             fma(D1, (T(1561) * K) * D1 - (T(1951) * K) * D2, fma(w2, D2, eps)));
    e1 = fma(D1, (T(244) * K) * D1 - (T(781) * K) * D2 + (T(293) * K) * D3,
             fma(D2, (T(961) * K) * D2 - (T(781) * K) * D3, fma((T(244) * K) * D3, D3, eps)));
    e2 = fma(D2, w2 - (T(1951) * K) * D3 + (T(683) * K) * D4,
             fma(D3, (T(1561) * K) * D3 - (T(1171) * K) * D4, fma((T(244) * K) * D4, D4, eps)));
}

template <typename T>
__device__ __forceinline__ void weno_differences(T f, T D0, T D1, T D2, T D3, T D4, WenoData<T>& w) {
    const T S0 = D1 - D0, S1 = D2 - D1, S2 = D3 - D2, S3 = D4 - D3;
    w.f = f;
    w.d = D2;
    w.s1 = T(3) * S1;
    w.s2 = T(3) * S2;
    w.t0 = T(3) * (S1 - S0);
    w.t2 = S3 - S2;
}

// from six values (the second and third pass, whose samples differ from piece to piece).
// FP32: q_i by approximate reciprocals.  FP64: the q_i times (e0 e1 e2)^2, which needs no division;
// e_i >= 1.8e-4 and the products stay in range for differences up to 1e33.
__device__ __forceinline__ void weno_weights(float e0, float e1, float e2, WenoData<float>& w) {
    const float r0 = weno_rcp(e0), r1 = weno_rcp(e1), r2 = weno_rcp(e2);
    w.q0 = r0 * r0;
    w.q1 = r1 * r1;
    w.q2 = r2 * r2;
}
__device__ __forceinline__ void weno_weights(double e0, double e1, double e2, WenoData<double>& w) {
    const double a = e1 * e2, b = e0 * e2, c = e0 * e1;
    w.q0 = a * a;
    w.q1 = b * b;
    w.q2 = c * c;
}
template <typename T>
__device__ __forceinline__ WenoData<T> weno_data(const T* f) {
    WenoData<T> w;
    const T D0 = f[1] - f[0], D1 = f[2] - f[1], D2 = f[3] - f[2], D3 = f[4] - f[3], D4 = f[5] - f[4];
    T e0, e1, e2;
    weno_indicators(D0, D1, D2, D3, D4, e0, e1, e2);
    weno_differences(f[2], D0, D1, D2, D3, D4, w);
    weno_weights(e0, e1, e2, w);
    return w;
}

// The stored record: eight values, the q_i normalised to sum 1 and the middle one left out
// (q1 = 1 - q0 - q2, off by at most one rounding of 1, like the normalised weights themselves).
template <typename T>
struct WenoRec {
    T f, d, s1, s2, t0, t2, q0, q2;
};

// Scaled by the smallest indicator, so the squares neither overflow nor all underflow.
template <typename T>
__device__ __forceinline__ WenoRec<T> weno_record(T f, T D0, T D1, T D2, T D3, T D4) {
    WenoData<T> w;
    T e0, e1, e2;
    weno_indicators(D0, D1, D2, D3, D4, e0, e1, e2);
    weno_differences(f, D0, D1, D2, D3, D4, w);
    const T em = fmin(e0, fmin(e1, e2));
    const T r0 = em / e0, r1 = em / e1, r2 = em / e2;
    const T sum = (r0 * r0 + r1 * r1) + r2 * r2;
    WenoRec<T> r;
    r.f = w.f; r.d = w.d; r.s1 = w.s1; r.s2 = w.s2; r.t0 = w.t0; r.t2 = w.t2;
    r.q0 = r0 * r0 / sum;
    r.q2 = r2 * r2 / sum;
    return r;
}

// Records of a node field F: rows (i, j) of Mz + 1 records, record b + 1 for the stencil whose
// third sample is node b (b = -1 .. Mz - 1; the sample indices clamped to the row).  Points of
// the domain lie at b >= -1 and b <= Mz - 1 along z on every field of the path.
__host__ __device__ __forceinline__ long long weno_rec_count(const NodeField& F) {
    return (long long)F.Mx * F.My * (F.Mz + 1);
}

// the record's weights made explicit
template <typename T>
__device__ __forceinline__ WenoData<T> weno_unpack(const WenoRec<T>& r) {
    return WenoData<T>{r.f, r.d, r.s1, r.s2, r.t0, r.t2, r.q0, (T(1) - r.q0) - r.q2, r.q2};
}

// 32 bytes of a record in one load (p 32-byte aligned: records are multiples of 32 bytes from the
// base of an allocation): half the requests of two 16-byte loads.  The quadrature of a density step
// at 128^3 takes 2.50 ms, 2.61 with two; of a velocity step on 120 x 161 x 77 cells 7.25, 7.39.
__device__ __forceinline__ void ldg32(const float4* p, float4& a, float4& b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}
__device__ __forceinline__ void ldg32(const double* p, double& a, double& b, double& c, double& d) {
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a), "=d"(b), "=d"(c), "=d"(d) : "l"(p));
}

// FP64 records: eight doubles
__device__ __forceinline__ WenoRec<double> ldg_rec(const WenoRec<double>* p) {
    const double* q = reinterpret_cast<const double*>(p);
    WenoRec<double> r;
    ldg32(q, r.f, r.d, r.s1, r.s2);
    ldg32(q + 4, r.t0, r.t2, r.q0, r.q2);
    return r;
}

struct WenoNewton {
    typedef WenoPos<float> Coef;
    typedef WenoData<float> Data;
    static constexpr int kGroup = 3;    // Gauss points of a half evaluated together
    static constexpr int kAhead = 4;    // rows of a plane loaded a group ahead, of 7
    __device__ static __forceinline__ Coef coef(float s) { return weno_pos(s); }
    __device__ static __forceinline__ Data data(const float* f) { return weno_data(f); }
    __device__ static __forceinline__ float at(const Data& w, const Coef& c) { return weno_at(w, c); }
    struct Row {       // the six y-pass values of a point
        float f[6];
        __device__ __forceinline__ void set(int ix, const Data& w, const Coef& c) { f[ix] = weno_at(w, c); }
        __device__ __forceinline__ Data data() const { return weno_data(f); }
    };
    struct Raw {
        float4 a, b;   // a WenoRec
        __device__ __forceinline__ Data data() const {
            return weno_unpack(WenoRec<float>{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w});
        }
    };
    struct Records {   // of the field: two words a record
        const float4* __restrict__ r;
        int stride;    // Mz + 1
        __device__ __forceinline__ Raw load(int row, int b1) const {
            Raw w;
            ldg32(r + 2LL * (row * stride + b1), w.a, w.b);
            return w;
        }
    };
    // of psi: the record's f is the pair's high word, the differences are the pairs'; the value is
    // taken relative to the face's base pair, with the low word from the psi array
    struct Psi {
        const float4* __restrict__ r;
        PsiLoad load;
        int stride, b1;
        __device__ __forceinline__ Data data(int row) const {
            Raw w;
            ldg32(r + 2LL * (row * stride + b1), w.a, w.b);
            const float lo = __ldg(&load.a[row * (stride - 1) + (b1 > 0 ? b1 - 1 : 0)].y);
            w.a.x = (w.a.x - load.hi0) + (lo - load.lo0);
            return w.data();
        }
    };
    static __device__ __forceinline__ Psi psi_rows(const float4* prec, const PsiLoad& pl, int Mz, int bz) {
        return Psi{prec, pl, Mz + 1, clampi(bz + 1, Mz)};
    }
};

struct WenoSamples {
    typedef WenoCoef<float> Coef;
    typedef Weno6Data Data;
    static constexpr int kGroup = 1;    // one: a second point's coefficients would spill
    static constexpr int kAhead = 4;
    __device__ static __forceinline__ Coef coef(float s) {
        float t[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) t[i] = s + float(2 - i);
        return weno_coef(t);
    }
    __device__ static __forceinline__ Data data(const float* f) { return weno6_data(f); }
    __device__ static __forceinline__ float at(const Data& w, const Coef& c) { return weno6_at(w, c); }
    // The six y-pass values of a point.  The fourth and the sixth enter the x-pass through
    // differences only: they are kept as quotients num * rcp, whose product the differences take
    // unrounded.
    struct Row {
        float f[6], n3, r3, n5, r5;
        __device__ __forceinline__ void set(int ix, const Data& w, const Coef& c) {
            if (ix == 3) weno6_quotient(w, c, n3, r3);
            else if (ix == 5) weno6_quotient(w, c, n5, r5);
            else f[ix] = weno6_at(w, c);
        }
        __device__ __forceinline__ Data data() const {
            Data w;
            w.f0 = f[0]; w.f1 = f[1]; w.f2 = f[2];
            w.D0 = f[1] - f[0]; w.D1 = f[2] - f[1]; w.D2 = fmaf(n3, r3, -f[2]);
            const float D3 = fmaf(-n3, r3, f[4]), D4 = fmaf(n5, r5, -f[4]);
            w.S0 = w.D1 - w.D0; w.S1 = w.D2 - w.D1; w.S2 = D3 - w.D2;
            w.T0 = w.S1 - w.S0; w.T1 = w.S2 - w.S1; w.T2 = (D4 - D3) - w.S2;
            weno6_recips(w.D0, w.D1, w.D2, D3, D4, w.r0, w.r1, w.r2);
            return w;
        }
    };
    struct Raw {
        float4 a, b;   // the samples, r0, r1
        float c;       // r2
        __device__ __forceinline__ Data data() const {
            const float f[6] = {a.x, a.y, a.z, a.w, b.x, b.y};
            float D3, D4;
            Data w = weno6_differences(f, D3, D4);
            w.r0 = b.z; w.r1 = b.w; w.r2 = c;
            return w;
        }
    };
    struct Records {   // two words a record and r2 in a plane of its own
        const float4* __restrict__ r;
        const float* __restrict__ r2;
        int stride;
        __device__ __forceinline__ Raw load(int row, int b1) const {
            const int i = row * stride + b1;
            Raw w;
            ldg32(r + 2LL * i, w.a, w.b);
            w.c = __ldg(r2 + i);
            return w;
        }
    };
    // psi relative to the face's base pair: the samples depend on the face, so their data are
    // formed per piece
    struct Psi {
        PsiLoad load;
        int Mz, bz;
        __device__ __forceinline__ Data data(int row) const {
            float f[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) f[i] = load(row * Mz + clampi(bz - 2 + i, Mz - 1));
            return weno6_data(f);
        }
    };
    static __device__ __forceinline__ Psi psi_rows(const float4*, const PsiLoad& pl, int Mz, int bz) {
        return Psi{pl, Mz, bz};
    }
};

// The same without records, for a session that has no memory for them: the z-pass reads the six samples
// and forms what a record holds, for each piece anew.  A density step at 96^3 takes 3.4 ms so (2.5 with
// records, 5.3 before there were any, 9.2 with every point interpolated on its own), a velocity step at
// 80^3 6.1 (5.2, 9.8, 16.2).
struct FieldRows {
    const float* __restrict__ a;
    int Mz;
    __device__ __forceinline__ void load(int row, int b1, float (&f)[6]) const {
#pragma unroll
        for (int i = 0; i < 6; ++i) f[i] = __ldg(a + row * Mz + clampi(b1 - 3 + i, Mz - 1));
    }
};
template <class W>
struct FromField : W {
    static constexpr int kAhead = 2;   // of six samples each
    struct Raw {
        float f[6];
        __device__ __forceinline__ typename W::Data data() const { return W::data(f); }
    };
    struct Records {
        FieldRows rows;
        __device__ __forceinline__ Raw load(int row, int b1) const {
            Raw w;
            rows.load(row, b1, w.f);
            return w;
        }
    };
    // psi relative to the face's base pair (as WenoSamples::Psi)
    struct Psi {
        PsiLoad load;
        int Mz, bz;
        __device__ __forceinline__ typename W::Data data(int row) const {
            float f[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) f[i] = load(row * Mz + clampi(bz - 2 + i, Mz - 1));
            return W::data(f);
        }
    };
    static __device__ __forceinline__ Psi psi_rows(const float4*, const PsiLoad& pl, int Mz, int bz) {
        return Psi{pl, Mz, bz};
    }
};

inline WenoNewton::Records newton_records(const NodeField& F, const void* buf) {
    return WenoNewton::Records{static_cast<const float4*>(buf), F.Mz + 1};
}
inline WenoSamples::Records sample_records(const NodeField& F, const void* buf) {
    const float4* r = static_cast<const float4*>(buf);
    return WenoSamples::Records{r, reinterpret_cast<const float*>(r + 2 * weno_rec_count(F)), F.Mz + 1};
}

// The z-pass over the 6 x 7 (x, y) rows of a stencil into the thread's shared column:
// zs[(7 ix + r) * STRIDE] is the value of row (bx - 2 + ix, by0 - 2 + r).  Seven rows for every
// lane: points of the upper half read the last one, and a warp nearly always holds some.  The
// loads of one group of rows are in flight while the other group is evaluated: loaded and
// evaluated plane by plane, each plane waited for L2 (issue slots 61% busy, 128^3).
template <class W, int STRIDE>
__device__ __forceinline__ void rec_zpass(const typename W::Records& rec, const NodeField& F, int bx, int b1, int by0,
                                          const typename W::Coef& cz, float* zs) {
    constexpr int A = W::kAhead;
    int rj[7];
#pragma unroll
    for (int r = 0; r < 7; ++r) rj[r] = clampi(by0 - 2 + r, F.My - 1);
    typename W::Raw lo[A], hi[7 - A];
    int row = clampi(bx - 2, F.Mx - 1) * F.My;
#pragma unroll
    for (int r = 0; r < A; ++r) lo[r] = rec.load(row + rj[r], b1);
#pragma unroll 1
    for (int ix = 0; ix < 6; ++ix) {
        float* z = zs + 7 * ix * STRIDE;
#pragma unroll
        for (int r = 0; r < 7 - A; ++r) hi[r] = rec.load(row + rj[A + r], b1);
#pragma unroll
        for (int r = 0; r < A; ++r) z[r * STRIDE] = W::at(lo[r].data(), cz);
        if (ix < 5) {
            row = clampi(bx - 1 + ix, F.Mx - 1) * F.My;
#pragma unroll
            for (int r = 0; r < A; ++r) lo[r] = rec.load(row + rj[r], b1);
        }
#pragma unroll
        for (int r = 0; r < 7 - A; ++r) z[(A + r) * STRIDE] = W::at(hi[r].data(), cz);
    }
}

// y- and x-passes at up to W::kGroup points (n of them, y coefficients cy) that share the six
// rows from column word `up`: the data of a y-stencil are formed once for all of them.
template <class W, int STRIDE>
__device__ __forceinline__ void rec_yx(const float* zs, int up, const typename W::Coef* cy, int n,
                                       const typename W::Coef& cx, float* out) {
    typename W::Row yv[W::kGroup];
#pragma unroll
    for (int ix = 0; ix < 6; ++ix) {
        float f[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) f[i] = zs[(7 * ix + i + up) * STRIDE];
        const typename W::Data w = W::data(f);
#pragma unroll
        for (int q = 0; q < W::kGroup; ++q) yv[q].set(ix, w, cy[q]);
    }
#pragma unroll
    for (int q = 0; q < W::kGroup; ++q)
        if (q < n) out[q] = W::at(yv[q].data(), cx);
}

// WENO6 on a node row of F (y on node by exactly): the (x, z) interpolant of the row, 7
// evaluations, equal to the full form in exact arithmetic (every candidate polynomial of the
// y-pass interpolates the node and the weights sum to one).
template <class W>
__device__ __forceinline__ float psi_noderow(const typename W::Psi& psi, const NodeField& F, int bx, int by,
                                             const typename W::Coef& cz, const typename W::Coef& cx) {
    const int j = clampi(by, F.My - 1);
    float xv[6];
#pragma unroll
    for (int ix = 0; ix < 6; ++ix) xv[ix] = W::at(psi.data(clampi(bx - 2 + ix, F.Mx - 1) * F.My + j), cz);
    return W::at(W::data(xv), cx);
}

}  // namespace fia
