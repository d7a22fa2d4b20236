// fia_advect.cu -- the flux-interpolated advection pass on the GPU.
//
// One pass of the reference (advect_density_flux_advection_3D_std_thread,
// move_substances_3d.cpp:585-841, and its velocity counterpart
// advect_velocity_flux_advection_3d.cpp:252-576) becomes four kernels:
//
//   k_psi_inc, k_psi_scan  psi = running y-integral of the field: the cells' increments, their sums
//                (calc_psi_3D.cpp:10-308, :311-537)
//   k_backtrace  one thread per UNIQUE cell vertex: x' = x - dt u(x), pin rule, clamp
//                (calc_backtraced_face_3D.cpp:9-160).  The reference backtraces every
//                vertex once per face that uses it (up to 24 times).
//   k_faces      one thread per UNIQUE face: clip the backtraced face in (xi,eta) space
//                at the integer iso-lines of its vertex colours (facecutter.h:59-324,
//                split_face_3D.cpp:17-93), and for every piece evaluate the quadrature
//                of polygon_3D.cpp:257-487 with WENO6 / linear interpolation; the face
//                flux is accumulated in registers.  The reference computes each interior
//                face twice (once per adjacent cell, with reversed vertex order); the two
//                computations produce the same pieces with opposite normals, so one
//                signed flux per face is exact.
//   k_gather     one thread per cell: rho' = (sum of the six signed face fluxes) / V.
//                Deterministic, no atomics (the reference's per-thread += is racy).
#include "fia_advect.cuh"
#include "fia_weno_rec.cuh"
#include "fia_trace.cuh"

#include <cmath>
#include <vector>
#include <algorithm>

namespace fia {

// ------------------------------------------------------------------------------------
// host helpers
// ------------------------------------------------------------------------------------
static void legendre(int n, double x, double* p, double* dp) {
    double p0 = 1.0, p1 = x;
    for (int m = 2; m <= n; ++m) {
        double p2 = ((2.0 * m - 1.0) * x * p1 - (m - 1.0) * p0) / m;
        p0 = p1; p1 = p2;
    }
    if (n == 0) { *p = 1.0; *dp = 0.0; return; }
    *p = p1;
    *dp = n * (x * p1 - p0) / (x * x - 1.0);
}

// Gauss-Legendre rule on [-1,1]: Newton iteration on P_k from Chebyshev-like starting
// points; nodes ordered centre first then -/+ pairs by increasing |x| (the order of
// gauss_quadrature_points.cpp:18-60); weights normalised to sum 1.  Fixed arrays only (no
// heap), so the allocation-free entry point shares it.
void make_gauss(int k, double* x, double* w) {
    const double pi = 3.14159265358979323846;
    double nx[kMaxGauss + 1], nw[kMaxGauss + 1];
    int n = 0;
    for (int i = 0; i < (k + 1) / 2; ++i) {
        double z = std::cos(pi * (i + 0.75) / (k + 0.5));
        for (int it = 0; it < 100; ++it) {
            double p, dp; legendre(k, z, &p, &dp);
            double dz = p / dp; z -= dz;
            if (std::fabs(dz) < 1e-17) break;
        }
        double p, dp; legendre(k, z, &p, &dp);
        double wt = 2.0 / ((1.0 - z * z) * dp * dp);
        if (std::fabs(z) < 1e-15) { nx[n] = 0.0; nw[n++] = wt; }
        else { nx[n] = -std::fabs(z); nw[n++] = wt; nx[n] = std::fabs(z); nw[n++] = wt; }
    }
    // stable insertion sort by |x|
    for (int i = 1; i < n; ++i)
        for (int j = i; j > 0 && std::fabs(nx[j]) < std::fabs(nx[j - 1]); --j) {
            std::swap(nx[j], nx[j - 1]); std::swap(nw[j], nw[j - 1]);
        }
    for (int i = 0; i < k; ++i) { x[i] = nx[i]; w[i] = nw[i] / 2.0; }
}

NodeField cell_field(const int* N, int comp) {
    NodeField F;
    F.Mx = N[0] + (comp == 0); F.My = N[1] + (comp == 1); F.Mz = N[2] + (comp == 2);
    F.ox = comp == 0 ? 0.0 : 0.5; F.oy = comp == 1 ? 0.0 : 0.5; F.oz = comp == 2 ? 0.0 : 0.5;
    return F;
}

NodeField psi_field(const NodeField& A) {
    NodeField P = A;
    P.My = A.My + 1;
    P.oy = A.oy - 0.5;
    return P;
}

NodeField field32(NodeField F) {
    F.oxf = (float)F.ox; F.oyf = (float)F.oy; F.ozf = (float)F.oz;
    return F;
}

PassDesc desc32(const PassDesc& d) {
    PassDesc e = d;
    e.A = field32(d.A);
    e.P = field32(d.P);
    for (int q = 0; q < kMaxGauss; ++q) { e.gxf[q] = (float)d.gx[q]; e.gwf[q] = (float)d.gw[q]; }
    e.hf = (float)d.h;
    e.invhf = (float)(1.0 / d.h);
    e.dthf = (float)(d.dt / d.h);
    e.color_off_f[0] = (float)d.color_off[0]; e.color_off_f[1] = (float)d.color_off[1];
    e.minimal_area_f = (float)d.minimal_area;
    return e;
}

// ------------------------------------------------------------------------------------
// psi(.,0,.) = 0, psi(.,j,.) = psi(.,j-1,.) + incr(j-1): the cells' increments, then their sums
// ------------------------------------------------------------------------------------
// The increment of cell (i, c, k) goes to psi row c + 1; a thread takes kPsiRun cells of a column.
// WENO6: cell c spans [c + oy - 1/2, c + oy + 1/2] cells, k Gauss points per half, at offsets from
// the nodes that no cell changes; the stencil data of its second half (base c) serve the first half
// of cell c + 1.  Bound by the FP64 pipe.  The psi of a 64^3 plain-form step took 2.0 ms of 22.4 as one
// thread per column (4096 chains of 64 cells, every point from its samples), 0.13 now.
constexpr int kPsiRun = 4, kPsiThreads = 128;
template <typename T, int MODE>
__global__ void __launch_bounds__(kPsiThreads) k_psi_inc(PassDesc d, const T* __restrict__ a, T* __restrict__ psi) {
    __shared__ WenoPos<T> pos[2 * kMaxGauss];
    const T h = T(d.h);
    if constexpr (MODE == PSI_WENO6) {
        if (threadIdx.x < 2 * d.k) {
            const int half = (int)threadIdx.x >= d.k, q = threadIdx.x - half * d.k;
            // from node c - 1 in the first half, from node c in the second
            const T y = T(0.25) * (T(1) + T(d.gx[q]));
            pos[threadIdx.x] = weno_pos(half ? y : y + T(0.5));
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
        const T* col = a + idx3(d.A, i, 0, k);
        T f[6];
#pragma unroll
        for (int m = 0; m < 6; ++m) f[m] = ldg(col + (long long)clampi(j0 - 3 + m, My - 1) * Mz);
        WenoData<T> w = weno_data(f);
#pragma unroll 1
        for (int j = j0; j < j1; ++j) {
            T inc = T(0);
#pragma unroll 1
            for (int q = 0; q < d.k; ++q) inc += weno_at(w, pos[q]) * T(d.gw[q]);
#pragma unroll
            for (int m = 0; m < 5; ++m) f[m] = f[m + 1];
            f[5] = ldg(col + (long long)clampi(j + 3, My - 1) * Mz);
            w = weno_data(f);
#pragma unroll 1
            for (int q = 0; q < d.k; ++q) inc += weno_at(w, pos[d.k + q]) * T(d.gw[q]);
            psi[idx3(d.P, i, j + 1, k)] = inc * (h / T(2));
        }
    } else {
        const T px = (T(i) + T(d.A.ox)) * h, pz = (T(k) + T(d.A.oz)) * h;
        for (int j = j0; j < j1; ++j) {
            const T y0 = ((T(j) + T(0.25)) + T(d.A.oy) - T(0.5)) * h;
            const T y1 = ((T(j) + T(0.75)) + T(d.A.oy) - T(0.5)) * h;
            psi[idx3(d.P, i, j + 1, k)] =
                lin3d(a, d.A, h, px, y0, pz) * (h / T(2)) + lin3d(a, d.A, h, px, y1, pz) * (h / T(2));
        }
    }
}
// one thread per (x, z) column, the increments loaded kScanAhead at a time (PLAIN: formed from the field)
constexpr int kScanAhead = 16, kScanThreads = 64;
template <typename T, bool PLAIN>
__global__ void __launch_bounds__(kScanThreads) k_psi_scan(PassDesc d, const T* __restrict__ a, T* __restrict__ psi) {
    const int My = d.A.My, Mz = d.A.Mz;
    const long long col = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= (long long)d.A.Mx * Mz) return;
    const int i = (int)(col / Mz), k = (int)(col % Mz);
    const T h = T(d.h);
    T* P = psi + idx3(d.P, i, 0, k);
    const T* A = a + idx3(d.A, i, 0, k);
    T acc = T(0);
    *P = T(0);
    auto at = [&](int j) { return PLAIN ? ldg(A + (long long)(j - 1) * Mz) * h : P[(long long)j * Mz]; };
    int j = 1;
    for (; j + kScanAhead - 1 <= My; j += kScanAhead) {
        T v[kScanAhead];
#pragma unroll
        for (int m = 0; m < kScanAhead; ++m) v[m] = at(j + m);
#pragma unroll
        for (int m = 0; m < kScanAhead; ++m) {
            acc = acc + v[m];
            P[(long long)(j + m) * Mz] = acc;
        }
    }
    for (; j <= My; ++j) {
        acc = acc + at(j);
        P[(long long)j * Mz] = acc;
    }
}

// ------------------------------------------------------------------------------------
// vertex positions
// ------------------------------------------------------------------------------------
// interp with WENO6 collapsed along the axes on which the point lies on a node plane of F
// (equal in exact arithmetic; the vertices at rest and the psi points of the pieces sit there)
// (PassDesc::full_weno switches it off, to measure what it saves)
template <typename T>
__device__ __forceinline__ T interp_c(const PassDesc& d, int method, const T* __restrict__ a, const NodeField& F, T h,
                                      T px, T py, T pz) {
    if (method == INTERP_WENO6 && !d.full_weno) return weno6_3d_collapse(a, F, h, px, py, pz);
    return interp(method, a, F, h, px, py, pz);
}

template <typename T>
__device__ __forceinline__ void vertex_rest_position(const PassDesc& d, int i, int j, int k, T* p) {
    const T h = T(d.h);
    p[0] = T(i) * h; p[1] = T(j) * h; p[2] = T(k) * h;
    if (d.comp >= 0) p[d.comp] -= T(1) * T(0.5) * h;
}

// uniform in [-1, 1) from a vertex index, an axis and a seed (splitmix64 finaliser)
__device__ __forceinline__ double jitter_unit(long long id, int axis, unsigned seed) {
    unsigned long long x = (unsigned long long)id * 3ull + (unsigned long long)axis + ((unsigned long long)seed << 40);
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    x ^= x >> 31;
    return (double)(x >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// one thread a vertex: linear interpolation, and WENO6 without the collapse (PassDesc::full_weno)
template <typename T>
__global__ void k_backtrace(PassDesc d, const T* __restrict__ u, const T* __restrict__ v,
                            const T* __restrict__ w, NodeField fu, NodeField fv, NodeField fw,
                            T* __restrict__ verts) {
    const int Lx = d.A.Mx + 1, Ly = d.A.My + 1, Lz = d.A.Mz + 1;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)Lx * Ly * Lz) return;
    const int k = (int)(id % Lz);
    const int j = (int)((id / Lz) % Ly);
    const int i = (int)(id / ((long long)Lz * Ly));
    const T h = T(d.h);
    T p[3];
    vertex_rest_position(d, i, j, k, p);
    bool pinned = false;
    if (d.comp >= 0) {
        const int vi = d.comp == 0 ? i : (d.comp == 1 ? j : k);
        pinned = (vi <= 1 || vi >= d.N[d.comp]);
    }
    if (!pinned) {
        const T vx = interp(d.interp, u, fu, h, p[0], p[1], p[2]);
        const T vy = interp(d.interp, v, fv, h, p[0], p[1], p[2]);
        const T vz = interp(d.interp, w, fw, h, p[0], p[1], p[2]);
        const T dt = T(d.dt);
        p[0] -= vx * dt; p[1] -= vy * dt; p[2] -= vz * dt;
        if (d.vertex_jitter != 0.0)
            for (int c = 0; c < 3; ++c) p[c] += T(d.vertex_jitter * jitter_unit(id, c, d.jitter_seed)) * h;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int e = (c == d.comp);
        const T lo = T(0) - T(e) * T(0.5) * h;
        const T hi = T(0) + h * T(d.N[c]) + T(e) * T(0.5) * h;
        if (p[c] < lo) p[c] = lo;
        if (p[c] > hi) p[c] = hi;
    }
    verts[3 * id + 0] = p[0]; verts[3 * id + 1] = p[1]; verts[3 * id + 2] = p[2];
}

// The same with WENO6 collapsed on the node planes, a tile of vertices and one velocity component a
// block (fia_trace.cuh).
template <int N>
__global__ void __launch_bounds__(kTraceThreads) k_trace64(PassDesc d, const double* __restrict__ u,
                                                           const double* __restrict__ v, const double* __restrict__ w,
                                                           NodeField fu, NodeField fv, NodeField fw,
                                                           double* __restrict__ verts, TraceTiles tiles) {
    extern __shared__ double trace_sm[];
    const int c = blockIdx.y;
    const double* a = c == 0 ? u : (c == 1 ? v : w);
    const NodeField F = c == 0 ? fu : (c == 1 ? fv : fw);
    const double off[3] = {F.ox, F.oy, F.oz}, h = d.h;
    const int L[3] = {d.A.Mx + 1, d.A.My + 1, d.A.Mz + 1};
    const double q[3] = {d.comp == 0 ? -0.5 : 0.0, d.comp == 1 ? -0.5 : 0.0, d.comp == 2 ? -0.5 : 0.0};
    const double e = c == d.comp ? 0.5 * h : 0.0;
    const double lo = -e, hi = h * double(c == 0 ? d.N[0] : (c == 1 ? d.N[1] : d.N[2])) + e;
    const int Np = d.comp == 0 ? d.N[0] : (d.comp == 1 ? d.N[1] : d.N[2]);
    trace_tile<N, TraceCoef64>(a, F, off, L, q, tiles, trace_sm, [&](int i, int j, int k, double val) {
        const int vi = d.comp == 0 ? i : (d.comp == 1 ? j : k);
        const long long id = ((long long)i * L[1] + j) * L[2] + k;
        double p = double(c == 0 ? i : (c == 1 ? j : k)) * h - e;
        if (!(d.comp >= 0 && (vi <= 1 || vi >= Np))) {
            p -= val * d.dt;
            if (d.vertex_jitter != 0.0) p += d.vertex_jitter * jitter_unit(id, c, d.jitter_seed) * h;
        }
        verts[3 * id + c] = p < lo ? lo : (p > hi ? hi : p);
    });
}

// Second trace of the flux MacCormack scheme (calc_backtraced_face_3D.cpp:9-128, time
// direction "backward"): x2 = x1 + dt u(x1), the velocity interpolated at the backtraced
// position x1, the pin rule of the first trace, then the clamp (:131-160).
template <typename T>
__global__ void k_forward_trace(PassDesc d, const T* __restrict__ u, const T* __restrict__ v,
                                const T* __restrict__ w, NodeField fu, NodeField fv, NodeField fw,
                                const T* __restrict__ verts, T* __restrict__ verts2) {
    const int Lx = d.A.Mx + 1, Ly = d.A.My + 1, Lz = d.A.Mz + 1;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)Lx * Ly * Lz) return;
    const int k = (int)(id % Lz);
    const int j = (int)((id / Lz) % Ly);
    const int i = (int)(id / ((long long)Lz * Ly));
    const T h = T(d.h);
    T p[3] = {verts[3 * id], verts[3 * id + 1], verts[3 * id + 2]};
    bool pinned = false;
    if (d.comp >= 0) {
        const int vi = d.comp == 0 ? i : (d.comp == 1 ? j : k);
        pinned = (vi <= 1 || vi >= d.N[d.comp]);
    }
    if (!pinned) {
        const T vx = interp(d.interp, u, fu, h, p[0], p[1], p[2]);
        const T vy = interp(d.interp, v, fv, h, p[0], p[1], p[2]);
        const T vz = interp(d.interp, w, fw, h, p[0], p[1], p[2]);
        const T dt = T(d.dt);
        p[0] += vx * dt; p[1] += vy * dt; p[2] += vz * dt;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int e = (c == d.comp);
        const T lo = T(0) - T(e) * T(0.5) * h;
        const T hi = T(0) + h * T(d.N[c]) + T(e) * T(0.5) * h;
        if (p[c] < lo) p[c] = lo;
        if (p[c] > hi) p[c] = hi;
    }
    verts2[3 * id + 0] = p[0]; verts2[3 * id + 1] = p[1]; verts2[3 * id + 2] = p[2];
}

// ------------------------------------------------------------------------------------
// clipping in (xi, eta) space with an explicit stack
// ------------------------------------------------------------------------------------
template <typename T>
struct CV { T p0, p1, c0, c1; };   // xi, eta, colour component 0, colour component 1

constexpr int kPool = 144;     // vertex pool (LIFO) for pending pieces
constexpr int kMaxVerts = 32;  // vertices per piece (MAX_TMP_POINTS of facecutter.h)
constexpr int kMaxStack = 48;

template <typename T> __device__ __forceinline__ T cv_c(const CV<T>& v, int dim) { return dim ? v.c1 : v.c0; }

// Robust bilinear map: v0 + xi (v1-v0) + eta (v3-v0) + xi eta (v0-v1+v2-v3); exact for
// faces lying in a grid plane (the form the oracle uses).
template <typename T>
__device__ __forceinline__ T bilin(const T* v, T xi, T eta) {
    const T a = v[1] - v[0], b = v[3] - v[0], c = (v[0] - v[1]) + (v[2] - v[3]);
    return v[0] + xi * a + eta * b + (xi * eta) * c;
}

template <typename T>
struct FaceGeom {
    T x[4], y[4], z[4];   // backtraced vertex coordinates in face order
};

// centroid and area of a polygon in (xi,eta) (facecutter.h:226-253)
template <typename T>
__device__ __forceinline__ void centroid(const T* px, const T* py, int num, T& cx, T& cy, T& area) {
    T a = T(0), sx = T(0), sy = T(0);
    for (int n = 0; n < num; ++n) {
        const int m = (n + 1 == num) ? 0 : n + 1;
        const T c = px[n] * py[m] - px[m] * py[n];
        a += c;
        sx += c * (px[n] + px[m]);
        sy += c * (py[n] + py[m]);
    }
    a = fabs(T(0.5) * a);
    if (a != T(0)) {
        const T s = T(1.0) / (T(6.0) * a);
        cx = sx * s; cy = sy * s;
    } else {
        sx = T(0); sy = T(0);
        for (int n = 0; n < num; ++n) { sx = sx + px[n]; sy = sy + py[n]; }
        const T s = T(1.0) / T(num);
        cx = sx * s; cy = sy * s;
    }
    area = a;
}

// 3D centroid and the y component of the scaled normal of an emitted piece (xi-eta polygon
// px/py with centroid (cxi, ceta); split_face_3D.cpp:67-93)
template <typename T>
__device__ __forceinline__ void piece_geom(const FaceGeom<T>& g, const T* px, const T* py, int num, T cxi, T ceta,
                                           T& cx, T& cy, T& cz, T& ny) {
    cx = bilin(g.x, cxi, ceta); cy = bilin(g.y, cxi, ceta); cz = bilin(g.z, cxi, ceta);
    if (num == 3) {
        const T ax = bilin(g.x, px[1], py[1]) - bilin(g.x, px[0], py[0]);
        const T az = bilin(g.z, px[1], py[1]) - bilin(g.z, px[0], py[0]);
        const T bx = bilin(g.x, px[2], py[2]) - bilin(g.x, px[0], py[0]);
        const T bz = bilin(g.z, px[2], py[2]) - bilin(g.z, px[0], py[0]);
        ny = T(0.5) * (az * bx - ax * bz);
    } else {
        T acc = T(0);
        T x0 = bilin(g.x, px[0], py[0]) - cx, z0 = bilin(g.z, px[0], py[0]) - cz;
        const T xs = x0, zs = z0;
        for (int n = 0; n < num; ++n) {
            T x1, z1;
            if (n + 1 == num) { x1 = xs; z1 = zs; }
            else { x1 = bilin(g.x, px[n + 1], py[n + 1]) - cx; z1 = bilin(g.z, px[n + 1], py[n + 1]) - cz; }
            acc += z0 * x1 - x0 * z1;
            x0 = x1; z0 = z1;
        }
        ny = acc * T(0.5);
    }
}

// The quadrature of one piece with centroid (cx, cy, cz) and y-normal ny (polygon_3D.cpp:257-487),
// every value interpolated on its own.
template <typename T>
__device__ __forceinline__ T piece_quad(const PassDesc& d, T cx, T cy, T cz, T ny, const T* __restrict__ a,
                                        const T* __restrict__ psi) {
    if (ny == T(0)) return T(0);
    const T h = T(d.h);
    T F = T(0);
    if (d.use_integral) {
        // polygon_3D.cpp:257-487 with the grid origin shifted by -h/2 along a staggered axis
        const T oy = (d.comp == 1) ? T(-1) * T(0.5) * h : T(0);
        const T ry = snap_int((cy - oy) / h);
        const int iy0 = (int)floor(ry);
        const T f = ry - T(iy0);
        if (f < T(0.5)) {
            const T lo = T(iy0) * h + oy, L = cy - lo;
            for (int q = 0; q < d.k; ++q) {
                const T yq = (L / T(2)) * T(d.gx[q]) + (L / T(2)) + lo;
                F += interp_c(d, d.interp, a, d.A, h, cx, yq, cz) * (ny * f * h * T(d.gw[q]));
            }
        } else {
            T lo = T(iy0) * h + oy, hi = (T(iy0) + T(0.5)) * h + oy, L = hi - lo;
            for (int q = 0; q < d.k; ++q) {
                const T yq = (L / T(2)) * T(d.gx[q]) + (L / T(2)) + lo;
                F += interp_c(d, d.interp, a, d.A, h, cx, yq, cz) * (ny * T(0.5) * h * T(d.gw[q]));
            }
            lo = (T(iy0) + T(0.5)) * h + oy; hi = (T(iy0) + f) * h + oy; L = hi - lo;
            for (int q = 0; q < d.k; ++q) {
                const T yq = (L / T(2)) * T(d.gx[q]) + (L / T(2)) + lo;
                F += interp_c(d, d.interp, a, d.A, h, cx, yq, cz) * (ny * (f - T(0.5)) * h * T(d.gw[q]));
            }
        }
        F += interp_c(d, d.interp, psi, d.P, h, cx, T(iy0) * h + oy, cz) * ny;
    } else {
        F += interp_c(d, d.interp, psi, d.P, h, cx, cy, cz) * ny;
    }
    return F;
}

// Accumulates the flux of one emitted piece (xi-eta polygon px/py with centroid c) and its
// volume point y n_y (polygon_3D.cpp:480-486).
template <typename T>
__device__ __forceinline__ T piece_flux(const PassDesc& d, const FaceGeom<T>& g, const T* px, const T* py,
                                        int num, T cxi, T ceta, const T* __restrict__ a,
                                        const T* __restrict__ psi, T* vol) {
    T cx, cy, cz, ny;
    piece_geom(g, px, py, num, cxi, ceta, cx, cy, cz, ny);
    if (vol) *vol += cy * ny;
    return piece_quad(d, cx, cy, cz, ny, a, psi);
}

// What the clipper does with each emitted piece: the per-face kernel evaluates it at once
// (EvalPiece), the piece pipeline stores it (StorePiece, below).
template <typename T>
struct EvalPiece {
    const PassDesc& d;
    const T* __restrict__ a;
    const T* __restrict__ psi;
    T* vol;
    __device__ __forceinline__ T operator()(const FaceGeom<T>& g, const T* px, const T* py, int num, T cxi,
                                            T ceta) const {
        return piece_flux(d, g, px, py, num, cxi, ceta, a, psi, vol);
    }
};

// Emits a polygon (optionally triangulated to minimal_area, facecutter.h:255-324).
template <typename T, class Emit>
__device__ T emit_polygon(const PassDesc& d, const FaceGeom<T>& g, const T* px, const T* py, int num,
                          const Emit& emit, unsigned& st, int& npieces) {
    T cx, cy, area;
    centroid(px, py, num, cx, cy, area);
    const T minA = T(d.minimal_area);
    if (!(area > minA)) {
        if (area != T(0)) { ++npieces; return emit(g, px, py, num, cx, cy); }
        return T(0);
    }
    // triangulate: fan from the centroid (num > 3) then recursive longest-edge bisection
    T F = T(0);
    T tri[24][6];
    int top = 0;
    if (num == 3) {
        tri[top][0] = px[0]; tri[top][1] = py[0]; tri[top][2] = px[1]; tri[top][3] = py[1];
        tri[top][4] = px[2]; tri[top][5] = py[2]; ++top;
    } else {
        for (int n = num - 1; n >= 0; --n) {
            const int m = (n + 1 == num) ? 0 : n + 1;
            if (top >= 24) { st |= ST_SUBDIV_OVERFLOW; return F; }
            tri[top][0] = cx; tri[top][1] = cy; tri[top][2] = px[n]; tri[top][3] = py[n];
            tri[top][4] = px[m]; tri[top][5] = py[m]; ++top;
        }
    }
    while (top > 0) {
        --top;
        T tx[3] = {tri[top][0], tri[top][2], tri[top][4]};
        T ty[3] = {tri[top][1], tri[top][3], tri[top][5]};
        T tcx, tcy, tarea;
        centroid(tx, ty, 3, tcx, tcy, tarea);
        if (tarea > minA) {
            // the first of the longest edges, lengths within kLongestEdgeTie counting as equal
            int mi = 0; T ml = T(-1);
            for (int n = 0; n < 3; ++n) {
                const int m = (n + 1) % 3;
                const T len = (tx[n] - tx[m]) * (tx[n] - tx[m]) + (ty[n] - ty[m]) * (ty[n] - ty[m]);
                if (len > ml * T(1.0 + kLongestEdgeTie)) { ml = len; mi = n; }
            }
            const int i1 = (mi + 1) % 3, i2 = (mi + 2) % 3;
            const T mx = T(0.5) * (tx[mi] + tx[i1]), my = T(0.5) * (ty[mi] + ty[i1]);
            if (top + 2 > 24) { st |= ST_SUBDIV_OVERFLOW; return F; }
            // push second half first so the first half is processed first
            tri[top][0] = mx; tri[top][1] = my; tri[top][2] = tx[i1]; tri[top][3] = ty[i1];
            tri[top][4] = tx[i2]; tri[top][5] = ty[i2]; ++top;
            tri[top][0] = tx[mi]; tri[top][1] = ty[mi]; tri[top][2] = mx; tri[top][3] = my;
            tri[top][4] = tx[i2]; tri[top][5] = ty[i2]; ++top;
        } else if (tarea != T(0)) {
            ++npieces;
            F += emit(g, tx, ty, 3, tcx, tcy);
        }
    }
    return F;
}

// Finite doubles ordered as integers, both zeros alike: the clipper's ranges and sides are comparisons,
// which as FP64 instructions take the pipe that bounds it (83% busy).  With them as integers, and one
// launch for the three families, the clip of a 64^3 step takes 4.5 ms, 5.4 without.
__device__ __forceinline__ long long order_key(double c) {
    long long b = __double_as_longlong(c);
    if (b == (long long)0x8000000000000000ULL) b = 0;
    return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double key_value(long long k) {
    return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffLL));
}

// Clips one face and returns its flux (sum over pieces of the quadrature terms).
// `multi` is set when some iso-line crosses a piece more than twice: the piece that holds
// the first vertex then merges several disjoint parts (facecutter.h:163-181), so the
// partition depends on the vertex order and the two adjacent cells see different pieces.
template <typename T, class Emit>
__device__ T clip_face(const PassDesc& d, const FaceGeom<T>& g, const Emit& emit, unsigned& st, int& npieces,
                       bool& multi) {
    const T h = T(d.h);
    CV<T> pool[kPool];
    unsigned char sstart[kMaxStack], snum[kMaxStack], sdim[kMaxStack];
    int sp = 0, top = 4;
    const T xi[4] = {T(0), T(1), T(1), T(0)}, eta[4] = {T(0), T(0), T(1), T(1)};
    bool finite = true;
    for (int q = 0; q < 4; ++q) {
        pool[q].p0 = xi[q]; pool[q].p1 = eta[q];
        pool[q].c0 = snap_int(g.x[q] / h - T(d.color_off[0]));
        pool[q].c1 = snap_int(g.z[q] / h - T(d.color_off[1]));
        finite = finite && isfinite(pool[q].c0) && isfinite(pool[q].c1) && isfinite(g.y[q]);
    }
    // every cut narrows the range of a polygon's finite colours, which bounds the loop below;
    // a face with a non-finite vertex (NaN or infinite velocity upstream) is not clipped
    if (!finite) { st |= ST_NONFINITE; return T(0); }
    sstart[0] = 0; snum[0] = 4; sdim[0] = 0; sp = 1;
    T F = T(0);
    CV<T> tmp0[kMaxVerts + 2];
    while (sp > 0) {
        --sp;
        const int pstart = sstart[sp], num = snum[sp], dim = sdim[sp];
        const CV<T>* poly = pool + pstart;
        long long kmn = order_key(cv_c(poly[0], dim)), kmx = kmn;
        for (int n = 1; n < num; ++n) {
            const long long c = order_key(cv_c(poly[n], dim));
            kmn = min(kmn, c); kmx = max(kmx, c);
        }
        const T mn = key_value(kmn), mx = key_value(kmx);
        int start = (int)ceil(mn), end = (int)floor(mx);
        if (mn - T(start) == T(0)) start += 1;
        if (mx - T(end) == T(0)) end -= 1;
        bool cut = false;
        if (start <= end) {
            if (pstart + 3 * num + 2 > kPool) { st |= ST_CLIP_OVERFLOW; top = pstart; continue; }
            const T iso = T(start);
            int h0 = 0, h1 = 0, slot = 0;
            int wpos = pstart + num;          // pieces on the far side are written here
            int p1start = wpos;
            int nchild = 0;
            unsigned char cst[kMaxStack], cnum[kMaxStack];
            tmp0[h0++] = poly[0];
            bool bad = false;
            const long long kiso = order_key(iso);
            const bool below0 = order_key(cv_c(poly[0], dim)) < kiso;
            bool below = below0;
            for (int n = 0; n < num && !bad; ++n) {
                const int m = (n + 1 == num) ? 0 : n + 1;
                const bool belowm = m == 0 ? below0 : order_key(cv_c(poly[m], dim)) < kiso;
                const bool crossed = below != belowm;
                below = belowm;
                if (crossed) {
                    const T v0 = cv_c(poly[n], dim) - iso, v1 = cv_c(poly[m], dim) - iso;
                    const T inv = T(1.0) / (v1 - v0);
                    const T t0 = v1 * inv, t1 = -v0 * inv;
                    cut = true;
                    CV<T> X;
                    X.p0 = t0 * poly[n].p0 + t1 * poly[m].p0;
                    X.p1 = t0 * poly[n].p1 + t1 * poly[m].p1;
                    const T other = snap_int(t0 * cv_c(poly[n], 1 - dim) + t1 * cv_c(poly[m], 1 - dim));
                    if (dim == 0) { X.c0 = iso; X.c1 = other; } else { X.c1 = iso; X.c0 = other; }
                    if (slot == 0) {
                        tmp0[h0++] = X;
                        slot = 1; h1 = 0; p1start = wpos;
                        if (t1 < T(1.0)) pool[p1start + h1++] = X;
                    } else {
                        pool[p1start + h1++] = X;
                        if (nchild >= kMaxStack - 1) { bad = true; break; }
                        cst[nchild] = (unsigned char)p1start; cnum[nchild] = (unsigned char)h1; ++nchild;
                        wpos = p1start + h1;
                        slot = 0;
                        if (t1 < T(1.0)) tmp0[h0++] = X;
                    }
                }
                if (n < num - 1) {
                    if (slot == 0) tmp0[h0++] = poly[m];
                    else pool[p1start + h1++] = poly[m];
                }
                if (h0 >= kMaxVerts || h1 >= kMaxVerts || p1start + h1 + 2 >= kPool) bad = true;
            }
            if (bad) { st |= ST_CLIP_OVERFLOW; top = pstart; continue; }
            if (nchild > 1) multi = true;
            if (cut) {
                if (slot != 0) { st |= ST_CLIP_ODD_CUT; top = pstart; continue; }
                if (wpos + h0 >= kPool || sp + nchild + 1 > kMaxStack) { st |= ST_CLIP_OVERFLOW; top = pstart; continue; }
                // piece 0 goes after the far-side pieces; then the block moves down over the parent
                for (int q = 0; q < h0; ++q) pool[wpos + q] = tmp0[q];
                const int src = pstart + num, len = wpos + h0 - src;
                for (int q = 0; q < len; ++q) pool[pstart + q] = pool[src + q];
                for (int c = 0; c < nchild; ++c) {
                    sstart[sp] = (unsigned char)(cst[c] - num); snum[sp] = cnum[c]; sdim[sp] = (unsigned char)dim; ++sp;
                }
                sstart[sp] = (unsigned char)(wpos - num); snum[sp] = (unsigned char)h0; sdim[sp] = (unsigned char)dim; ++sp;
                top = pstart + len;
            }
        }
        if (!cut) {
            if (dim == 0) {
                sstart[sp] = (unsigned char)pstart; snum[sp] = (unsigned char)num; sdim[sp] = 1; ++sp;
                top = pstart + num;
            } else {
                if (num >= 3) {
                    T px[kMaxVerts], py[kMaxVerts];
                    for (int q = 0; q < num; ++q) { px[q] = poly[q].p0; py[q] = poly[q].p1; }
                    F += emit_polygon(d, g, px, py, num, emit, st, npieces);
                }
                top = pstart;
            }
        }
    }
    (void)top;
    return F;
}

// Face families: 0 = faces normal to x, 1 = normal to y, 2 = normal to z, in the vertex
// order of the face as seen from the lower cell (faces 1, 2, 5 of
// backtrace_..._for_integrate_density.cpp:83-112).
__device__ __forceinline__ void face_corners(int fam, int i, int j, int k, int* ci, int* cj, int* ck) {
    if (fam == 0) {
        ci[0] = i; cj[0] = j;     ck[0] = k;
        ci[1] = i; cj[1] = j + 1; ck[1] = k;
        ci[2] = i; cj[2] = j + 1; ck[2] = k + 1;
        ci[3] = i; cj[3] = j;     ck[3] = k + 1;
    } else if (fam == 1) {
        ci[0] = i;     cj[0] = j; ck[0] = k;
        ci[1] = i;     cj[1] = j; ck[1] = k + 1;
        ci[2] = i + 1; cj[2] = j; ck[2] = k + 1;
        ci[3] = i + 1; cj[3] = j; ck[3] = k;
    } else {
        ci[0] = i;     cj[0] = j;     ck[0] = k;
        ci[1] = i + 1; cj[1] = j;     ck[1] = k;
        ci[2] = i + 1; cj[2] = j + 1; ck[2] = k;
        ci[3] = i;     cj[3] = j + 1; ck[3] = k;
    }
}

// the four corners of face id of family fam: backtraced (verts) or at rest
template <typename T>
__device__ __forceinline__ void face_geom(const PassDesc& d, int fam, long long id, const T* __restrict__ verts,
                                          FaceGeom<T>& g) {
    const int Fy = d.A.My + (fam == 1), Fz = d.A.Mz + (fam == 2);
    const int k = (int)(id % Fz);
    const int j = (int)((id / Fz) % Fy);
    const int i = (int)(id / ((long long)Fz * Fy));
    int ci[4], cj[4], ck[4];
    face_corners(fam, i, j, k, ci, cj, ck);
    const int Ly = d.A.My + 1, Lz = d.A.Mz + 1;
    for (int q = 0; q < 4; ++q) {
        if (d.zero_velocity) {
            T p[3];
            vertex_rest_position(d, ci[q], cj[q], ck[q], p);
            g.x[q] = p[0]; g.y[q] = p[1]; g.z[q] = p[2];
        } else {
            const long long vid = ((long long)ci[q] * Ly + cj[q]) * Lz + ck[q];
            g.x[q] = verts[3 * vid]; g.y[q] = verts[3 * vid + 1]; g.z[q] = verts[3 * vid + 2];
        }
    }
}

// the upper cell's own face: vertex order (v0, v3, v2, v1), which is the reference's x-/y-/z-
// face order (backtrace_..._for_integrate_density.cpp:77-112)
template <typename T>
__device__ __forceinline__ FaceGeom<T> upper_face(const FaceGeom<T>& g) {
    FaceGeom<T> r = g;
    r.x[1] = g.x[3]; r.y[1] = g.y[3]; r.z[1] = g.z[3];
    r.x[3] = g.x[1]; r.y[3] = g.y[1]; r.z[3] = g.z[1];
    return r;
}

// The flux of face id of family fam, clipped and integrated piece by piece as the clipper emits
// them: flux = wgt * F (acc = 0) or flux + wgt * F (acc = 1) -- the weighted faces of the flux
// MacCormack scheme accumulate into one flux per face (wgt = 1, acc = 0 otherwise).
template <typename T>
__device__ __forceinline__ void face_eval(const PassDesc& d, int fam, long long id, const T* __restrict__ a,
                                          const T* __restrict__ psi, const T* __restrict__ verts,
                                          T* __restrict__ flux, T* __restrict__ flux_rev, T wgt, int acc,
                                          T* __restrict__ fvol, T* __restrict__ fvol_rev, unsigned& st,
                                          int& npieces, int& nmulti) {
    FaceGeom<T> g;
    face_geom(d, fam, id, verts, g);
    bool multi = false;
    T V = T(0), Vr = T(0);
    const T F = clip_face(d, g, EvalPiece<T>{d, a, psi, fvol ? &V : nullptr}, st, npieces, multi);
    T Fr = -F;
    Vr = -V;
    if (multi) {
        const FaceGeom<T> r = upper_face(g);
        int np2 = 0; bool m2 = false;
        Vr = T(0);
        Fr = clip_face(d, r, EvalPiece<T>{d, a, psi, fvol ? &Vr : nullptr}, st, np2, m2);
        ++nmulti;
    }
    if (!isfinite(F) || !isfinite(Fr)) st |= ST_NONFINITE;
    flux[id] = acc ? flux[id] + wgt * F : wgt * F;
    flux_rev[id] = acc ? flux_rev[id] + wgt * Fr : wgt * Fr;
    if (fvol) {
        fvol[id] = acc ? fvol[id] + wgt * V : wgt * V;
        fvol_rev[id] = acc ? fvol_rev[id] + wgt * Vr : wgt * Vr;
    }
}

template <typename T>
__global__ void __launch_bounds__(128) k_faces(PassDesc d, int fam, const T* __restrict__ a,
                                               const T* __restrict__ psi, const T* __restrict__ verts,
                                               T* __restrict__ flux, T* __restrict__ flux_rev,
                                               unsigned* status, unsigned long long* counters, T wgt, int acc,
                                               T* __restrict__ fvol, T* __restrict__ fvol_rev) {
    const int Fx = d.A.Mx + (fam == 0), Fy = d.A.My + (fam == 1), Fz = d.A.Mz + (fam == 2);
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long nface = (long long)Fx * Fy * Fz;
    unsigned st = 0;
    int npieces = 0, nmulti = 0;
    if (id < nface) face_eval(d, fam, id, a, psi, verts, flux, flux_rev, wgt, acc, fvol, fvol_rev, st, npieces, nmulti);
    // warp-aggregated counters and status
    unsigned long long pc = (unsigned long long)npieces;
    unsigned fc = id < nface ? 1u : 0u, mc = (unsigned)nmulti;
    for (int o = 16; o > 0; o >>= 1) {
        pc += __shfl_down_sync(0xffffffffu, pc, o);
        fc += __shfl_down_sync(0xffffffffu, fc, o);
        mc += __shfl_down_sync(0xffffffffu, mc, o);
        st |= __shfl_down_sync(0xffffffffu, st, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (fc) { atomicAdd(&counters[0], (unsigned long long)fc); atomicAdd(&counters[1], pc); }
        if (mc) atomicAdd(&counters[2], (unsigned long long)mc);
        if (st) atomicOr(status, st);
    }
}

// ------------------------------------------------------------------------------------
// The plain form's piece pipeline: k_clip64 (one thread per face: the clip, its pieces
// appended contiguously per face), k_quad64 (one thread per piece: the quadrature) and
// k_facesum64 (one thread per face: its pieces' fluxes summed in emission order).  The clip,
// the per-piece arithmetic and the order of every sum are those of k_faces, which evaluates
// each piece as the clipper emits it: there the lanes of a warp wait for the face with the
// most pieces (a third of them active on average); here each lane has one piece.
// ------------------------------------------------------------------------------------
constexpr int kMaxPieces64 = 64;   // pieces of one face, both clips (as the FP32 store)

struct StorePiece64 {
    double4_32a* p;
    int* n;
    bool* spill;   // the face has more pieces than the buffer: it is evaluated by k_faces_deferred64
    __device__ __forceinline__ double operator()(const FaceGeom<double>& g, const double* px, const double* py, int num,
                                                 double cxi, double ceta) const {
        if (*n >= kMaxPieces64) { *spill = true; return 0.0; }
        double cx, cy, cz, ny;
        piece_geom(g, px, py, num, cxi, ceta, cx, cy, cz, ny);
        p[(*n)++] = make_double4_32a(cx, cy, cz, ny);
        return 0.0;
    }
};

__device__ __forceinline__ int2* range64(const PieceStore64& ps, int fam) {
    return fam == 0 ? ps.range[0] : (fam == 1 ? ps.range[1] : ps.range[2]);
}

__global__ void __launch_bounds__(128) k_clip64(PassDesc d, FamilyBlocks fb, const double* __restrict__ verts, PieceStore64 ps,
                                                unsigned* status, unsigned long long* counters) {
    const int fam = fb.family(blockIdx.x);
    const long long nface = family_faces(d, fam);
    const long long id = (long long)(blockIdx.x - fb.start(fam)) * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    unsigned st = 0;
    int npieces = 0, n = 0, nfwd = 0;
    bool multi = false, spill = false;
    double4_32a buf[kMaxPieces64];
    if (id < nface) {
        FaceGeom<double> g;
        face_geom(d, fam, id, verts, g);
        clip_face(d, g, StorePiece64{buf, &n, &spill}, st, npieces, multi);
        nfwd = n;
        if (multi) {
            int np2 = 0;
            bool m2 = false;
            clip_face(d, upper_face(g), StorePiece64{buf, &n, &spill}, st, np2, m2);
        }
        if (spill) {
            // too many pieces for the buffer (triangulated faces at high CFL): the face is
            // listed and evaluated as a whole by k_faces_deferred64
            n = 0;
            ps.deferred[atomicAdd(ps.count + 1, 1u)] = (fam << 29) | (int)id;
        }
    }
    const long long start = warp_slots(ps.count, n, lane);
    if (id < nface) {
        // a range beyond the capacity is kept as it is: the host sees the count, grows the
        // store and clips again
        if (start + n <= ps.cap)
            for (int q = 0; q < n; ++q) ps.rec[start + q] = buf[q];
        range64(ps, fam)[id] = spill ? make_int2(-1, 0)
                                     : make_int2((int)start, nfwd | ((n - nfwd) << 15) | ((multi ? 1 : 0) << 30));
    }
    unsigned long long pc = (unsigned long long)npieces;
    unsigned fc = id < nface ? 1u : 0u, mc = multi ? 1u : 0u;
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

constexpr int kQuad64Threads = 128;
constexpr int kQuad64Group = 3;   // Gauss points of a half that share their y-stencil data

// One record per node row and stencil base of a field (fia_weno_rec.cuh), of the advected field and
// of psi alike.
__global__ void k_records64(NodeField F, const double* __restrict__ field, WenoRec<double>* __restrict__ rec) {
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= weno_rec_count(F)) return;
    const long long row = id / (F.Mz + 1);
    const int b = (int)(id - row * (F.Mz + 1)) - 1;
    double f[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) f[i] = __ldg(field + row * F.Mz + clampi(b - 2 + i, F.Mz - 1));
    rec[id] = weno_record(f[2], f[1] - f[0], f[2] - f[1], f[3] - f[2], f[4] - f[3], f[5] - f[4]);
}

// stencil base and offset of a position (in cells from node 0) along one axis; a position within
// rounding of a node sits on it
__device__ __forceinline__ int base64(double r, double& s) {
    const double sn = snap_int(r);
    const int b = sn == rint(sn) ? (int)sn : (int)floor(r);
    s = r - double(b);
    return b;
}

// What a z-interpolation at stencil base b1 - 1 of a row needs: from the field's records, or, in a session
// that has no memory for them, from the six samples (a density step at 40^3: 6.5 and 9.1 ms; 20.7
// before there were records).
struct RowRecords {
    const WenoRec<double>* __restrict__ r;
    int Mz;
    __device__ __forceinline__ WenoData<double> data(int row, int b1) const {
        return weno_unpack(ldg_rec(r + (long long)row * (Mz + 1) + b1));
    }
};
struct RowSamples {
    const double* __restrict__ a;
    int Mz;
    __device__ __forceinline__ WenoData<double> data(int row, int b1) const {
        double f[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) f[i] = __ldg(a + (long long)row * Mz + clampi(b1 - 3 + i, Mz - 1));
        return weno_data(f);
    }
};

// WENO6 of row (., j) at (x, z): 7 evaluations
template <class Rows>
__device__ __forceinline__ double row64(const Rows& rows, const NodeField& F, int bx, int b1, int j,
                                        const WenoPos<double>& pz, const WenoPos<double>& px) {
    double xv[6];
#pragma unroll 1
    for (int ix = 0; ix < 6; ++ix) xv[ix] = weno_at(rows.data(clampi(bx - 2 + ix, F.Mx - 1) * F.My + j, b1), pz);
    return weno_at(weno_data(xv), px);
}

// piece_quad with WENO6: the z-pass of the 6 x 7 (x, y) stencil rows into the
// thread's column zs, then, for each half of the cell below the centroid, the y-stencils' data
// once for its Gauss points (as piece_quad32, fia_advect32.cu).  Bound by the FP64 pipe, and so by
// its count of FP64 instructions: about 2400 a piece against 6500 with every 1D interpolant
// formed from its samples; three passes of a 64^3 density step 51.1 -> 13.6 ms.
template <class Rows>
__device__ __forceinline__ double piece_quad64(const PassDesc& d, double cx, double cy, double cz, double ny,
                                               const Rows& arec, const Rows& prec, const double* __restrict__ psi,
                                               double* zs) {
    const double h = d.h;
    double sx, sz;
    const int bx = base64((cx - d.A.ox * h) / h, sx);
    const int b1 = clampi(base64((cz - d.A.oz * h) / h, sz) + 1, d.A.Mz);
    const WenoPos<double> px = weno_pos(sx), pz = weno_pos(sz);
    if (!d.use_integral) {
        double sy;
        const int by = base64((cy - d.P.oy * h) / h, sy);
        if (fabs(sy) < 1e-9 && snap_int((cy - d.P.oy * h) / h) == double(by))   // a face at rest
            return row64(prec, d.P, bx, b1, clampi(by, d.P.My - 1), pz, px) * ny;
        return weno6_3d_collapse(psi, d.P, h, cx, cy, cz) * ny;
    }
    const double oy = (d.comp == 1) ? -0.5 * h : 0.0;
    const double ry = snap_int((cy - oy) / h);
    const int iy0 = (int)floor(ry);
    const double f = ry - double(iy0);
    const bool two = !(f < 0.5);
#pragma unroll 1
    for (int ix = 0; ix < 6; ++ix) {
        const int row0 = clampi(bx - 2 + ix, d.A.Mx - 1) * d.A.My;
#pragma unroll 1
        for (int r = 0; r < 7; ++r) {
            zs[(7 * ix + r) * kQuad64Threads] = weno_at(arec.data(row0 + clampi(iy0 - 3 + r, d.A.My - 1), b1), pz);
        }
    }
    const int k = d.k;
    double F = 0.0;
#pragma unroll 1
    for (int half = 0; half < (two ? 2 : 1); ++half) {
        const double len = half ? f - 0.5 : (two ? 0.5 : f);   // of the interval, in cells
        const double s0 = half ? 0.0 : 0.5;                    // its lower end past the third row of its stencil
        const double wf = ny * len * h;
#pragma unroll 1
        for (int q0 = 0; q0 < k; q0 += kQuad64Group) {
            const int n = min(kQuad64Group, k - q0);
            double s[kQuad64Group], yv[kQuad64Group][6];
#pragma unroll
            for (int q = 0; q < kQuad64Group; ++q) s[q] = s0 + (0.5 * len) * (d.gx[q < n ? q0 + q : q0] + 1.0);
#pragma unroll
            for (int ix = 0; ix < 6; ++ix) {
                double v[6];
#pragma unroll
                for (int i = 0; i < 6; ++i) v[i] = zs[(7 * ix + i + half) * kQuad64Threads];
                const WenoData<double> w = weno_data(v);
#pragma unroll
                for (int q = 0; q < kQuad64Group; ++q)
                    if (q < n) yv[q][ix] = weno_at(w, weno_pos(s[q]));
            }
#pragma unroll
            for (int q = 0; q < kQuad64Group; ++q)
                if (q < n) F += weno_at(weno_data(yv[q]), px) * (wf * d.gw[q0 + q]);
        }
    }
    return F + row64(prec, d.P, bx, b1, clampi(iy0, d.P.My - 1), pz, px) * ny;
}

// a piece's flux takes the place of its centroid's x
__global__ void __launch_bounds__(kQuad64Threads) k_quad64(PassDesc d, const double* __restrict__ a,
                                                           const double* __restrict__ psi, PieceStore64 ps,
                                                           long long npc) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < npc; t += (long long)gridDim.x * blockDim.x) {
        const double4_32a p = ps.rec[t];
        ps.rec[t].x = piece_quad(d, p.x, p.y, p.z, p.w, a, psi);
    }
}
template <class Rows>
__global__ void __launch_bounds__(kQuad64Threads) k_quad64_weno(PassDesc d, Rows arec, Rows prec,
                                                                const double* __restrict__ psi, PieceStore64 ps,
                                                                long long npc) {
    __shared__ double zcol[42 * kQuad64Threads];   // each thread's z-pass column
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < npc; t += (long long)gridDim.x * blockDim.x) {
        const double4_32a p = ps.rec[t];
        ps.rec[t].x = p.w == 0.0 ? 0.0 : piece_quad64(d, p.x, p.y, p.z, p.w, arec, prec, psi, zcol + threadIdx.x);
    }
}

__global__ void k_facesum64(PassDesc d, int fam, PieceStore64 ps, double* __restrict__ flux,
                            double* __restrict__ flux_rev, unsigned* status, double wgt, int acc,
                            double* __restrict__ fvol, double* __restrict__ fvol_rev) {
    const long long nface = (long long)(d.A.Mx + (fam == 0)) * (d.A.My + (fam == 1)) * (d.A.Mz + (fam == 2));
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= nface) return;
    const int2 r = range64(ps, fam)[id];
    if (r.x < 0) return;   // a listed face: k_faces_deferred64 writes it
    const int nf = r.y & 0x7fff, nr = (r.y >> 15) & 0x7fff;
    const bool multi = (r.y >> 30) & 1;
    double F = 0.0, V = 0.0;
    for (int q = 0; q < nf; ++q) {
        F += ps.rec[(long long)r.x + q].x;
        if (fvol) { const double4_32a p = ps.rec[(long long)r.x + q]; V += p.y * p.w; }
    }
    double Fr = -F, Vr = -V;
    if (multi) {
        Fr = 0.0; Vr = 0.0;
        for (int q = nf; q < nf + nr; ++q) {
            Fr += ps.rec[(long long)r.x + q].x;
            if (fvol) { const double4_32a p = ps.rec[(long long)r.x + q]; Vr += p.y * p.w; }
        }
    }
    if (!isfinite(F) || !isfinite(Fr)) atomicOr(status, (unsigned)ST_NONFINITE);
    flux[id] = acc ? flux[id] + wgt * F : wgt * F;
    flux_rev[id] = acc ? flux_rev[id] + wgt * Fr : wgt * Fr;
    if (fvol) {
        fvol[id] = acc ? fvol[id] + wgt * V : wgt * V;
        fvol_rev[id] = acc ? fvol_rev[id] + wgt * Vr : wgt * Vr;
    }
}

// The faces k_clip64 listed (all families), evaluated as k_faces does; their counters were
// counted by k_clip64.  Grid-stride over the list length in ps.count[1].
__global__ void __launch_bounds__(128) k_faces_deferred64(PassDesc d, const double* __restrict__ a,
                                                          const double* __restrict__ psi,
                                                          const double* __restrict__ verts, PieceStore64 ps,
                                                          double* fx, double* fy, double* fz, double* rx, double* ry,
                                                          double* rz, unsigned* status, double wgt, int acc,
                                                          double* vx, double* vy, double* vz, double* vrx,
                                                          double* vry, double* vrz) {
    const long long nd = (long long)ps.count[1];
    unsigned st = 0;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nd; t += (long long)gridDim.x * blockDim.x) {
        const int tag = ps.deferred[t];
        const int fam = tag >> 29;
        const long long id = tag & ((1 << 29) - 1);
        int np = 0, nm = 0;
        double* f = fam == 0 ? fx : (fam == 1 ? fy : fz);
        double* r = fam == 0 ? rx : (fam == 1 ? ry : rz);
        double* v = vx ? (fam == 0 ? vx : (fam == 1 ? vy : vz)) : nullptr;
        double* vr = vx ? (fam == 0 ? vrx : (fam == 1 ? vry : vrz)) : nullptr;
        face_eval(d, fam, id, a, psi, verts, f, r, wgt, acc, v, vr, st, np, nm);
    }
    if (st) atomicOr(status, st);
}

// rho'(i,j,k) = (Fx(i+1) + Rx(i) + Fy(j+1) + Ry(j) + Fz(k+1) + Rz(k)) / V, where F is the
// flux of a face as the lower cell's face and R as the upper cell's (R = -F unless the
// clip partition depends on the vertex order).
template <typename T>
__global__ void k_gather(PassDesc d, const T* __restrict__ fx, const T* __restrict__ fy,
                         const T* __restrict__ fz, const T* __restrict__ rx, const T* __restrict__ ry,
                         const T* __restrict__ rz, const T* __restrict__ in, T* __restrict__ out, int mode) {
    const int Mx = d.A.Mx, My = d.A.My, Mz = d.A.Mz;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)Mx * My * Mz) return;
    const int k = (int)(id % Mz);
    const int j = (int)((id / Mz) % My);
    const int i = (int)(id / ((long long)Mz * My));
    const T h = T(d.h);
    const T V = h * h * h;
    const long long ix0 = ((long long)i * My + j) * Mz + k;             // (Mx+1) x My x Mz
    const long long ix1 = ((long long)(i + 1) * My + j) * Mz + k;
    const long long iy0 = ((long long)i * (My + 1) + j) * Mz + k;       // Mx x (My+1) x Mz
    const long long iy1 = ((long long)i * (My + 1) + j + 1) * Mz + k;
    const long long iz0 = ((long long)i * My + j) * (Mz + 1) + k;       // Mx x My x (Mz+1)
    const T s = ((fx[ix1] + rx[ix0]) + (fy[iy1] + ry[iy0])) + (fz[iz0 + 1] + rz[iz0]);
    const T val = s / V;
    if (mode == 0) out[id] = val;
    else if (mode == 1) out[id] = in[id] - val;
    else if (mode == 2) out[id] = out[id] + val;
    else out[id] = s;
}

// ------------------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------------------
static inline unsigned blocks_for(long long n, int t) { return (unsigned)((n + t - 1) / t); }

template <typename T>
cudaError_t launch_psi(const PassDesc& d, const T* a, T* psi, cudaStream_t s) {
    const long long cols = (long long)d.A.Mx * d.A.Mz;
    const unsigned inc = blocks_for(cols * ((d.A.My + kPsiRun - 1) / kPsiRun), kPsiThreads);
    if (d.psi_mode == PSI_WENO6) k_psi_inc<T, PSI_WENO6><<<inc, kPsiThreads, 0, s>>>(d, a, psi);
    else if (d.psi_mode == PSI_LINEAR) k_psi_inc<T, PSI_LINEAR><<<inc, kPsiThreads, 0, s>>>(d, a, psi);
    const unsigned scan = blocks_for(cols, kScanThreads);
    if (d.psi_mode == PSI_PLAIN) k_psi_scan<T, true><<<scan, kScanThreads, 0, s>>>(d, a, psi);
    else k_psi_scan<T, false><<<scan, kScanThreads, 0, s>>>(d, a, psi);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_backtrace(const PassDesc& d, const VelocityFields& vel, T* verts, cudaStream_t s) {
    if constexpr (sizeof(T) == sizeof(double)) {
        // as in the chosen form: 8 x 8 tiles, 4 x 4 where those would leave SMs without a block
        if (d.interp == INTERP_WENO6 && !d.full_weno) {
            const int L[3] = {d.A.Mx + 1, d.A.My + 1, d.A.Mz + 1};
            const TraceTiles t8 = trace_tiles(L, 8, 16), t4 = trace_tiles(L, 4, 16);
            const bool big = 3 * trace_blocks(L, 8, t8) >= 152 * 2;
            const TraceTiles t = big ? t8 : t4;
            const dim3 g(trace_blocks(L, big ? 8 : 4, t), 3);
            const double *u = (const double*)vel.u, *v = (const double*)vel.v, *w = (const double*)vel.w;
            if (big) k_trace64<8><<<g, kTraceThreads, trace_smem(8, t, 8), s>>>(d, u, v, w, vel.fu, vel.fv, vel.fw, verts, t);
            else k_trace64<4><<<g, kTraceThreads, trace_smem(4, t, 8), s>>>(d, u, v, w, vel.fu, vel.fv, vel.fw, verts, t);
            return cudaGetLastError();
        }
    }
    const long long n = (long long)(d.A.Mx + 1) * (d.A.My + 1) * (d.A.Mz + 1);
    k_backtrace<T><<<blocks_for(n, 128), 128, 0, s>>>(d, (const T*)vel.u, (const T*)vel.v, (const T*)vel.w,
                                                      vel.fu, vel.fv, vel.fw, verts);
    return cudaGetLastError();
}

template <typename T>
static cudaError_t launch_faces_from(const PassDesc& d, const T* a, const PassWork<T>& w, const T* verts, T wgt,
                                     int acc, cudaStream_t s) {
    for (int fam = 0; fam < 3; ++fam) {
        const long long n = (long long)(d.A.Mx + (fam == 0)) * (d.A.My + (fam == 1)) * (d.A.Mz + (fam == 2));
        prof_mark(w, 0, s);
        k_faces<T><<<blocks_for(n, 128), 128, 0, s>>>(d, fam, a, w.psi, verts, w.flux[fam], w.flux_rev[fam],
                                                      w.status, w.counters, wgt, acc,
                                                      d.volumes ? w.fvol[fam] : nullptr,
                                                      d.volumes ? w.fvol_rev[fam] : nullptr);
        prof_mark(w, 1, s);
    }
    return cudaGetLastError();
}

// WENO6 from records: where the pass interpolates with it, unless every evaluation is wanted in
// full or the records found no memory (fia_create)
static bool weno_records64(const PassDesc& d, const PassWork<double>& w) {
    return w.pieces64 && w.records->field && d.interp == INTERP_WENO6 && !d.full_weno;
}

// One face stage of the piece pipeline: clip (growing the store and clipping again when it is
// too small), per-piece quadrature, per-face sums weighted into the face fluxes.
static cudaError_t face_stage64(const PassDesc& d, const double* a, const PassWork<double>& w, const double* verts,
                                double wgt, int acc, cudaStream_t s) {
    PieceStore64& ps = *w.pieces64;
    long long nface[3], big = 0;
    for (int fam = 0; fam < 3; ++fam) {
        nface[fam] = (long long)(d.A.Mx + (fam == 0)) * (d.A.My + (fam == 1)) * (d.A.Mz + (fam == 2));
        big = nface[fam] > big ? nface[fam] : big;
    }
    unsigned npc = 0;
    // the work counters as they were before the clip: a second attempt starts from them again
    cudaError_t ec = cudaMemcpyAsync(ps.saved, w.counters, 5 * sizeof(unsigned long long), cudaMemcpyDeviceToDevice, s);
    if (ec != cudaSuccess) return ec;
    for (int attempt = 0; attempt < 2; ++attempt) {
        cudaError_t e = cudaMemsetAsync(ps.count, 0, 2 * sizeof(unsigned), s);
        if (e == cudaSuccess && attempt > 0)
            e = cudaMemcpyAsync(w.counters, ps.saved, 5 * sizeof(unsigned long long), cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) return e;
        const FamilyBlocks fb = family_blocks(nface, false, 128);
        k_clip64<<<fb.first[3], 128, 0, s>>>(d, fb, verts, ps, w.status, w.counters);
        e = cudaMemcpyAsync(&npc, ps.count, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return e;
        if ((long long)npc <= ps.cap) break;
        // more pieces than the store holds: grow it and clip again
        e = piece_store64_reserve(ps, (long long)npc + npc / 4 + 1024, big, *w.records);
        if (e != cudaSuccess) return e;
    }
    if ((long long)npc > ps.cap) return cudaErrorMemoryAllocation;
    if (npc > 0) {
        const long long nb = std::min<long long>(blocks_for(npc, kQuad64Threads), 152LL * 16);
        prof_mark(w, 0, s);
        if (weno_records64(d, w))
            k_quad64_weno<<<(unsigned)nb, kQuad64Threads, 0, s>>>(d, RowRecords{(const WenoRec<double>*)w.records->field, d.A.Mz},
                                                                  RowRecords{(const WenoRec<double>*)w.records->psi, d.P.Mz}, w.psi,
                                                                  ps, (long long)npc);
        else if (d.interp == INTERP_WENO6 && !d.full_weno)
            k_quad64_weno<<<(unsigned)nb, kQuad64Threads, 0, s>>>(d, RowSamples{a, d.A.Mz}, RowSamples{w.psi, d.P.Mz}, w.psi,
                                                                  ps, (long long)npc);
        else
            k_quad64<<<(unsigned)nb, kQuad64Threads, 0, s>>>(d, a, w.psi, ps, (long long)npc);
        prof_mark(w, 1, s);
    }
    for (int fam = 0; fam < 3; ++fam)
        k_facesum64<<<blocks_for(nface[fam], 256), 256, 0, s>>>(d, fam, ps, w.flux[fam], w.flux_rev[fam], w.status, wgt,
                                                              acc, d.volumes ? w.fvol[fam] : nullptr,
                                                              d.volumes ? w.fvol_rev[fam] : nullptr);
    const bool vol = d.volumes != 0;
    k_faces_deferred64<<<152, 128, 0, s>>>(d, a, w.psi, verts, ps, w.flux[0], w.flux[1], w.flux[2], w.flux_rev[0],
                                           w.flux_rev[1], w.flux_rev[2], w.status, wgt, acc,
                                           vol ? w.fvol[0] : nullptr, vol ? w.fvol[1] : nullptr,
                                           vol ? w.fvol[2] : nullptr, vol ? w.fvol_rev[0] : nullptr,
                                           vol ? w.fvol_rev[1] : nullptr, vol ? w.fvol_rev[2] : nullptr);
    return cudaGetLastError();
}

// The piece pipeline where its face tags (family << 29 | index) hold every face; one thread
// per face otherwise (grids beyond about 800^3) and where the session has no piece store.
template <typename T>
static cudaError_t faces_weighted(const PassDesc& d, const T* a, const PassWork<T>& w, const T* verts, T wgt, int acc,
                                  cudaStream_t s) {
    if constexpr (sizeof(T) == sizeof(double)) {
        long long big = 0;
        for (int fam = 0; fam < 3; ++fam) {
            const long long nf = (long long)(d.A.Mx + (fam == 0)) * (d.A.My + (fam == 1)) * (d.A.Mz + (fam == 2));
            big = nf > big ? nf : big;
        }
        if (w.pieces64 && big < (1LL << 29)) return face_stage64(d, a, w, verts, wgt, acc, s);
    }
    return launch_faces_from<T>(d, a, w, verts, wgt, acc, s);
}

template <typename T>
cudaError_t launch_faces(const PassDesc& d, const T* a, const PassWork<T>& w, cudaStream_t s) {
    return faces_weighted<T>(d, a, w, w.verts, T(1), 0, s);
}

cudaError_t RecordStore::make(size_t field_bytes, size_t psi_bytes) {
    const size_t at = (field_bytes + 255) & ~(size_t)255;
    const cudaError_t e = cudaMalloc(&field, at + psi_bytes);
    if (e == cudaSuccess) {
        psi = (char*)field + at;
    } else {
        field = nullptr;
        cudaGetLastError();
    }
    return e;
}

cudaError_t RecordStore::alloc(void** p, size_t bytes) {
    auto get = [&] {
        if (fail > 0) {
            --fail;
            return cudaErrorMemoryAllocation;
        }
        return cudaMalloc(p, bytes);
    };
    cudaError_t e = get();
    if (e == cudaErrorMemoryAllocation && field) {
        release();
        e = get();
    }
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
    }
    return e;
}

void RecordStore::release() {
    cudaDeviceSynchronize();
    cudaFree(field);
    field = psi = nullptr;
}

cudaError_t piece_store64_reserve(PieceStore64& p, long long pieces, long long faces_per_family, RecordStore& mem) {
    cudaDeviceSynchronize();
    // ranges hold 31-bit starts
    if (pieces >= (1LL << 31)) pieces = (1LL << 31) - 1;
    if (pieces > p.cap) {
        cudaFree(p.rec);
        p.rec = nullptr; p.cap = 0;
        cudaError_t e = mem.alloc((void**)&p.rec, pieces * sizeof(double4_32a));
        if (e != cudaSuccess) return e;
        p.cap = pieces;
    }
    if (!p.count) {
        cudaError_t e = mem.alloc((void**)&p.count, 2 * sizeof(unsigned));
        if (e == cudaSuccess) e = mem.alloc((void**)&p.saved, 5 * sizeof(unsigned long long));
        if (e != cudaSuccess) return e;
    }
    if (!p.range[0]) {
        for (int f = 0; f < 3; ++f) {
            cudaError_t e = mem.alloc((void**)&p.range[f], faces_per_family * sizeof(int2));
            if (e != cudaSuccess) return e;
        }
        cudaError_t e = mem.alloc((void**)&p.deferred, 3 * faces_per_family * sizeof(int));
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void piece_store64_free(PieceStore64& p) {
    cudaFree(p.rec); cudaFree(p.count); cudaFree(p.deferred); cudaFree(p.saved);
    for (int f = 0; f < 3; ++f) cudaFree(p.range[f]);
    p = PieceStore64();
}

template <typename T>
cudaError_t launch_gather(const PassDesc& d, const PassWork<T>& w, const T* in, T* out, int mode, cudaStream_t s) {
    const long long n = (long long)d.A.Mx * d.A.My * d.A.Mz;
    k_gather<T><<<blocks_for(n, 256), 256, 0, s>>>(d, w.flux[0], w.flux[1], w.flux[2], w.flux_rev[0],
                                                   w.flux_rev[1], w.flux_rev[2], in, out, mode);
    return cudaGetLastError();
}

template <typename T>
cudaError_t run_pass(const PassDesc& d, const VelocityFields& vel, const T* a, const PassWork<T>& w,
                     const T* in, T* out, int mode, cudaStream_t s) {
    cudaError_t e = launch_psi<T>(d, a, w.psi, s);
    if (e != cudaSuccess) return e;
    if constexpr (sizeof(T) == sizeof(double)) {
        if (weno_records64(d, w)) {
            if (d.use_integral)
                k_records64<<<blocks_for(weno_rec_count(d.A), 256), 256, 0, s>>>(d.A, a, (WenoRec<double>*)w.records->field);
            k_records64<<<blocks_for(weno_rec_count(d.P), 256), 256, 0, s>>>(d.P, w.psi, (WenoRec<double>*)w.records->psi);
        }
    }
    if (!d.zero_velocity) {
        e = launch_backtrace<T>(d, vel, w.verts, s);
        if (e != cudaSuccess) return e;
    }
    if (!d.maccormack || d.zero_velocity) {
        // one face per face slot; with zero velocity the MacCormack faces coincide and their
        // weights sum to one
        e = launch_faces<T>(d, a, w, s);
    } else {
        if (!w.verts2) return cudaErrorInvalidValue;
        const long long nv = (long long)(d.A.Mx + 1) * (d.A.My + 1) * (d.A.Mz + 1);
        k_forward_trace<T><<<blocks_for(nv, 128), 128, 0, s>>>(d, (const T*)vel.u, (const T*)vel.v, (const T*)vel.w,
                                                              vel.fu, vel.fv, vel.fw, w.verts, w.verts2);
        PassDesc rest = d;
        rest.zero_velocity = 1;
        e = faces_weighted<T>(rest, a, w, w.verts, T(0.5), 0, s);            // the face at rest
        if (e == cudaSuccess) e = faces_weighted<T>(d, a, w, w.verts, T(1), 1, s);   // backtraced
        if (e == cudaSuccess) e = faces_weighted<T>(d, a, w, w.verts2, T(-0.5), 1, s);   // traced back
    }
    if (e != cudaSuccess) return e;
    if (d.volumes) {
        if (!w.vol || !w.fvol[0]) return cudaErrorInvalidValue;
        const long long n = (long long)d.A.Mx * d.A.My * d.A.Mz;
        k_gather<T><<<blocks_for(n, 256), 256, 0, s>>>(d, w.fvol[0], w.fvol[1], w.fvol[2], w.fvol_rev[0],
                                                       w.fvol_rev[1], w.fvol_rev[2], nullptr, w.vol, 3);
    }
    return launch_gather<T>(d, w, in, out, mode, s);
}

template cudaError_t launch_psi<double>(const PassDesc&, const double*, double*, cudaStream_t);
template cudaError_t launch_backtrace<double>(const PassDesc&, const VelocityFields&, double*, cudaStream_t);
template cudaError_t launch_faces<double>(const PassDesc&, const double*, const PassWork<double>&, cudaStream_t);
template cudaError_t launch_gather<double>(const PassDesc&, const PassWork<double>&, const double*, double*, int, cudaStream_t);
template cudaError_t run_pass<double>(const PassDesc&, const VelocityFields&, const double*, const PassWork<double>&,
                                      const double*, double*, int, cudaStream_t);

}  // namespace fia
