// fia_trace.cuh -- WENO6 velocities at the vertices' rest positions, a tile of vertices at a time.
//
// A vertex at rest lies on a node plane of a velocity component's lattice, or halfway between two,
// along each axis.  Along the first kind the interpolant is the node's value; along the second the
// six samples are interpolated at 1/2.  Vertex by vertex that is 21 one-dimensional evaluations for a
// density vertex (7 a component) and 45 for a velocity vertex (43 for the component itself); but
// neighbours share their inner passes.  A block takes N x N x TZ vertices of one component: the
// z-pass of all rows under the tile's stencils, the y-pass of those, the x-pass of those, each in
// shared memory, which leaves 2.6 and 5.3 evaluations a vertex and component at N = 8 (3.3 and 8.3 at 4).
// The items of a pass are dealt to the threads in one sequence, so the tile's depth TZ divides the
// vertices along z evenly instead of padding them to a warp.
//
// Bound by FP32 issue (FP64: by its pipe).  A 128^3 density pass: 391 us one vertex a thread, 132
// now; the plain form at 64^3: 1.24 ms, 0.36; a velocity pass on 120 x 161 x 77 cells 0.34 ms, 0.09.
#pragma once
#include "fia_weno_rec.cuh"

namespace fia {

constexpr int kTraceThreads = 256;

// one evaluation at a position; FP32 as weno6_eval, bit for bit
struct TraceCoef32 {
    WenoCoef<float> c;
    __device__ __forceinline__ explicit TraceCoef32(float s) {
        float t[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) t[i] = s + float(2 - i);
        c = weno_coef(t);
    }
    __device__ __forceinline__ float operator()(const float* f) const { return weno6_at(weno6_data(f), c); }
};
struct TraceCoef64 {
    WenoPos<double> p;
    __device__ __forceinline__ explicit TraceCoef64(double s) : p(weno_pos(s)) {}
    __device__ __forceinline__ double operator()(const double* f) const { return weno_at(weno_data(f), p); }
};

// tiles of N x N x tz vertices
struct TraceTiles {
    int ny, nz, tz;
};

// store(i, j, k, value) for every vertex of the tile (L: vertices along each axis, q: the rest
// position relative to the vertex's indices).  sh holds (N + 5)(2 N + 5) tz values.
template <int N, class Coef, typename T, class Store>
__device__ __forceinline__ void trace_tile(const T* __restrict__ a, const NodeField& F, const T* off, const int* L,
                                           const T* q, const TraceTiles& tiles, T* sh, Store store) {
    int b[3];        // base node of vertex 0
    T s[3];
    bool on[3];      // on a node plane
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const T r = q[c] - off[c], f = floor(r);
        b[c] = (int)f;
        s[c] = r - f;
        on[c] = s[c] == T(0);
    }
    const Coef coef(on[0] ? (on[1] ? s[2] : s[1]) : s[0]);   // every other offset is 1/2
    const unsigned t = blockIdx.x, ty = t / tiles.nz;
    const int k0 = (int)(t - ty * tiles.nz) * tiles.tz, j0 = (int)(ty % tiles.ny) * N, i0 = (int)(ty / tiles.ny) * N;
    const int nz = min(tiles.tz, L[2] - k0);
    const int ex = on[0] ? N : N + 5, ey = on[1] ? N : N + 5;   // rows under the tile
    const int rx = i0 + b[0] - (on[0] ? 0 : 2), ry = j0 + b[1] - (on[1] ? 0 : 2);
    const T* src = sh;
    // z-pass: sh[(ix ey + iy) nz + z]
    for (int e = threadIdx.x; e < ex * ey * nz; e += kTraceThreads) {
        const int r = e / nz, z = e - r * nz, ix = r / ey;
        const T* row = a + idx3(F, clampi(rx + ix, F.Mx - 1), clampi(ry + r - ix * ey, F.My - 1), 0);
        const int kb = k0 + z + b[2];
        if (on[2]) {
            sh[e] = __ldg(row + clampi(kb, F.Mz - 1));
        } else {
            T f[6];
#pragma unroll
            for (int m = 0; m < 6; ++m) f[m] = __ldg(row + clampi(kb - 2 + m, F.Mz - 1));
            sh[e] = coef(f);
        }
    }
    __syncthreads();
    // y-pass: [(ix N + j) nz + z]
    if (!on[1]) {
        T* dst = sh + ex * ey * nz;
        for (int e = threadIdx.x; e < ex * N * nz; e += kTraceThreads) {
            const int r = e / nz, z = e - r * nz, ix = r / N, j = r - ix * N;
            T f[6];
#pragma unroll
            for (int m = 0; m < 6; ++m) f[m] = sh[(ix * ey + j + m) * nz + z];
            dst[e] = coef(f);
        }
        __syncthreads();
        src = dst;
    }
    // x-pass
    for (int e = threadIdx.x; e < N * N * nz; e += kTraceThreads) {
        const int r = e / nz, z = e - r * nz, i = r / N, j = r - i * N;
        T v = src[e];
        if (!on[0]) {
            T f[6];
#pragma unroll
            for (int m = 0; m < 6; ++m) f[m] = src[e + m * N * nz];
            v = coef(f);
        }
        if (i0 + i < L[0] && j0 + j < L[1]) store(i0 + i, j0 + j, k0 + z, v);
    }
}

// tiles of n x n vertices, at most zmax deep
inline TraceTiles trace_tiles(const int* L, int n, int zmax) {
    const int nz = (L[2] + zmax - 1) / zmax, tz = (L[2] + nz - 1) / nz;
    return TraceTiles{(L[1] + n - 1) / n, (L[2] + tz - 1) / tz, tz};
}
inline unsigned trace_blocks(const int* L, int n, const TraceTiles& t) {
    return (unsigned)((L[0] + n - 1) / n) * (unsigned)t.ny * (unsigned)t.nz;
}
inline size_t trace_smem(int n, const TraceTiles& t, size_t es) { return (size_t)(n + 5) * (2 * n + 5) * t.tz * es; }

}  // namespace fia
