// Particle-to-node scatter of the reference-layout paths (plain, implicit,
// adjoint): one warp takes 32 consecutive particles of the pass.
//
// Every quantity scattered has the separable form (w = wx wy wz at node o)
//   q_r(o) = sum_a Ha_r[o_a] prod_{b != a} wb[o_b],
//   Ha_r[o] = wa[o] K(r,a) (Z_a(o) - X_a) + wa'[o] S(r,a)   (+ wx[o] c_r, a = 0),
// i.e. w (c + K (Z - X)) + S grad w.  Each lane first writes its particle's
// weights and factors to shared memory (scatter_row); then groups of 3^(d-1)
// lanes, a lane per (x, y) offset of the stencil, walk the warp's particles in
// order and sum the nodes along the last axis in registers (scatter_warp).  A
// lane goes to global memory only where the run's next particle has another
// first node: a step by one node along the last axis sends one node and shifts
// the registers, any other step sends all three.  One thread per particle
// with one atomic per node value and particle was bound by the atomics
// (FP64, 242,752 particles: P2G 165 us, forces 140 us); particles that share
// cells, as seeded or sorted ones do, now share their atomics too.  Particles in
// no order at all send as many atomics as before and are no slower: 296,352 of
// them on a 44^3 grid, P2G and forces in FP64 338 -> 301 us, in FP32 364 -> 324.
#pragma once
#include "mpm_internal.h"

namespace plain {

using namespace mpm;

constexpr int kScatterThreads = 128;   // 4 warps: 39 KB of shared memory in FP64

template<int d> struct ScatterShape {
    static constexpr int LANES = d == 3 ? 9 : 3;      // per particle
    static constexpr int GROUPS = 32 / LANES;         // particles at a time
    // weights, factors, mass; odd, so that the lanes' rows start on different banks
    static constexpr int LEN = 3 * d * (d + 1) + 1;
};

template<class T, int d> struct ScatterWarp {
    T row[32][ScatterShape<d>::LEN];
    int64_t base[32];                                 // flat index of the first node; < 0: no particle
};

// Weights, factors and mass of one particle.  K, S column-major or null (zero).
template<class T, int d> __device__ __forceinline__ void scatter_row(T* row, const Axis<T>* ax, const T* X, const double* dmin,
    const double* dx, const T* c, const T* K, const T* S, T m)
{
#pragma unroll
    for(int a = 0; a < d; a++)
#pragma unroll
        for(int o = 0; o < 3; o++) {
            const T w = ax[a].w[o];
            row[3 * a + o] = w;
            const T off = K ? w * ((T)dmin[a] + ((T)(ax[a].base + o) + (T).5) * (T)dx[a] - X[a]) : (T)0;
#pragma unroll
            for(int r = 0; r < d; r++) {
                T h = a == 0 ? w * c[r] : (T)0;
                if(K) h += off * K[r + d * a];
                if(S) h += ax[a].dw[o] * S[r + d * a];
                row[3 * d + (3 * a + o) * d + r] = h;
            }
        }
    row[ScatterShape<d>::LEN - 1] = m;
}

// Sums of the warp's particles, sent node by node: send(node, q) with q[0..d-1]
// the vector and, with MASS, q[d] the mass.  stride: flat nodes per step of axis
// 0 and, in 3D, of axis 1.
template<class T, int d, bool MASS, class SEND>
__device__ __forceinline__ void scatter_warp(const ScatterWarp<T, d>& W, int64_t stride0, int64_t stride1, SEND&& send)
{
    constexpr int LANES = ScatterShape<d>::LANES, GROUPS = ScatterShape<d>::GROUPS, LEN = ScatterShape<d>::LEN, Q = d + (MASS ? 1 : 0);
    const int lane = threadIdx.x & 31, g = lane / LANES, l = lane % LANES;
    if(g >= GROUPS) return;
    const int i = d == 3 ? l / 3 : l, j = d == 3 ? l % 3 : 0;
    const int64_t off = i * stride0 + (d == 3 ? j * stride1 : 0);
    T A[3][Q];
#pragma unroll
    for(int k = 0; k < 3; k++)
#pragma unroll
        for(int r = 0; r < Q; r++) A[k][r] = 0;
    int64_t cur = -1;
    const int p1 = 32 * (g + 1) / GROUPS;
    for(int p = 32 * g / GROUPS; p < p1; p++) {
        const int64_t b = W.base[p];
        if(b < 0) continue;
        if(b != cur) {
            if(cur >= 0) send(cur + off, A[0]);
            const bool next = cur >= 0 && b == cur + 1;
            if(cur >= 0 && !next) { send(cur + off + 1, A[1]); send(cur + off + 2, A[2]); }
#pragma unroll
            for(int r = 0; r < Q; r++) {
                A[0][r] = next ? A[1][r] : (T)0;
                A[1][r] = next ? A[2][r] : (T)0;
                A[2][r] = 0;
            }
            cur = b;
        }
        const T* row = W.row[p];
        const T wx = row[i], wxy = d == 3 ? wx * row[3 + j] : wx;
        T z[3], P[d];
#pragma unroll
        for(int k = 0; k < 3; k++) z[k] = row[3 * (d - 1) + k];
#pragma unroll
        for(int r = 0; r < d; r++) {
            const T hx = row[3 * d + i * d + r];
            P[r] = d == 3 ? hx * row[3 + j] + wx * row[3 * d + (3 + j) * d + r] : hx;
        }
#pragma unroll
        for(int k = 0; k < 3; k++) {
#pragma unroll
            for(int r = 0; r < d; r++) A[k][r] += P[r] * z[k] + wxy * row[3 * d + (3 * (d - 1) + k) * d + r];
            if(MASS) A[k][d] += row[LEN - 1] * wxy * z[k];
        }
    }
    if(cur >= 0) {
#pragma unroll
        for(int k = 0; k < 3; k++) send(cur + off + k, A[k]);
    }
}

}  // namespace plain
