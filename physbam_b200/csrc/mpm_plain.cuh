// Reference-layout kernel arguments and the particle stencil shared by the
// plain path (mpm_plain.cu) and the implicit solve (mpm_implicit.cu).
#pragma once
#include "mpm_internal.h"

namespace plain {

using namespace mpm;

template<class T> struct PlainArgs {
    SceneParams sp;
    int64_t n, gn;
    int gs[3];
    T *X, *V, *F, *B;
    const T *mass, *vol, *mu, *lam;
    T* pft;
    uint8_t* valid;
    T *gm, *gmv, *gv0, *gf, *gv, *gvf;
    // where G2P writes the particles (their own arrays, or a recorded rollout's next
    // state), and the grid update's record of mass, velocity and velocity before the
    // collision projection (null: none)
    T *oX, *oV, *oF, *oB;
    uint8_t* ovalid;
    T *rm, *rv, *ru;
    T dt;
    unsigned* flags;
    int mark_left;
    int reflect;          // reflection boundary conditions on
    int side[6];          // their types per side (mpm_bc_type)
    const ObjMotion* motion;   // moving collision objects (bit j of `moving`): their substep frames
    unsigned moving;
    const uint8_t* pmodel;     // per-particle constitutive model, or null (sp.model for all)
    const uint8_t* pmask;      // particles the plasticity acts on, or null (all)
    uint8_t* tile_flag;        // node tiles: P2G's flags, the list and its length; null: every node
    const uint32_t *tiles, *tile_count;
};

constexpr int kTileNodes = 32;

// f(i) over the nodes of the listed tiles (a warp per tile), or over all gn nodes.
template<class FN> __device__ __forceinline__ void for_tiles(int64_t gn, const uint32_t* tiles, const uint32_t* count, FN&& f)
{
    const uint32_t nt = tiles ? *count : (uint32_t)((gn + kTileNodes - 1) / kTileNodes);
    const uint32_t nw = gridDim.x * (blockDim.x >> 5);
    for(uint32_t t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < nt; t += nw) {
        const int64_t i = (int64_t)(tiles ? tiles[t] : t) * kTileNodes + (threadIdx.x & 31);
        if(i < gn) f(i);
    }
}

template<class T, class FN> __device__ __forceinline__ void for_nodes(const PlainArgs<T>& a, FN&& f)
{
    for_tiles(a.gn, a.tiles, a.tile_count, f);
}

// Grids of this many nodes and more are passed over by the list of tiles that
// P2G touched, which costs a launch and the flags.  Every node / the list, ms per call: 2D
// block, 100 substeps, 4,900 nodes 1.74 / 1.94, 39,204 1.87 / 2.15, 68,644 1.95 / 2.16;
// plain FP64 spheres, 64 substeps, 54,872 nodes 2.87 / 2.92, 74,088 2.97 / 3.01, 97,336 3.12
// / 3.09, 157,464 3.52 / 3.35, 343,000 5.6 / 4.65, 1,061,208 14.0 / 9.5; implicit substep 74,088
// 2.66 / 2.55, 343,000 3.32 / 3.07.  The line goes by the grid's size alone: bodies that
// fill the grid gain nothing from the list and pay 2 to 3 % for it (44^3 to 64^3).
constexpr int64_t kListedGrid = 90000;

inline bool list_tiles(const mpm_handle* h) { return !h->reflect.enabled && h->plain.gn >= kListedGrid; }

// The constitutive model of particle p: its own, or the handle's.
template<class T> __device__ __forceinline__ int model_of(const PlainArgs<T>& a, int64_t p)
{
    return a.pmodel ? (int)a.pmodel[p] : a.sp.model;
}

template<class T, int d> struct Stencil {
    Axis<T> ax[3];
    int base[3];
};

// Weights of one particle; returns false if the 3^d stencil leaves the ghosted grid.
template<class T, int d> __device__ bool make_stencil(const PlainArgs<T>& a, const T* X, Stencil<T, d>& s)
{
    bool ok = true;
#pragma unroll
    for(int k = 0; k < d; k++) {
        s.ax[k] = spline_axis<T>(X[k], (T)a.sp.dmin[k], (T)a.sp.dx[k], (T)a.sp.inv_dx[k]);
        s.base[k] = s.ax[k].base;
        int lo = s.base[k] + MPM_GHOST, hi = lo + 2;
        if(lo < 0 || hi >= a.gs[k]) ok = false;
    }
    return ok;
}

// Tensor-product node q (RANGE_ITERATOR order, last axis fastest):
// PARTICLE_GRID_WEIGHTS_SPLINE::Compute (PARTICLE_GRID_WEIGHTS_SPLINE.cpp:33-56).
template<class T, int d> __device__ __forceinline__ void node(const PlainArgs<T>& a, const Stencil<T, d>& s, int q,
    int64_t& flat, T& w, T* g, T* Z)
{
    int off[3];
    if(d == 3) { off[0] = q / 9; off[1] = (q / 3) % 3; off[2] = q % 3; }
    else { off[0] = q / 3; off[1] = q % 3; off[2] = 0; }
    T aw[3];
#pragma unroll
    for(int k = 0; k < d; k++) aw[k] = s.ax[k].w[off[k]];
    w = aw[0] * aw[1];
    if(d == 3) w *= aw[2];
#pragma unroll
    for(int k = 0; k < d; k++) g[k] = 1;
#pragma unroll
    for(int j = 0; j < d; j++) {
        T dj = s.ax[j].dw[off[j]];
#pragma unroll
        for(int i = 0; i < d; i++) g[i] *= i == j ? dj : aw[j];
    }
    flat = 0;
#pragma unroll
    for(int k = 0; k < d; k++) {
        int idx = s.base[k] + off[k];
        flat = flat * a.gs[k] + (idx + MPM_GHOST);
        Z[k] = (T)a.sp.dmin[k] + ((T)idx + (T).5) * (T)a.sp.dx[k];
    }
}

// Flat index of a stencil's first node, and the flat strides of axes 0 and 1.
template<class T, int d> __device__ __forceinline__ int64_t first_node(const PlainArgs<T>& a, const Stencil<T, d>& s)
{
    int64_t flat = 0;
#pragma unroll
    for(int k = 0; k < d; k++) flat = flat * a.gs[k] + (s.base[k] + MPM_GHOST);
    return flat;
}

template<class T> __device__ __forceinline__ int64_t node_stride(const PlainArgs<T>& a, int d, int axis)
{
    int64_t n = 1;
    for(int k = axis + 1; k < d; k++) n *= a.gs[k];
    return n;
}

template<class T> inline PlainArgs<T> args(mpm_handle* h, double dt)
{
    PlainArgs<T> a;
    PlainState& s = h->plain;
    a.sp = h->sp;
    a.n = s.n;
    a.gn = s.gn;
    for(int k = 0; k < 3; k++) a.gs[k] = k < h->sp.dim ? h->sp.counts[k] + 2 * MPM_GHOST : 1;
    a.X = (T*)s.X; a.V = (T*)s.V; a.F = (T*)s.F; a.B = (T*)s.B;
    a.mass = (const T*)s.mass; a.vol = (const T*)s.vol; a.mu = (const T*)s.mu; a.lam = (const T*)s.lam;
    a.pft = (T*)s.pft; a.valid = s.valid;
    a.oX = a.X; a.oV = a.V; a.oF = a.F; a.oB = a.B; a.ovalid = a.valid;
    a.rm = a.rv = a.ru = nullptr;
    if(s.record) {
        const PlainRecord& r = *s.record;
        a.X = (T*)r.in; a.V = a.X + 3 * s.n; a.F = a.X + 6 * s.n; a.B = a.X + 15 * s.n;
        a.valid = r.valid;
        a.pft = (T*)r.pft;
        if(r.out) {
            a.oX = (T*)r.out; a.oV = a.oX + 3 * s.n; a.oF = a.oX + 6 * s.n; a.oB = a.oX + 15 * s.n;
            a.ovalid = r.out_valid;
        }
        a.rm = (T*)r.gm; a.rv = (T*)r.gv; a.ru = (T*)r.gu;
    }
    a.gm = (T*)s.gm; a.gmv = (T*)s.gmv; a.gv0 = (T*)s.gv0; a.gf = (T*)s.gf; a.gv = (T*)s.gv; a.gvf = (T*)s.gvf;
    a.dt = (T)dt;
    a.flags = h->d_flags;
    a.mark_left = h->plastic.kind != MPM_PLASTICITY_NONE;
    a.reflect = h->reflect.enabled;
    for(int k = 0; k < 6; k++) a.side[k] = h->reflect.enabled ? h->reflect.side_type[k] : MPM_BC_FREE;
    a.pmodel = s.pmodel;
    a.pmask = s.pmask;
    a.motion = h->motion_dev;
    a.moving = h->motion_dev ? h->moving : 0u;
    // the grid may be of a P2G before list_tiles changed (a setter between the phases)
    const bool listed = list_tiles(h) && s.grid_listed;
    a.tile_flag = listed ? s.tile_flag : nullptr;
    a.tiles = listed ? s.tiles : nullptr;
    a.tile_count = s.tile_count;
    return a;
}

}  // namespace plain
