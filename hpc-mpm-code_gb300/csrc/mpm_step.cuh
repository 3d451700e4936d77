// Arguments and building blocks shared by the explicit step's kernels
// (mpm_explicit.cu, mpm_cells.cu).
#pragma once

#include "mpm_device.cuh"

namespace mpm {

template <typename R>
struct StepArgs {
    KGeom<R> g;
    Particles<R> P;
    int64_t num;
    const WorkItem *work;
    const int *nwork;
    const int *cstart;          // nbricks * (BRC + 1)
    int *miss;                  // particles that left their sorted cell, processed by a deferred pass
    const int *blist;           // bricks holding particles (brick order) and their count
    const int *nblist;
    const BrickShare *shares;   // the same bricks and the further shares of crowded ones, and their count
    const int *nshares;
    const int *tlist;           // active node tiles of this step (tile order) and their count
    const int *ntlist;
    int nbrick[3];
    unsigned long long *acc;    // NACC * nodec
    unsigned long long *acc2;   // 3 * nodec
    unsigned long long *facc;   // nodec (F-bar contexts)
    R *G;                       // gather field for the velocity gather (3 * nodec)
    R *nei;                     // nodec
    R *nvel2;                   // 3 * nodec
    R *nvel_dl, *naccel_dl;     // 3 * nodec each, written only in download mode
    const double *nvol;
    const unsigned char *bcflag;
    const R *bcval;
    unsigned char *tileflag;
    double *eu_part;            // sums of nei^2 by CTA of k_grid1
    int eu_parts;               // how many
    DevCtl *ctl;
    const int *iprop;
    const double *matprop;
    const float *matpropf;      // the same table in FP32 (the FP32 particle kernels)
    R dt, facl, mtol, grav[3];
    int parity;
    int scheme;
    int shifting;
    int all_tiles;              // process every tile in the grid passes (download mode)
    int gnorm;                  // FP32 gathers divide by their weight sum
    int implicit;               // implicit solid: the force fields carry sum N m a (AccelP2G)
    int fbar;                   // F-bar projection: k_grid2 leaves the nodal volume sums to k_fbar_grid
    int sigma_in;               // some material's stress update reads the previous stress (model 0)
    int single_mat;             // one material: every particle's matid is 0
    int fluidj;                 // Tait fluid only: F field 0 holds J - 1, fields 1-8 unused (FP32)
    // traversal directions of the particle kernels: each starts where the
    // previous particle pass ended, so its first bricks are still in L2
    int rev_p2g, rev_g2p, rev_upd;
    int begin;                  // the P2G kernel starts the step itself (p2g_scales), no k_step_reset before it
    double nump;                // particle count as a bound factor
    double mmax;                // max particle mass
    double gshape;              // bound on |dN/dx|
    double gsum;                // bound on sum_i |dN_i/dx|
};

// ----------------------------------------------------------------- helpers
template <typename R>
__device__ __forceinline__ R ld(const R *p) { return __ldg(p); }

__device__ __forceinline__ void tile_coords(int t, const int *nt, int &tx, int &ty, int &tz) {
    tx = t % nt[0];
    ty = (t / nt[0]) % nt[1];
    tz = t / (nt[0] * nt[1]);
}

template <typename R>
__device__ __forceinline__ int tile_of_node(const KGeom<R> &g, int gx, int gy, int gz) {
    return gx / TILE + g.ntile[0] * (gy / TILE + g.ntile[1] * (gz / TILE));
}

template <typename R>
__device__ __forceinline__ size_t node_id(const KGeom<R> &g, int gx, int gy, int gz) {
    return (size_t)gx + (size_t)g.nnc[0] * ((size_t)gy + (size_t)g.nnc[1] * (size_t)gz);
}

// Fixed-point scales.  Computed by one thread of a CTA (FP64 scalar work)
// and shared; producer and consumer kernels derive them from the same
// device-resident bounds, so they agree exactly.

// the bound of P2G scale k (0 mass, 1 volume, 2 momentum, 3 force) of the step
// of the given parity
template <typename R>
__device__ double bound_p2g(const StepArgs<R> &a, int parity, int k) {
    const volatile unsigned *nb = a.ctl->nxt[parity];
    if (k == 0) return a.nump * a.mmax;
    if (k == 1) return a.nump * (double)bits_f(nb[B_VOLMAX]);
    if (k == 2) return a.nump * a.mmax * (double)bits_f(nb[B_VMAX]);
    if (a.implicit) return a.nump * a.mmax * (double)bits_f(nb[B_AMAX]) * 1.0000001;
    const double gabs = fmax(fabs((double)a.grav[0]), fmax(fabs((double)a.grav[1]), fabs((double)a.grav[2])));
    return a.nump * ((double)bits_f(nb[B_VOLSMAX]) * 3.0 * a.gshape + a.mmax * gabs * fabs((double)a.facl));
}
// the bound of the gather's scales of this step: k = 0 the MUSL momentum, 1 the
// shifting's |geup|^2, from the grid maxima of k_grid1
template <typename R>
__device__ double bound_musl(const StepArgs<R> &a, int k) {
    const unsigned *nb = a.ctl->nxt[a.parity];
    const volatile unsigned *cur = a.ctl->cur;
    if (k == 0) {
        double vb = (double)bits_f(cur[C_GMAX]);
        if (a.scheme == MPM_FLIP) vb = (double)bits_f(nb[B_VMAX]) + fabs((double)a.dt) * vb;
        return a.nump * a.mmax * vb * 1.0000001;
    }
    const double gb = 2.0 * (double)bits_f(nb[B_VOLMAX]) * a.gsum * (double)bits_f(cur[C_NEIMAX]);
    return a.nump * 3.0 * gb * gb * 1.0000001;
}
// What a step resets before its first kernel records anything: the per-step
// counters and the bounds for the next step (one warp, a slot per lane).
template <typename R>
__device__ __forceinline__ void begin_step_ctl(const StepArgs<R> &a) {
    DevCtl *ctl = a.ctl;
    const int lane = threadIdx.x & 31;
    if (lane == 6) ctl->geup_acc = 0ull;
    else if (lane >= 8 && lane < 8 + B_NB) ctl->nxt[a.parity ^ 1][lane - 8] = 0u;
    else if (lane >= 16 && lane < 16 + C_NC) ctl->cur[lane - 16] = 0u;
}
static_assert(B_NB <= 8 && C_NC <= 16, "one lane per slot");

// The scales of a step: the P2G ones by k_step_reset or, where the P2G kernel
// starts the step itself, by each of its CTAs; the gather/MUSL ones by the first
// kernel that gathers (they depend on the grid maxima that k_grid1 records).
// Kernels copy them into shared memory.
template <typename R>
__device__ __forceinline__ void load_scales_from(const Scales *src, Scales &sh) {
    constexpr int W = (int)(sizeof(Scales) / 4);
    if ((int)threadIdx.x < W) reinterpret_cast<unsigned *>(&sh)[threadIdx.x] = reinterpret_cast<const unsigned *>(src)[threadIdx.x];
    __syncthreads();
}
template <typename R>
__device__ __forceinline__ void load_scales(const StepArgs<R> &a, Scales &sh) {
    load_scales_from<R>(&a.ctl->sc_p2g, sh);
}
// The P2G kernel's scales, from its first warp (the caller's next barrier
// publishes them).  With a.begin it is the step's first kernel: every CTA derives
// the scales from the bounds of the step before, and CTA 0 records them and
// resets what the later kernels record.  (A one-warp kernel for this before every
// P2G cost 3 us of a 33 us step of 8,000 particles.)
template <typename R>
__device__ __forceinline__ void p2g_scales(const StepArgs<R> &a, Scales &sh) {
    if (threadIdx.x >= 32) return;
    if (threadIdx.x < 4) {
        const Fix f = a.begin ? make_fix(bound_p2g(a, a.parity, threadIdx.x)) : (&a.ctl->sc_p2g.m)[threadIdx.x];
        (&sh.m)[threadIdx.x] = f;
        if (a.begin && blockIdx.x == 0) (&a.ctl->sc_p2g.m)[threadIdx.x] = f;
    }
    if (a.begin && blockIdx.x == 0) begin_step_ctl(a);
}
template <typename R>
__device__ __forceinline__ void load_scales_musl(const StepArgs<R> &a, Scales &sh) {
    load_scales_from<R>(&a.ctl->sc_musl, sh);
}
// The scales of the first kernel that gathers from k_grid1's fields: every CTA
// derives them from the grid's maxima, and CTA 0 (`all`: every CTA, where CTA 0 may
// have no work) records them for the passes behind it.  (The last CTA of k_grid1
// did this before, 4 us of every step: it waited for all others, read back their
// partials, and the gather waited for it.)
template <typename R>
__device__ __forceinline__ void musl_scales(const StepArgs<R> &a, Scales &sh, bool all = false) {
    if (threadIdx.x < 6) {
        const Fix f = threadIdx.x < 4 ? (&a.ctl->sc_p2g.m)[threadIdx.x] : make_fix(bound_musl(a, (int)threadIdx.x - 4));
        (&sh.m)[threadIdx.x] = f;
        if (all || blockIdx.x == 0) (&a.ctl->sc_musl.m)[threadIdx.x] = f;
    }
    __syncthreads();
}
// The momentum scale of the affine re-projection, from the velocities that the
// gather recorded (the caller's next barrier publishes it); CTA 0 records it.
template <typename R>
__device__ __forceinline__ Fix affine_fix(const StepArgs<R> &a) {
    return make_fix(a.nump * a.mmax * (double)bits_f(a.ctl->nxt[a.parity ^ 1][B_VMAX]) * 1.0000001);
}
template <typename R>
__device__ __forceinline__ void affine_scales(const StepArgs<R> &a, Scales &sh) {
    if (threadIdx.x != 0) return;
    const Fix f = affine_fix(a);
    sh.q = f;
    if (blockIdx.x == 0) a.ctl->sc_musl.q = f;
}

// Block-wide reduction (fixed order: deterministic); result valid in thread 0.
template <typename T, typename Op>
__device__ __forceinline__ T block_reduce(T v, Op op, T *sh) {
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_down_sync(0xffffffffu, v, o));
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    T r = sh[0];
    if (threadIdx.x == 0)
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) r = op(r, sh[w]);
    return r;
}

struct OpAddD { __device__ double operator()(double a, double b) const { return a + b; } };
struct OpAddL { __device__ long long operator()(long long a, long long b) const { return a + b; } };
struct OpAddI { __device__ int operator()(int a, int b) const { return a + b; } };
struct OpMaxF { __device__ float operator()(float a, float b) const { return fmaxf(a, b); } };

// The eight P2G contributions of one particle to one node
// (StandardVarP2G x3, ComputeInternalForce + ComputeExternalForce,
// material_point.h:223-247, solid_material_point.h:48-73).
template <typename R>
__device__ __forceinline__ void p2g_terms(R N, R d0, R d1, R d2, R m, R vol, const R *v, const R *s, R mfx, R mfy,
                                          R mfz, R *q) {
    const R Nm = N * m;
    q[0] = Nm;
    q[1] = N * vol;
    q[2] = Nm * v[0];
    q[3] = Nm * v[1];
    q[4] = Nm * v[2];
    q[5] = -vol * (s[0] * d0 + s[5] * d1 + s[4] * d2) + N * mfx;
    q[6] = -vol * (s[5] * d0 + s[1] * d1 + s[3] * d2) + N * mfy;
    q[7] = -vol * (s[4] * d0 + s[3] * d1 + s[2] * d2) + N * mfz;
}

template <typename R>
__device__ __forceinline__ void fx_terms(const R *q, const Scales &S, long long *o) {
    o[0] = fx(q[0], S.m);
    o[1] = fx(q[1], S.v);
    o[2] = fx(q[2], S.p);
    o[3] = fx(q[3], S.p);
    o[4] = fx(q[4], S.p);
    o[5] = fx(q[5], S.f);
    o[6] = fx(q[6], S.f);
    o[7] = fx(q[7], S.f);
}

__device__ __forceinline__ void brick_origin(int b, const int *nb, int &ox, int &oy, int &oz) {
    ox = (b % nb[0]) * BRX;
    oy = ((b / nb[0]) % nb[1]) * BRY;
    oz = (b / (nb[0] * nb[1])) * BRZ;
}

// Control-point coordinate xyc[idx][d] along one axis (DefineCpPos,
// module/mesh.h:32-47, on one rank: the open-knot end points of a quadratic
// axis sit on the walls).
template <typename R, int O>
__device__ __forceinline__ R cp_coord(const KGeom<R> &g, int d, int idx) {
    if (O == 1) return g.xmin[d] + g.dx[d] * (R)idx;
    if (idx == 0) return g.xmin[d];
    if (idx == g.nnc[d] - 1) return g.xmin[d] + g.dx[d] * (R)g.nel[d];
    return g.xmin[d] + g.dx[d] * ((R)idx - (R)0.5);
}

// v + A (x_i - x_p): the velocity a TPIC / APIC particle carries to node i
// (TPIC::VarP2G / APIC::VarP2G, module/map_and_interpolate.h:62-77,104-130,
// with the coordinate read as xyc[nid][j]).
template <typename R>
__device__ __forceinline__ void affine_velocity(const R *v, const R *A, R d0, R d1, R d2, R *out) {
#pragma unroll
    for (int c = 0; c < 3; c++) out[c] = v[c] + (A[3 * c] * d0 + A[3 * c + 1] * d1 + A[3 * c + 2] * d2);
}

// ------------------------------------------------------------ cell-local axes
// The quadratic B-spline of MakSf (module/shape_function.cpp:52-105) inside
// cell c of an axis with nel cells, as functions of t: node k = 0, 1, 2 has
//   w0 = s0 (1 - t)^2, w1 = a1 t^2 + b1 t + c1, w2 = s2 t^2
// with the open-knot pieces at the two walls.  (The pieces meet with equal
// values and slopes, so choosing them by the cell is exact at its faces too.)
template <typename R>
struct QuadCoef {
    R s0, a1, b1, c1, s2;
};
template <typename R>
__device__ __forceinline__ QuadCoef<R> quad_coef(int c, int nel) {
    const bool lo = c == 0, hi = c == nel - 1;
    QuadCoef<R> q;
    q.s0 = lo ? (R)1 : (R)0.5;
    q.a1 = (lo || hi) ? (R)-1.5 : (R)-1;
    q.b1 = lo ? (R)2 : (R)1;
    q.c1 = lo ? (R)0 : (R)0.5;
    q.s2 = hi ? (R)1 : (R)0.5;
    return q;
}

// weights and derivatives of an axis' nodes at offset t of cell c
template <typename R, int O>
struct CellAxis;
template <typename R>
struct CellAxis<R, 1> {
    R inv;
    __device__ __forceinline__ CellAxis(int, int, R inv_dx) : inv(inv_dx) {}
    __device__ __forceinline__ void eval(R t, R *w, R *d) const {
        w[0] = (R)1 - t;
        w[1] = t;
        d[0] = -inv;
        d[1] = inv;
    }
};
template <typename R>
struct CellAxis<R, 2> {
    QuadCoef<R> q;
    R inv;
    __device__ __forceinline__ CellAxis(int c, int nel, R inv_dx) : q(quad_coef<R>(c, nel)), inv(inv_dx) {}
    __device__ __forceinline__ void eval(R t, R *w, R *d) const {
        const R u = (R)1 - t, su = q.s0 * u, st = q.s2 * t, at = q.a1 * t;
        w[0] = su * u;
        w[1] = fma(at + q.b1, t, q.c1);
        w[2] = st * t;
        d[0] = (R)-2 * su * inv;
        d[1] = fma((R)2, at, q.b1) * inv;
        d[2] = (R)2 * st * inv;
    }
};

// Offset of x from the lower face of cell c, in cells.
template <typename R>
__device__ __forceinline__ R cell_t(R x, const KGeom<R> &g, int d, int c) {
    return (x - (g.xmin[d] + g.dx[d] * (R)c)) * g.inv_dx[d];
}
// Whether an offset lies inside (0, 1) and farther from its ends than rounding
// can move it (FP64: 1e-9 and 1e-6, above the rounding of the offset up to a
// million cells; the test reads the high words of the numbers, since an FP64
// comparison takes a slot of the FP64 pipe).
__device__ __forceinline__ bool off_faces(float t) { return t > 1e-3f && t < 0.999f; }
__device__ __forceinline__ bool off_faces(double t) {
    const unsigned hi = (unsigned)__double2hiint(t);   // a negative t, an infinity and a NaN are above 1
    return hi > 0x3E112E0Bu && hi < 0x3FEFFFFFu;       // 1e-9 and 1 - 2^-20
}
// cell_of without its FP64 division away from the cell faces (a guess from FP32
// arithmetic, which the offset confirms); t the offset in that cell, oob set where
// x lies outside the grid (the cell is then the nearest one)
template <typename R>
__device__ __forceinline__ int fast_cell(R x, const KGeom<R> &g, int d, R &t, bool &oob) {
    int c = __float2int_rd((float)(x - g.xmin[d]) * (float)g.inv_dx[d]);
    t = cell_t(x, g, d, c);
    if ((unsigned)c >= (unsigned)g.nel[d] || !off_faces(t)) {
        c = cell_of(x, g, d, oob);
        t = cell_t(x, g, d, c);
    }
    return c;
}
// axis_eval's weights of a point outside the grid: the linear hats fall off beyond
// their node (1 - |x - x_i| / dx), where those of CellAxis would go on rising
template <typename R, int O>
__device__ __forceinline__ void outside_weights(R x, const KGeom<R> &g, int d, int c, R *w, R *dw) {
    Axis<R, O> a;
    axis_eval<R, O>(x, g, d, c, a);
#pragma unroll
    for (int k = 0; k <= O; k++) w[k] = a.w[k], dw[k] = a.dw[k];
}

// sum_n N_n f_n (VAL) and sum_n dN_n/dx f_n (GRAD) of a nodal field over a cell's
// nodes (b0 the first, sy and sz the strides), summed axis by axis: rows, layers,
// cell.  36 FMAs for value and gradient of a linear cell where weights and
// products node by node take about 100.
template <typename R, int OX, int OY, int OZ>
struct CellWeights {
    R wx[OX + 1], dx[OX + 1], wy[OY + 1], dy[OY + 1], wz[OZ + 1], dz[OZ + 1];
};
template <bool VAL, bool GRAD, typename R, int OX, int OY, int OZ>
__device__ __forceinline__ void cell_field(const R *f, size_t b0, size_t sy, size_t sz,
                                           const CellWeights<R, OX, OY, OZ> &w, R &val, R *g) {
    R v = (R)0, gx = (R)0, gy = (R)0, gz = (R)0;
#pragma unroll
    for (int k = 0; k <= OZ; k++) {
        R l = (R)0, lx = (R)0, ly = (R)0;
#pragma unroll
        for (int j = 0; j <= OY; j++) {
            R r = (R)0, rx = (R)0;
#pragma unroll
            for (int i = 0; i <= OX; i++) {
                const R q = ld(f + b0 + i + j * sy + k * sz);
                r = fma(w.wx[i], q, r);
                if (GRAD) rx = fma(w.dx[i], q, rx);
            }
            l = fma(w.wy[j], r, l);
            if (GRAD) lx = fma(w.wy[j], rx, lx);
            if (GRAD) ly = fma(w.dy[j], r, ly);
        }
        if (VAL) v = fma(w.wz[k], l, v);
        if (GRAD) gx = fma(w.wz[k], lx, gx);
        if (GRAD) gy = fma(w.wz[k], ly, gy);
        if (GRAD) gz = fma(w.dz[k], l, gz);
    }
    if (VAL) val = v;
    if (GRAD) g[0] = gx, g[1] = gy, g[2] = gz;
}
// the cell of a point, its node weights and its first node
template <typename R, int OX, int OY, int OZ>
__device__ __forceinline__ size_t cell_weights(const KGeom<R> &g, const R *x, CellWeights<R, OX, OY, OZ> &w) {
    R t0, t1, t2;
    bool oob = false;
    const int cx = fast_cell(x[0], g, 0, t0, oob), cy = fast_cell(x[1], g, 1, t1, oob),
              cz = fast_cell(x[2], g, 2, t2, oob);
    CellAxis<R, OX>(cx, g.nel[0], g.inv_dx[0]).eval(t0, w.wx, w.dx);
    CellAxis<R, OY>(cy, g.nel[1], g.inv_dx[1]).eval(t1, w.wy, w.dy);
    CellAxis<R, OZ>(cz, g.nel[2], g.inv_dx[2]).eval(t2, w.wz, w.dz);
    if (oob) {   // the weights of its P2G (k_cell_misses)
        outside_weights<R, OX>(x[0], g, 0, cx, w.wx, w.dx);
        outside_weights<R, OY>(x[1], g, 1, cy, w.wy, w.dy);
        outside_weights<R, OZ>(x[2], g, 2, cz, w.wz, w.dz);
    }
    return node_id(g, cx, cy, cz);
}

// ------------------------------------------------------------- mpm_cells.cu
// What a cell scatter sums: the eight P2G fields (plain, with the affine
// momentum of TPIC / APIC, with the implicit solid's N m a in the force
// fields) or the MUSL momentum (plain, affine).
enum CellKind { CELL_P2G = 0, CELL_P2G_AFF, CELL_P2G_ACC, CELL_MUSL, CELL_MUSL_AFF };
// The scatter of kind `kind` as per-cell register sums, then the deferred pass
// over the particles that left their sorted cell; two launches on st.
template <typename R>
void launch_cell_scatter(const StepArgs<R> &a, const int *order, int kind, int nbricks, int nsm, bool pdl,
                         cudaStream_t st);
// The velocity gather of PIC / FLIP and sum |geup|^2, one thread per particle.
template <typename R>
void launch_gather(const StepArgs<R> &a, const int *order, int nsm, bool pdl, cudaStream_t st);

}  // namespace mpm
