// Scatters and gathers of the explicit step for every shape order and both
// precisions: FP64 grids, quadratic B-splines, and the P2G of the implicit
// solid.  (FP32 linear explicit grids have kernels of their own in
// mpm_explicit.cu.)
//
// Scatter (k_cell_scatter).  Particles are sorted by cell, so a thread can sum
// a cell's contributions to some of its nodes in registers in particle order,
// without atomics: P threads per cell, thread (j, k) owning the nodes of one
// row (all i) of the cell's (OX+1)(OY+1)(OZ+1) nodes, or the rows of one
// z-layer on FP64 linear grids.  A crowded brick is cut into shares (share_run in
// mpm_sort.cu).  The sums of the CTA's cells go to shared memory once and a node
// pass adds the cells around each node in a fixed order before one int64
// fixed-point RED per node and field.  Deterministic: every sum is in a fixed order,
// or of integers.  The staging box it replaces spent its time in 64-bit
// shared-memory atomics, one per particle, node and field.  P2G class per step,
// staging box -> here: FP64 linear, 201,872 particles, 296 -> 128 us; FP32
// B-splines, 216,000 particles, 444 -> 66 us; FP64 B-splines, 46,656 particles,
// 643 -> 146 us; implicit FP32 linear, 1,728,000 particles, 802 -> 116 us (66 with plain
// FP32 sums).
//
// FP32 (B-splines, and the implicit solid's P2G on linear grids) forms each
// contribution as the staging box (mpm_explicit.cu) does and sums it in an
// unevaluated pair of FP32 numbers (two-sum: 48 bits), which is as exact as the
// box's int64 sums and leaves the step's results as they were.  (Plain FP32 sums
// of the B-splines took 47 us in place of 66, but the sums of 216 contributions are
// far more exact than an FP32 number, and the stresses of a nearly uniform velocity
// field moved by 5e-5; the implicit P2G's nodal mass, 64 particles per cell, was up to
// 3.2 x 2^-24 off, and within 2 x 2^-24 with pairs.  int64 sums took 185 us, in the float
// to int64 conversions.)
// 32 cells per CTA and two CTAs per SM: 16, 64 or one CTA measured 78 to 95 us.
// FP64 sums are kept in FP64.
//
// There, within a cell the weights are polynomials of the offset t in [0, 1)
// from its lower face, with coefficients that depend on the cell alone
// (CellAxis): no division, no search for the spline's piece.  FP64 grids are
// bound by the FP64 pipe (2 FMAs per SM and clock; ncu: 71 % busy in the linear
// P2G, 292 FP64 instructions per particle), so a row's products are formed once,
// a node costs 11 FMAs, and the in-cell test reads the high words of the offsets
// in place of 6 FP64 comparisons (135 -> 128 us).
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <type_traits>

#include "mpm_step.cuh"

namespace mpm {

// one node of an axis: weight (a t + b) t + c, derivative (2 a t + b) / dx
template <typename R, int O>
struct CellNode;
template <typename R>
struct CellNode<R, 1> {
    R s, c, di;
    __device__ __forceinline__ CellNode(int k, int, int, R inv_dx)
        : s(k ? (R)1 : (R)-1), c(k ? (R)0 : (R)1), di(k ? inv_dx : -inv_dx) {}
    __device__ __forceinline__ void eval(R t, R &w, R &d) const {
        w = fma(s, t, c);
        d = di;
    }
};
template <typename R>
struct CellNode<R, 2> {
    R a, b, c, inv;
    __device__ __forceinline__ CellNode(int k, int cell, int nel, R inv_dx) : inv(inv_dx) {
        const QuadCoef<R> q = quad_coef<R>(cell, nel);
        a = k == 0 ? q.s0 : k == 1 ? q.a1 : q.s2;
        b = k == 0 ? (R)-2 * q.s0 : k == 1 ? q.b1 : (R)0;
        c = k == 0 ? q.s0 : k == 1 ? q.c1 : (R)0;
    }
    __device__ __forceinline__ void eval(R t, R &w, R &d) const {
        const R at = a * t;
        w = fma(at + b, t, c);
        d = (at + at + b) * inv;
    }
};

// axis_eval's nodes inside a known cell, with its arithmetic: the piece of each
// node follows from the cell, so what is left per particle is the polynomial.
// (At a cell's faces axis_eval may round h onto the neighbouring piece, whose
// value and slope there are the same.)
template <typename R, int O>
struct PieceNode;
template <typename R>
struct PieceNode<R, 2> {
    R xy, hs, s1, s2, s3, d1, d2;
    __device__ __forceinline__ PieceNode(int k, int cell, const KGeom<R> &g, int d) {
        const int n = cell + k, nnc = g.nnc[d];
        xy = g.xmin[d] + g.dx[d] * (R)(n - 2);
        hs = n == 0 ? (R)2 : n == 1 ? (R)1 : (R)0;
        if (n == 0) { s1 = 1; s2 = -2; s3 = 1; d1 = 2; d2 = -2; }
        else if (n == 1 && k == 1) { s1 = -1.5; s2 = 2; s3 = 0; d1 = -3; d2 = 2; }
        else if (n == 1) { s1 = 0.5; s2 = -2; s3 = 2; d1 = 1; d2 = -2; }
        else if (n == nnc - 1) { s1 = 1; s2 = 0; s3 = 0; d1 = 2; d2 = 0; }
        else if (n == nnc - 2 && k == 1) { s1 = -1.5; s2 = 4; s3 = -2; d1 = -3; d2 = 4; }
        else if (k == 2) { s1 = 0.5; s2 = 0; s3 = 0; d1 = 1; d2 = 0; }
        else if (k == 1) { s1 = -1; s2 = 3; s3 = -1.5; d1 = -2; d2 = 3; }
        else { s1 = 0.5; s2 = -3; s3 = 4.5; d1 = 1; d2 = -3; }
    }
    __device__ __forceinline__ void eval(R x, const KGeom<R> &g, int d, R &w, R &dw) const {
        const R h = (x - xy) * g.inv_dx[d] - hs;
        w = (s1 * h + s2) * h + s3;
        dw = (d1 * h + d2) * g.inv_dx[d];
    }
};
template <typename R>
struct PieceNode<R, 1> {
    R xy, di;
    __device__ __forceinline__ PieceNode(int k, int cell, const KGeom<R> &g, int d)
        : xy(g.xmin[d] + g.dx[d] * (R)(cell + k)), di(k ? g.inv_dx[d] : -g.inv_dx[d]) {}
    __device__ __forceinline__ void eval(R x, const KGeom<R> &g, int d, R &w, R &dw) const {
        w = (R)1 - fabs(x - xy) * g.inv_dx[d];
        dw = di;
    }
};

// Whether x lies in cell c as cell_of decides it (the reference's
// floor((x - xmin) / dx) in FP64).  Away from the faces the offset alone tells;
// near one cell_of does, with its division.  A point outside the grid is in none.
template <typename R>
__device__ __forceinline__ bool in_cell_axis(R x, R t, const KGeom<R> &g, int d, int c) {
    if (off_faces(t)) return true;
    if (!(t > (R)-1e-3 && t < (R)1.001)) return false;
    bool oob = false;
    return cell_of(x, g, d, oob) == c && !oob;
}

// ------------------------------------------------------------------- scatter
// Two sums of FP32 numbers, each an unevaluated pair s + e with s = fl(s + e):
// Knuth's two-sum on packed FP32 operations (two per instruction), a - b
// written as fma(b, -1, a).  Each step rounds to nearest as written, which the
// error-free transformation relies on.
using F2 = unsigned long long;   // two packed FP32 numbers
__device__ __forceinline__ F2 f2_pack(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_unpack(F2 v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(0xBF800000BF800000ull), "l"(a));
    return r;
}
struct alignas(16) Pair2 {
    F2 s, e;
    __device__ __forceinline__ void add(F2 q) {
        const F2 t = f2_add(s, q), b = f2_sub(t, s);
        e = f2_add(e, f2_add(f2_sub(s, f2_sub(t, b)), f2_sub(q, b)));
        s = t;
    }
};
template <typename R>
__device__ __forceinline__ void sum_add(R &s, R q) { s += q; }
__device__ __forceinline__ void sum_add(Pair2 &s, const Pair2 &q) {
    s.add(q.s);
    s.e = f2_add(s.e, q.e);
}
// the fixed-point value of sum w (0 or 1 of a Pair2)
template <typename R>
__device__ __forceinline__ long long sum_fixed(R s, int, const Fix &F) { return fx(s, F); }
__device__ __forceinline__ long long sum_fixed(const Pair2 &p, int w, const Fix &F) {
    float s[2], e[2];
    f2_unpack(p.s, s[0], s[1]);
    f2_unpack(p.e, e[0], e[1]);
    const float v = w ? s[1] : s[0], r = w ? e[1] : e[0];
    return (v == 0.0f && r == 0.0f) ? 0ll : fx(v, F) + fx(r, F);
}

template <typename R, int OX, int OY, int OZ>
struct CellShape {
    // FP32 (B-splines, and the implicit solid's P2G): sums as exact as the staging box's
    static constexpr bool EXACT = sizeof(R) == 4;
    using Sum = typename std::conditional<EXACT, Pair2, R>::type;
    static constexpr int W = EXACT ? 2 : 1;               // fields per sum
    static constexpr int NX = OX + 1, NY = OY + 1, NZ = OZ + 1, NE = NX * NY * NZ;
    // rows per thread: both rows of a z-layer when FP64 and linear, one row otherwise
    // (pairs take twice the registers)
    static constexpr int JP = (!EXACT && OX == 1 && OY == 1) ? NY : 1;
    static constexpr int P = NZ * (NY / JP);              // threads per cell
    // cells of a CTA (z-slabs of a brick): as many as leave the accumulators,
    // 8 JP NX values per thread, in registers.  FP64 B-splines: 32 cells; with 64
    // the P2G of 46,656 particles takes 139 us in place of 146, but that of 17,472
    // 89 in place of 51, and with 16 they take 187 and 54
    static constexpr int CELLS = P == 2 ? BRC : P == 9 || sizeof(R) == 8 ? BRC / 4 : BRC / 2;
    static constexpr int SLABS = BRC / CELLS, BZ = BRZ / SLABS;
    static constexpr int THREADS = CELLS * P;
    static constexpr int MINB = (EXACT || P == 2) ? 2 : 1;   // CTAs per SM to compile for
    static constexpr int BX = BRX + OX, BY = BRY + OY, BZN = BZ + OZ, BOX = BX * BY * BZN;
    static constexpr int FR = 4 / W;                      // sums per round of the node pass
    static constexpr size_t SMEM = sizeof(Sum) * FR * NE * CELLS;
};

// One particle's contributions to the nodes (i, j0, kk) of its cell, formed as
// the staging box does (k_p2g_box, k_g2p_musl_box, k_affine_musl)
template <typename R, int OX, int OY, int OZ, int KIND, int NG>
__device__ __forceinline__ void cell_terms_exact(const StepArgs<R> &a, const PieceNode<R, OY> &ay,
                                                 const PieceNode<R, OZ> &az, int p, int cx, int cy, int cz, int j0, int kk, R x0, R x1, R x2, R m, const R *v,
                                                 Pair2 (&acc)[NG][1][OX + 1]) {
    constexpr bool MUSL = KIND == CELL_MUSL || KIND == CELL_MUSL_AFF;
    constexpr bool AFF = KIND == CELL_P2G_AFF || KIND == CELL_MUSL_AFF;
    const Particles<R> &P = a.P;
    R wx[OX + 1], dx[OX + 1], wy, dy, wz, dz;
    if (OX == 2 && cx >= 2 && cx <= a.g.nel[0] - 3) {   // no wall piece: constants instead of 21 registers
        constexpr R c1[3] = {0.5, -1, 0.5}, c2[3] = {-3, 3, 0}, c3[3] = {4.5, -1.5, 0}, e1[3] = {1, -2, 1},
                    e2[3] = {-3, 3, 0};
#pragma unroll
        for (int i = 0; i <= OX; i++) {
            const R xy = a.g.xmin[0] + a.g.dx[0] * (R)(cx + i - 2);
            const R h = (x0 - xy) * a.g.inv_dx[0];
            wx[i] = (c1[i] * h + c2[i]) * h + c3[i];
            dx[i] = (e1[i] * h + e2[i]) * a.g.inv_dx[0];
        }
    } else {
#pragma unroll
        for (int i = 0; i <= OX; i++) PieceNode<R, OX>(i, cx, a.g, 0).eval(x0, a.g, 0, wx[i], dx[i]);
    }
    ay.eval(x1, a.g, 1, wy, dy);
    az.eval(x2, a.g, 2, wz, dz);
    R vol = (R)0, s[6], A[AFF ? 9 : 1], mg[3];
    if constexpr (!MUSL) {
        vol = ld(P.vol + p);
#pragma unroll
        for (int e = 0; e < 6; e++) s[e] = ld(P.s[e] + p);
#pragma unroll
        for (int c = 0; c < 3; c++) mg[c] = m * (a.grav[c] * a.facl);
    }
    if constexpr (AFF) {
#pragma unroll
        for (int e = 0; e < 9; e++) A[e] = ld(P.C[e] + p);
    }
#pragma unroll
    for (int i = 0; i <= OX; i++) {
        const R wxy = wx[i] * wy;
        R vn[3] = {v[0], v[1], v[2]};
        if constexpr (AFF)
            affine_velocity(v, A, cp_coord<R, OX>(a.g, 0, cx + i) - x0, cp_coord<R, OY>(a.g, 1, cy + j0) - x1,
                            cp_coord<R, OZ>(a.g, 2, cz + kk) - x2, vn);
        if constexpr (MUSL) {
            const R Nm = wxy * wz * m;
            acc[0][0][i].add(f2_pack(Nm * vn[0], Nm * vn[1]));
            acc[1][0][i].add(f2_pack(Nm * vn[2], (R)0));
        } else {
            R q[NACC];
            p2g_terms(wxy * wz, dx[i] * wy * wz, wx[i] * dy * wz, wxy * dz, m, vol, vn, s, mg[0], mg[1], mg[2], q);
            if constexpr (KIND == CELL_P2G_ACC) {
                const R Nm = wxy * wz * m;
#pragma unroll
                for (int c = 0; c < 3; c++) q[5 + c] = Nm * ld(P.a[c] + p);
            }
#pragma unroll
            for (int f = 0; f < NG; f++) acc[f][0][i].add(f2_pack(q[2 * f], q[2 * f + 1]));
        }
    }
}

template <typename R, int OX, int OY, int OZ, int KIND>
__global__ void __launch_bounds__(CellShape<R, OX, OY, OZ>::THREADS, CellShape<R, OX, OY, OZ>::MINB) k_cell_scatter(StepArgs<R> a) {
    using C = CellShape<R, OX, OY, OZ>;
    constexpr int NX = C::NX, NY = C::NY, JP = C::JP, P = C::P, CELLS = C::CELLS;
    constexpr bool MUSL = KIND == CELL_MUSL || KIND == CELL_MUSL_AFF;
    constexpr bool AFF = KIND == CELL_P2G_AFF || KIND == CELL_MUSL_AFF;
    constexpr int NF = MUSL ? 3 : NACC;
    constexpr int W = C::W, NG = (NF + W - 1) / W;   // sums per node
    pdl_wait();
    extern __shared__ __align__(16) unsigned char cell_smem[];
    using Sum = typename C::Sum;
    Sum *corner = reinterpret_cast<Sum *>(cell_smem);   // [FR][NE][CELLS]
    __shared__ Scales S;
    if (KIND == CELL_MUSL_AFF) affine_scales(a, S);
    else if (MUSL) load_scales_musl(a, S);
    else p2g_scales(a, S);   // read after the first barrier of a slab
    const int lc = threadIdx.x / P, part = threadIdx.x % P;
    const int kk = part % C::NZ, j0 = (part / C::NZ) * JP;
    const Particles<R> &Q = a.P;
    int misses = 0;
    const int nitem = *a.nshares * C::SLABS;
    for (int it = blockIdx.x; it < nitem; it += gridDim.x) {
        const BrickShare bs = a.shares[it / C::SLABS];
        const int b = bs.brick, slab = it % C::SLABS;
        const int *cs = a.cstart + (size_t)b * (BRC + 1) + slab * CELLS;
        if (cs[0] == cs[CELLS]) continue;   // an empty slab (uniform across the CTA)
        int ox, oy, oz;
        brick_origin(b, a.nbrick, ox, oy, oz);
        oz += slab * C::BZ;
        const int cx = ox + lc % BRX, cy = oy + (lc / BRX) % BRY, cz = oz + lc / (BRX * BRY);
        int p0 = cs[lc], p1 = cs[lc + 1];
        if (bs.count > 1) {   // this share's run of the cell's particles
            const int run = (p1 - p0 + bs.count - 1) / bs.count;
            p0 = min(p1, p0 + bs.share * run);
            p1 = min(p1, p0 + run);
        }
        Sum acc[NG][JP][NX];
#pragma unroll
        for (int f = 0; f < NG; f++)
#pragma unroll
            for (int j = 0; j < JP; j++)
#pragma unroll
                for (int i = 0; i < NX; i++) acc[f][j][i] = Sum{};
        const CellAxis<R, OX> ax(cx, a.g.nel[0], a.g.inv_dx[0]);
        const CellNode<R, OY> ay(j0, cy, a.g.nel[1], a.g.inv_dx[1]);
        const CellNode<R, OZ> az(kk, cz, a.g.nel[2], a.g.inv_dx[2]);
        const PieceNode<R, OY> py(j0, cy, a.g, 1);
        const PieceNode<R, OZ> pz(kk, cz, a.g, 2);
        for (int p = p0; p < p1; p++) {
            const R x0 = ld(Q.x[0] + p), x1 = ld(Q.x[1] + p), x2 = ld(Q.x[2] + p);
            const R m = ld(Q.m + p);
            const R v[3] = {ld(Q.v[0] + p), ld(Q.v[1] + p), ld(Q.v[2] + p)};
            const R t0 = cell_t(x0, a.g, 0, cx), t1 = cell_t(x1, a.g, 1, cy), t2 = cell_t(x2, a.g, 2, cz);
            if (!(in_cell_axis(x0, t0, a.g, 0, cx) && in_cell_axis(x1, t1, a.g, 1, cy) &&
                  in_cell_axis(x2, t2, a.g, 2, cz))) {
                // a particle outside its sorted cell: the deferred pass (k_cell_misses)
                if (part == 0) {
                    misses++;
                    a.miss[atomicAdd(MUSL ? &a.ctl->n_miss_musl : &a.ctl->n_miss_p2g, 1u)] = p;
                }
                continue;
            }
            if constexpr (C::EXACT) {
                cell_terms_exact<R, OX, OY, OZ, KIND>(a, py, pz, p, cx, cy, cz, j0, kk, x0, x1, x2, m, v, acc);
            }
            if constexpr (!C::EXACT) {
            R wx[NX], dx[NX], wz, dz;
            ax.eval(t0, wx, dx);
            az.eval(t2, wz, dz);
            R vol, s[6], pa[3], A[AFF ? 9 : 1];
            if constexpr (!MUSL) vol = ld(Q.vol + p);
            if constexpr (KIND == CELL_P2G || KIND == CELL_P2G_AFF) {
#pragma unroll
                for (int e = 0; e < 6; e++) s[e] = vol * ld(Q.s[e] + p);
            }
            if constexpr (KIND == CELL_P2G_ACC) {
#pragma unroll
                for (int c = 0; c < 3; c++) pa[c] = m * ld(Q.a[c] + p);
            }
            if constexpr (AFF) {
#pragma unroll
                for (int e = 0; e < 9; e++) A[e] = ld(Q.C[e] + p);
            }
#pragma unroll
            for (int j = 0; j < JP; j++) {
                R wy, dy;
                if constexpr (JP == 1) {
                    ay.eval(t1, wy, dy);
                } else {   // linear: rows 0 and 1
                    wy = j ? t1 : (R)1 - t1;
                    dy = j ? a.g.inv_dx[1] : -a.g.inv_dx[1];
                }
                const R wjk = wy * wz, qm = m * wjk;
                constexpr int F0 = MUSL ? 0 : 2;   // first momentum field
                if constexpr (AFF) {
                    const R d1 = cp_coord<R, OY>(a.g, 1, cy + j0 + j) - x1, d2 = cp_coord<R, OZ>(a.g, 2, cz + kk) - x2;
                    R base[3];
#pragma unroll
                    for (int c = 0; c < 3; c++) base[c] = v[c] + (A[3 * c + 1] * d1 + A[3 * c + 2] * d2);
#pragma unroll
                    for (int i = 0; i < NX; i++) {
                        const R Nm = qm * wx[i], d0 = cp_coord<R, OX>(a.g, 0, cx + i) - x0;
                        if constexpr (!MUSL) acc[0][j][i] += Nm;
#pragma unroll
                        for (int c = 0; c < 3; c++)
                            acc[F0 + c][j][i] = fma(Nm, fma(A[3 * c], d0, base[c]), acc[F0 + c][j][i]);
                    }
                } else {
                    const R qv[3] = {qm * v[0], qm * v[1], qm * v[2]};
#pragma unroll
                    for (int i = 0; i < NX; i++) {
                        if constexpr (!MUSL) acc[0][j][i] = fma(qm, wx[i], acc[0][j][i]);
#pragma unroll
                        for (int c = 0; c < 3; c++) acc[F0 + c][j][i] = fma(qv[c], wx[i], acc[F0 + c][j][i]);
                    }
                }
                if constexpr (!MUSL) {
                    const R qv = vol * wjk;
#pragma unroll
                    for (int i = 0; i < NX; i++) acc[1][j][i] = fma(qv, wx[i], acc[1][j][i]);
                }
                if constexpr (KIND == CELL_P2G || KIND == CELL_P2G_AFF) {
                    // -vol sigma dN: the x-derivative of the row, and the rest along its weights
                    const R gy = dy * wz, gz = wy * dz;
                    const R sx[3] = {s[0], s[5], s[4]}, sy[3] = {s[5], s[1], s[3]}, sz[3] = {s[4], s[3], s[2]};
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const R fx_ = -sx[c] * wjk, fr = -fma(sy[c], gy, sz[c] * gz);
#pragma unroll
                        for (int i = 0; i < NX; i++)
                            acc[5 + c][j][i] = fma(fx_, dx[i], fma(fr, wx[i], acc[5 + c][j][i]));
                    }
                }
                if constexpr (KIND == CELL_P2G_ACC) {
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const R q = pa[c] * wjk;
#pragma unroll
                        for (int i = 0; i < NX; i++) acc[5 + c][j][i] = fma(q, wx[i], acc[5 + c][j][i]);
                    }
                }
            }
            }
        }
        if constexpr (!C::EXACT && (KIND == CELL_P2G || KIND == CELL_P2G_AFF)) {
            // the weight of the mass summed above
            const R gv[3] = {a.grav[0] * a.facl, a.grav[1] * a.facl, a.grav[2] * a.facl};
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int j = 0; j < JP; j++)
#pragma unroll
                    for (int i = 0; i < NX; i++) acc[5 + c][j][i] = fma(acc[0][j][i], gv[c], acc[5 + c][j][i]);
        }
        // the node pass, FR sums at a time
#pragma unroll
        for (int f0 = 0; f0 < NG; f0 += C::FR) {
            constexpr int FR = C::FR;
#pragma unroll
            for (int f = 0; f < FR; f++)
                if (f0 + f < NG) {
#pragma unroll
                    for (int j = 0; j < JP; j++)
#pragma unroll
                        for (int i = 0; i < NX; i++)
                            corner[(f * C::NE + i + NX * (j0 + j + NY * kk)) * CELLS + lc] = acc[f0 + f < NG ? f0 + f : 0][j][i];
                }
            __syncthreads();
            const int nfr = NG - f0 < FR ? NG - f0 : FR;
            for (int q = threadIdx.x; q < C::BOX * nfr; q += C::THREADS) {
                const int n = q % C::BOX, f = q / C::BOX;
                const int nx = n % C::BX, ny = (n / C::BX) % C::BY, nz = n / (C::BX * C::BY);
                const int gx = ox + nx, gy = oy + ny, gz = oz + nz;
                if (gx >= a.g.nnc[0] || gy >= a.g.nnc[1] || gz >= a.g.nnc[2]) continue;
                const Sum *cf = corner + (size_t)f * C::NE * CELLS;
                Sum sum{};
#pragma unroll
                for (int k = 0; k < C::NZ; k++)
#pragma unroll
                    for (int j = 0; j < NY; j++)
#pragma unroll
                        for (int i = 0; i < NX; i++) {
                            const int ex = nx - i, ey = ny - j, ez = nz - k;
                            if ((unsigned)ex < (unsigned)BRX && (unsigned)ey < (unsigned)BRY &&
                                (unsigned)ez < (unsigned)C::BZ)
                                sum_add(sum, cf[(i + NX * (j + NY * k)) * CELLS + ex + BRX * (ey + BRY * ez)]);
                        }
                if (!MUSL && f0 + f == 0) a.tileflag[tile_of_node(a.g, gx, gy, gz)] = 1;
                unsigned long long *dst = (MUSL ? a.acc2 : a.acc) + node_id(a.g, gx, gy, gz);
#pragma unroll
                for (int w = 0; w < W; w++) {
                    const int fg = (f0 + f) * W + w;
                    const Fix &F = MUSL ? S.q : fg == 0 ? S.m : fg == 1 ? S.v : fg <= 4 ? S.p : S.f;
                    const long long v = sum_fixed(sum, w, F);
                    if (v && fg < NF) atomic_add_i64(&dst[(size_t)fg * a.g.nodec], v);
                }
            }
            __syncthreads();   // shared memory is reused by the next round
        }
    }
    if (!MUSL && misses) atomicAdd(&a.ctl->tile_misses, (unsigned)misses);
}

// The deferred pass: the particles that left their sorted cell (or the grid),
// NE threads per particle, one per node, with fixed-point atomics (order
// independent, so the result does not depend on the queue's order).
template <typename R, int OX, int OY, int OZ, int KIND>
__global__ void __launch_bounds__(256) k_cell_misses(StepArgs<R> a) {
    constexpr int NX = OX + 1, NY = OY + 1, NE = NX * NY * (OZ + 1);
    constexpr bool MUSL = KIND == CELL_MUSL || KIND == CELL_MUSL_AFF;
    constexpr bool AFF = KIND == CELL_P2G_AFF || KIND == CELL_MUSL_AFF;
    pdl_wait();
    __shared__ Scales S;
    if (MUSL) load_scales_musl(a, S);
    else load_scales(a, S);
    const unsigned n = MUSL ? a.ctl->n_miss_musl : a.ctl->n_miss_p2g;
    const Particles<R> &P = a.P;
    unsigned oobs = 0;
    for (size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x; g < (size_t)NE * n;
         g += (size_t)gridDim.x * blockDim.x) {
        const int p = a.miss[g / NE], e = (int)(g % NE);
        const int i = e % NX, j = (e / NX) % NY, k = e / (NX * NY);
        const R x0 = ld(P.x[0] + p), x1 = ld(P.x[1] + p), x2 = ld(P.x[2] + p), m = ld(P.m + p);
        bool oob = false;
        const int cx = cell_of(x0, a.g, 0, oob), cy = cell_of(x1, a.g, 1, oob), cz = cell_of(x2, a.g, 2, oob);
        oobs += oob && e == 0;
        Axis<R, OX> ax;
        Axis<R, OY> ay;
        Axis<R, OZ> az;
        axis_eval<R, OX>(x0, a.g, 0, cx, ax);
        axis_eval<R, OY>(x1, a.g, 1, cy, ay);
        axis_eval<R, OZ>(x2, a.g, 2, cz, az);
        // this node's weights (selected, so that the axes stay in registers)
        R wx = ax.w[0], dx = ax.dw[0], wy = ay.w[0], dy = ay.dw[0], wz = az.w[0], dz = az.dw[0];
#pragma unroll
        for (int q = 1; q <= OX; q++)
            if (i == q) wx = ax.w[q], dx = ax.dw[q];
#pragma unroll
        for (int q = 1; q <= OY; q++)
            if (j == q) wy = ay.w[q], dy = ay.dw[q];
#pragma unroll
        for (int q = 1; q <= OZ; q++)
            if (k == q) wz = az.w[q], dz = az.dw[q];
        R v[3] = {ld(P.v[0] + p), ld(P.v[1] + p), ld(P.v[2] + p)};
        if constexpr (AFF) {
            R A[9], vn[3];
#pragma unroll
            for (int q = 0; q < 9; q++) A[q] = ld(P.C[q] + p);
            affine_velocity(v, A, cp_coord<R, OX>(a.g, 0, cx + i) - x0, cp_coord<R, OY>(a.g, 1, cy + j) - x1,
                            cp_coord<R, OZ>(a.g, 2, cz + k) - x2, vn);
            v[0] = vn[0], v[1] = vn[1], v[2] = vn[2];
        }
        const size_t N = (size_t)a.g.nodec, gn = node_id(a.g, cx + i, cy + j, cz + k);
        const R w = wx * wy * wz;
        if constexpr (MUSL) {
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const long long q = fx(w * m * v[c], S.q);
                if (q) atomic_add_i64(&a.acc2[c * N + gn], q);
            }
        } else {
            R s[6];
#pragma unroll
            for (int q = 0; q < 6; q++) s[q] = ld(P.s[q] + p);
            R q[NACC];
            p2g_terms(w, dx * wy * wz, wx * dy * wz, wx * wy * dz, m, ld(P.vol + p), v, s, m * (a.grav[0] * a.facl),
                      m * (a.grav[1] * a.facl), m * (a.grav[2] * a.facl), q);
            if constexpr (KIND == CELL_P2G_ACC) {
                // AccelP2G (map_and_interpolate.cpp:42-53): nforce += N m a
#pragma unroll
                for (int c = 0; c < 3; c++) q[5 + c] = w * m * ld(P.a[c] + p);
            }
            long long o[NACC];
            fx_terms(q, S, o);
#pragma unroll
            for (int f = 0; f < NACC; f++)
                if (o[f]) atomic_add_i64(&a.acc[(size_t)f * N + gn], o[f]);
            a.tileflag[tile_of_node(a.g, cx + i, cy + j, cz + k)] = 1;
        }
    }
    if (!MUSL && oobs) atomicAdd(&a.ctl->err_oob, oobs);
}

// -------------------------------------------------------------------- gather
// PIC: v = sum N G, FLIP: v += dt sum N G; geup = 2 vol sum dN nei and the sum
// of its squares (only when the shifting is on).  FP64 sums axis by axis
// (cell_field).
// With the MUSL scatter it replaces one staging-box kernel: 221 -> 99 us (FP64
// linear, 201,872 particles), 180 -> 50 us (FP32 B-splines, 216,000), 393 -> 99
// us (FP64 B-splines, 46,656).
template <typename R, int OX, int OY, int OZ>
__global__ void __launch_bounds__(256) k_gather(StepArgs<R> a) {
    constexpr int NX = OX + 1, NY = OY + 1, NZ = OZ + 1;
    pdl_wait();
    __shared__ Scales S;
    __shared__ long long sh_l[32];
    __shared__ float sh_f[32];
    musl_scales(a, S);
    const size_t N = (size_t)a.g.nodec, sy = (size_t)a.g.nnc[0], sz = sy * (size_t)a.g.nnc[1];
    const Particles<R> &P = a.P;
    const bool flip = a.scheme == MPM_FLIP, shift = a.shifting != 0;
    long long gacc = 0;
    float vmax = 0.0f;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < a.num; p += (int64_t)gridDim.x * blockDim.x) {
        R v[3] = {(R)0, (R)0, (R)0}, gu[3] = {(R)0, (R)0, (R)0};
        if constexpr (sizeof(R) == 4) {
            // FP32 B-splines: node by node, to the bit as k_g2p_musl_box
            const R x0 = ld(P.x[0] + p), x1 = ld(P.x[1] + p), x2 = ld(P.x[2] + p);
            bool oob = false;
            const int cx = cell_of(x0, a.g, 0, oob), cy = cell_of(x1, a.g, 1, oob), cz = cell_of(x2, a.g, 2, oob);
            Axis<R, OX> ax;
            Axis<R, OY> ay;
            Axis<R, OZ> az;
            axis_eval<R, OX>(x0, a.g, 0, cx, ax);
            axis_eval<R, OY>(x1, a.g, 1, cy, ay);
            axis_eval<R, OZ>(x2, a.g, 2, cz, az);
            if (flip) {
#pragma unroll
                for (int c = 0; c < 3; c++) v[c] = ld(P.v[c] + p);
            }
            const size_t b0 = node_id(a.g, cx, cy, cz);
#pragma unroll
            for (int k = 0; k < NZ; k++)
#pragma unroll
                for (int j = 0; j < NY; j++)
#pragma unroll
                    for (int i = 0; i < NX; i++) {
                        const R wxy = ax.w[i] * ay.w[j];
                        const R N_ = wxy * az.w[k];
                        const size_t gn = b0 + i + j * sy + k * sz;
                        if (flip) {
                            const R Nd = N_ * a.dt;
#pragma unroll
                            for (int c = 0; c < 3; c++) v[c] += Nd * ld(a.G + c * N + gn);
                        } else {
#pragma unroll
                            for (int c = 0; c < 3; c++) v[c] += N_ * ld(a.G + c * N + gn);
                        }
                        if (shift) {
                            const R e = ld(a.nei + gn);
                            gu[0] += ax.dw[i] * ay.w[j] * az.w[k] * e;
                            gu[1] += ax.w[i] * ay.dw[j] * az.w[k] * e;
                            gu[2] += wxy * az.dw[k] * e;
                        }
                    }
        } else {
            const R x[3] = {ld(P.x[0] + p), ld(P.x[1] + p), ld(P.x[2] + p)};
            CellWeights<R, OX, OY, OZ> w;
            const size_t b0 = cell_weights(a.g, x, w);
#pragma unroll
            for (int c = 0; c < 3; c++) cell_field<true, false>(a.G + c * N, b0, sy, sz, w, v[c], gu);
            R none;
            if (shift) cell_field<false, true>(a.nei, b0, sy, sz, w, none, gu);
#pragma unroll
            for (int c = 0; c < 3; c++)
                if (flip) v[c] = fma(a.dt, v[c], ld(P.v[c] + p));
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            P.v[c][p] = v[c];
        }
        vmax = fmaxf(vmax, fmaxf(fabsf((float)v[0]), fmaxf(fabsf((float)v[1]), fabsf((float)v[2]))));
        if (shift) {
            const R tv = (R)2 * ld(P.vol + p);
            const R g0 = gu[0] * tv, g1 = gu[1] * tv, g2 = gu[2] * tv;
            gacc += fx(g0 * g0 + g1 * g1 + g2 * g2, S.gd);
        }
    }
    const long long gsum = block_reduce(gacc, OpAddL(), sh_l);
    const float vm = block_reduce(vmax, OpMaxF(), sh_f);
    if (threadIdx.x == 0) {
        if (gsum) atomicAdd(&a.ctl->geup_acc, (unsigned long long)gsum);
        if (vm > 0.0f) atomic_max_pos(&a.ctl->nxt[a.parity ^ 1][B_VMAX], vm * 1.000001f);
    }
}

// ------------------------------------------------------------------ host side
template <typename R, int OX, int OY, int OZ, int KIND>
static void scatter_kind(const StepArgs<R> &a, int nbricks, int nsm, bool pdl, cudaStream_t st) {
    using C = CellShape<R, OX, OY, OZ>;
    auto *k = k_cell_scatter<R, OX, OY, OZ, KIND>;
    static int per_sm = 0;   // resident CTAs per SM
    if (per_sm == 0) {
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
        int q = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q, k, C::THREADS, C::SMEM) != cudaSuccess || q < 1) q = 1;
        per_sm = q;
    }
    // A CTA per brick's slab, as many as are resident.  Where the bricks leave room, more
    // for the shares of crowded ones, but not to the last place: the CTAs of a grid
    // that fills the chip are dealt out so that some SMs get two of the first ones
    // (FP64 linear, 97,336 particles, 168 bricks: 85 us in place of 53).
    const long long full = (long long)per_sm * nsm, bricks = (long long)nbricks * C::SLABS,
                    shares = a.num / SHARE_RUN * C::SLABS;
    const int grid = (int)(bricks >= full ? full : std::max(bricks, std::min(full - 8, bricks + shares)));
    launch(pdl, k, grid, C::THREADS, C::SMEM, st, a);
    launch(pdl, k_cell_misses<R, OX, OY, OZ, KIND>, 2 * nsm, 256, 0, st, a);
}

template <typename R, int OX, int OY, int OZ>
static void scatter_order(const StepArgs<R> &a, int kind, int nbricks, int nsm, bool pdl, cudaStream_t st) {
    if (kind == CELL_P2G_ACC) scatter_kind<R, OX, OY, OZ, CELL_P2G_ACC>(a, nbricks, nsm, pdl, st);
    // FP32 linear explicit grids have kernels of their own
    if constexpr (!(sizeof(R) == 4 && OX == 1 && OY == 1 && OZ == 1)) {
        if (kind == CELL_P2G) scatter_kind<R, OX, OY, OZ, CELL_P2G>(a, nbricks, nsm, pdl, st);
        else if (kind == CELL_P2G_AFF) scatter_kind<R, OX, OY, OZ, CELL_P2G_AFF>(a, nbricks, nsm, pdl, st);
        else if (kind == CELL_MUSL) scatter_kind<R, OX, OY, OZ, CELL_MUSL>(a, nbricks, nsm, pdl, st);
        else if (kind == CELL_MUSL_AFF) scatter_kind<R, OX, OY, OZ, CELL_MUSL_AFF>(a, nbricks, nsm, pdl, st);
    }
}

template <typename R>
void launch_cell_scatter(const StepArgs<R> &a, const int *o, int kind, int nbricks, int nsm, bool pdl,
                         cudaStream_t st) {
    if (o[0] == 1) scatter_order<R, 1, 1, 1>(a, kind, nbricks, nsm, pdl, st);
    else if (o[1] == 2) scatter_order<R, 2, 2, 2>(a, kind, nbricks, nsm, pdl, st);
    else scatter_order<R, 2, 1, 2>(a, kind, nbricks, nsm, pdl, st);
}

template <typename R>
void launch_gather(const StepArgs<R> &a, const int *o, int nsm, bool pdl, cudaStream_t st) {
    const long long nb = (a.num + 255) / 256;
    const int grid = (int)(nb < 8LL * nsm ? nb : 8LL * nsm);
    if (o[0] == 1) {
        if constexpr (sizeof(R) == 8) launch(pdl, k_gather<R, 1, 1, 1>, grid, 256, 0, st, a);
    } else if (o[1] == 2) {
        launch(pdl, k_gather<R, 2, 2, 2>, grid, 256, 0, st, a);
    } else {
        launch(pdl, k_gather<R, 2, 1, 2>, grid, 256, 0, st, a);
    }
}

template void launch_cell_scatter<float>(const StepArgs<float> &, const int *, int, int, int, bool, cudaStream_t);
template void launch_cell_scatter<double>(const StepArgs<double> &, const int *, int, int, int, bool, cudaStream_t);
template void launch_gather<float>(const StepArgs<float> &, const int *, int, bool, cudaStream_t);
template void launch_gather<double>(const StepArgs<double> &, const int *, int, bool, cudaStream_t);

}  // namespace mpm
