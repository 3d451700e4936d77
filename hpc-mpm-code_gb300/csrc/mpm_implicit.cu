// Implicit solid MPM on the GPU (FP64): generalized-alpha / Newmark time
// integration, Newton iteration, assembly of the stiffness operator into a
// 27-point block stencil, symmetric diagonal scaling, and a preconditioned
// conjugate-gradient solve with FP64 reductions.
//
// Reference (module/solid/implicit/, module/solver/, module/nonlinear_time_integration.cpp):
//   Particle2Node            var_trans_solid_implicit.cpp:20-80      -> run_p2g (AccelP2G mode) + k_imp_grid
//   SolveSolid (Newton)      solve_solid_implicit.cpp:65-103         -> implicit_newton
//   BCNRSet / Predict        implicit_mpm_solid.h:55-64,
//                            nonlinear_time_integration.cpp:59-71    -> k_imp_bcnr, k_imp_predict
//   AssembleSystem           solve_solid_implicit.cpp:105-204        -> k_imp_assemble, k_imp_assemble_cells, k_imp_rhs_diag
//   ComputeTangentModulus    solve_solid_implicit.cpp:34-63          -> pair loop of k_imp_assemble
//   BuildDiagonalPreconditioner crsmat.cpp:87-184                     -> k_imp_rhs_diag, k_imp_scale
//   MatVecMult               solver.cpp:405-433                      -> k_imp_matvec, k_imp_matvec_split
//   GPBiCGSafe               solver.cpp:19-141                       -> conjugate gradients (the scaled
//                            system is symmetric), stopped on the same squared-norm ratio
//   CheckNRConvergence       solver.cpp:484-593                      -> newton_residuals
//   Node2Particle            var_trans_solid_implicit.cpp:106-167,
//                            nonlinear_time_integration.cpp:73-96    -> k_imp_g2p, k_imp_shift
//
// Matrix storage: for control point n and stencil slot s (the neighbours
// n + (dx, dy, dz) with |dx| <= rx, |dy| <= ry, |dz| <= rz, where the radius
// of an axis is its shape order: 1 for linear shape functions, 2 for the
// quadratic B-spline, so 27, 75 or 125 slots; s = (dx+rx) + sx ((dy+ry) +
// sy (dz+rz)), sx = 2 rx + 1), the 3x3 block entry q = s * 9 + 3 a + b lives
// at A[aidx(q, n, qp)], tiled by 32 control points and by pairs of entries:
// ((n / 32) * qp + q / 2) * 64 + (n % 32) * 2 + q % 2, qp = ceil(9 ns / 2).
// A thread reads entry pairs as one vector load and a warp reading its 32
// nodes' values walks one contiguous range (coalesced and DRAM-page
// friendly); no column indices (the grid is structured).
//
// Precision: a context of precision 64 computes and stores everything in
// FP64 (the parity mode).  Precision 32 keeps the particles (F as H = F - I),
// the assembly arithmetic and the matrix in FP32 and the matvec of the
// Krylov iterations in FP32 arithmetic; the Krylov vectors, their inner
// products and norms, the true residual b - A x (the FP32-stored matrix
// applied in FP64 arithmetic), the Newton check and the nodal kinematics
// stay FP64.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <type_traits>
#include <vector>

#include "mpm_device.cuh"
#include "mpm_nn.cuh"

namespace mpm {
mpm_status run_p2g(mpm_ctx *c, double facl);
}

struct ImpState {
    int nr_flag = 0;
    double alpha_f = 1, alpha_m = 1, gamma = 0.5, beta = 0.25, nb[6] = {0};
    int prec = 64;                         // 64: FP64 operator; 32: FP32 particles, assembly and matrix
    int qp = 122;                          // entry pairs per node of the stencil matrix (aidx)
    void *A = nullptr;                     // 9 ns values per node (FP64 or FP32), tiled by 32 nodes (aidx)
    double *adiag = nullptr, *b = nullptr;  // 3 * nodec
    double *x = nullptr, *r = nullptr, *p = nullptr, *Ap = nullptr, *xs = nullptr;
    double *ndispl = nullptr, *nvel = nullptr, *naccel = nullptr, *naccel_k = nullptr;
    double *nmass = nullptr, *nvof = nullptr, *nei = nullptr;
    double *bcval64 = nullptr;             // 3 * nodec prescribed BC values in FP64 (implicit_bc_changed)
    void *stress_k = nullptr;              // 6 * num, Newton stress of the step (particle precision)
    void *geup = nullptr;                  // 3 * num (particle precision)
    double *part = nullptr;                // reduction partials
    double *scal = nullptr;                // device scalars
    double *h_scal = nullptr;              // pinned mirror
    int nblk = 0;
    int64_t num_alloc = 0;
    int64_t krylov_total = 0, newton_total = 0;
    double last_rel = 0.0;
    // flexible CG with the learned preconditioner
    mpm_nn *net = nullptr;
    double *z = nullptr, *bs = nullptr;    // preconditioned residual, scaled RHS (3 * nodec)
    double *xstar = nullptr, *ev = nullptr; // training-pair harvest: converged solution, error
    double *gp = nullptr, *gq = nullptr;    // flexible GCR: GM directions and their images (GM * 3 * nodec)
    double *gqq = nullptr, *gbeta = nullptr;  // |A p|^2 of each kept direction, projection coefficients
    float *gqf = nullptr;                   // FP32 copies of the kept images (GM * 3 * nodec), for the dots
    size_t gst = 0;                         // values per direction slot: 3 * nodec, up to a multiple of four
    int64_t cg_launches = 0, gcr_launches = 0;   // launches in g_cg and g_gcr
    float *gp32 = nullptr, *gq32 = nullptr;  // FP32 operator: the directions and images in FP32 (GM * 3 * nodec)
    float *p32 = nullptr;                   // FP32 operator: the CG direction in FP32
    float *nf32 = nullptr;                  // FP32 copies of ndispl, nvel, naccel (3 N each) and nei (N) for the particles
    float *dfx = nullptr;                   // FP32 operator: x split into high and low FP32 parts (2 * 3 * nodec)
    unsigned *cnt = nullptr;                // block counters of the single-launch reductions (zero between launches)
    bool isotropic = false;                 // every material's tangent is isotropic (models -1, 0, 1)
    int fallbacks = 0;                      // solves that switched from the network to Jacobi
    int nn_applications = 0;
    // CUDA graphs of 8 Krylov iterations (CG; FCG with the network; FCG with Jacobi)
    cudaGraphExec_t g_cg = nullptr, g_fcg_nn = nullptr, g_fcg_jac = nullptr, g_gcr = nullptr;
    mpm_nn *g_net = nullptr;
    bool no_graph = false;
    bool gcr = true;      // learned preconditioner: flexible GCR first (else flexible CG only)
    int gm = 4;           // GCR window in use (1, 2, 4 or 8 <= GM directions; 4 measured fastest on the cantilever)
    bool debug = false;   // MPM_GB300_KRYLOV_TRACE set: residual history to stderr
};

namespace mpm {

constexpr int GM = 8;   // directions kept by the flexible GCR solver

enum Scal { S_RR0 = 0, S_RR1, S_PAP, S_RR_INIT, S_RES, S_IDOF, S_EU, S_GD, S_ZQ, S_PR, S_RRC, S_DZZ, S_DZR, S_THR, S_ITER, S_DONE, S_ALPHA, S_BETA, S_NSCAL };

struct ImpArgs {
    int nnc[3];
    int nel[3];
    int nodec;
    double xmin[3], dx[3], inv_dx[3];
    double dt, facl, mtol, grav[3];
    double af, am, gamma, nb[6];
    int nr_flag;
    int shifting;
    int scheme;
    int rad[3];   // stencil radius per axis (the shape order)
    int ns;       // stencil slots (2 rad + 1 per axis)
    int qp;       // entry pairs per node (aidx)
    int64_t num;
    const unsigned char *bcflag;
    const double *bcval;
    const double *nvol;
    const int *iprop;
    const double *matprop;
};

__host__ __device__ __forceinline__ size_t aidx(int q, int n, int qp) {
    return (((size_t)(n >> 5) * qp + (size_t)(q >> 1)) << 6) + (size_t)((n & 31) << 1) + (size_t)(q & 1);
}
static size_t a_size(int nodec, int qp) { return (size_t)((nodec + 31) / 32) * 64 * (size_t)qp; }

static ImpArgs imp_args(mpm_ctx *c) {
    ImpArgs a;
    memset(&a, 0, sizeof(a));
    for (int d = 0; d < 3; d++) {
        a.nnc[d] = c->g.nnc[d];
        a.nel[d] = c->g.nel[d];
        a.xmin[d] = c->g.xmin[d];
        a.dx[d] = c->g.dx[d];
        a.inv_dx[d] = 1.0 / c->g.dx[d];
        a.grav[d] = c->gravity[d];
    }
    a.nodec = c->g.nodec;
    a.dt = c->dt;
    a.facl = c->facl;
    a.mtol = c->mtol;
    ImpState *s = c->imp;
    a.af = s->alpha_f;
    a.am = s->alpha_m;
    a.gamma = s->gamma;
    for (int k = 0; k < 6; k++) a.nb[k] = s->nb[k];
    a.nr_flag = s->nr_flag;
    a.shifting = c->shifting;
    a.scheme = c->scheme;
    a.ns = 1;
    for (int d = 0; d < 3; d++) {
        a.rad[d] = c->g.order[d];
        a.ns *= 2 * a.rad[d] + 1;
    }
    a.qp = (9 * a.ns + 1) / 2;
    a.num = c->num;
    a.bcflag = c->d_bcflag;
    // prescribed values in FP64 whatever the context's precision (an FP32
    // context keeps its own copy in FP32, d_bcval)
    a.bcval = s->bcval64;
    a.nvol = c->d_nvol;
    a.iprop = c->d_iprop;
    a.matprop = c->d_matprop;
    return a;
}

// Particle fields of an implicit context (precision R; FP32 stores H = F - I in F)
template <typename R>
struct PView {
    R *x[3], *v[3], *F[9], *s[6], *m, *vol0, *vol, *acc[3];
    int *matid;
};

template <typename R>
static PView<R> pview(mpm_ctx *c) {
    PView<R> v;
    size_t n = c->pstride;
    R *f = (R *)c->pbuf[c->cur];
    for (int k = 0; k < 3; k++) v.x[k] = f + k * n;
    for (int k = 0; k < 3; k++) v.v[k] = f + (3 + k) * n;
    for (int k = 0; k < 9; k++) v.F[k] = f + (6 + k) * n;
    for (int k = 0; k < 6; k++) v.s[k] = f + (15 + k) * n;
    v.m = f + 21 * n;
    v.vol0 = f + 22 * n;
    v.vol = f + 23 * n;
    for (int k = 0; k < 3; k++) v.acc[k] = f + (24 + k) * n;
    v.matid = (int *)(f + 27 * n);
    return v;
}

__device__ __forceinline__ void node_ijk(int n, const int *nnc, int &i, int &j, int &k) {
    i = n % nnc[0];
    j = (n / nnc[0]) % nnc[1];
    k = n / (nnc[0] * nnc[1]);
}

template <typename R>
__device__ __forceinline__ KGeom<R> kgeom(const ImpArgs &a) {
    KGeom<R> g;
    for (int d = 0; d < 3; d++) {
        g.xmin[d] = (R)a.xmin[d];
        g.dx[d] = (R)a.dx[d];
        g.inv_dx[d] = (R)a.inv_dx[d];
        g.nel[d] = a.nel[d];
        g.nnc[d] = a.nnc[d];
        g.ntile[d] = 0;
    }
    g.nodec = a.nodec;
    return g;
}

// Shape functions at x (MakSf, module/shape_function.cpp:8-119) for shape
// orders OX, OY, OZ: weights, gradients and control-point ids of the
// (OX+1)(OY+1)(OZ+1) nodes in MakSf order (x fastest), and each node's
// offset inside the element's node box (for the stencil slot).
template <typename R, int OX, int OY, int OZ>
__device__ __forceinline__ void shape_nodes(const ImpArgs &a, const KGeom<R> &g, const R *x, R *N, R (*dN)[3],
                                            int *nid, bool &oob) {
    const int cx = cell_of(x[0], g, 0, oob), cy = cell_of(x[1], g, 1, oob), cz = cell_of(x[2], g, 2, oob);
    Axis<R, OX> ax;
    Axis<R, OY> ay;
    Axis<R, OZ> az;
    axis_eval<R, OX>(x[0], g, 0, cx, ax);
    axis_eval<R, OY>(x[1], g, 1, cy, ay);
    axis_eval<R, OZ>(x[2], g, 2, cz, az);
    int id = 0;
#pragma unroll
    for (int k = 0; k <= OZ; k++)
#pragma unroll
        for (int j = 0; j <= OY; j++)
#pragma unroll
            for (int i = 0; i <= OX; i++) {
                N[id] = ax.w[i] * ay.w[j] * az.w[k];
                dN[id][0] = ax.dw[i] * ay.w[j] * az.w[k];
                dN[id][1] = ax.w[i] * ay.dw[j] * az.w[k];
                dN[id][2] = ax.w[i] * ay.w[j] * az.dw[k];
                nid[id] = (cx + i) + a.nnc[0] * ((cy + j) + a.nnc[1] * (cz + k));
                id++;
            }
}

// ------------------------------------------------------------ node kernels
// Particle2Node's grid part: nvel = p/m, naccel = f/m, BCs (var_trans_solid_implicit.cpp:47-75)
__global__ void k_imp_grid(ImpArgs a, const unsigned long long *acc, const double *inv, double *nmass, double *nvof,
                           double *nvel, double *naccel) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= a.nodec) return;
    const size_t N = (size_t)a.nodec;
    const double m = (double)(long long)acc[n] * inv[0];
    nmass[n] = m;
    nvof[n] = (double)(long long)acc[N + n] * inv[1];
    const unsigned char bf = a.bcflag[n];
    for (int c = 0; c < 3; c++) {
        double v = 0.0, ac = 0.0;
        if (m > a.mtol) {
            v = (double)(long long)acc[(2 + c) * N + n] * inv[2] / m;
            ac = (double)(long long)acc[(5 + c) * N + n] * inv[3] / m;
        }
        if (bf & (1 << c)) {
            v = a.bcval[c * N + n] * a.facl;
            ac = 0.0;
        }
        nvel[c * N + n] = v;
        naccel[c * N + n] = ac;
    }
}

// BCNRSet (BCSetDt on ndispl) then PredictNewmarkBetaVelAndAccel's acceleration
__global__ void k_imp_predict(ImpArgs a, double *ndispl, const double *nvel, const double *naccel, double *naccel_k,
                              double *nvel_k, int set_bc) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= a.nodec) return;
    const size_t N = (size_t)a.nodec;
    const unsigned char bf = a.bcflag[n];
    for (int c = 0; c < 3; c++) {
        const size_t i = c * N + n;
        if (set_bc && (bf & (1 << c))) ndispl[i] = a.bcval[i] * a.dt * a.facl;
        const double d = ndispl[i];
        naccel_k[i] = a.nb[3] * d - a.nb[4] * nvel[i] - a.nb[5] * naccel[i];
        if (nvel_k) nvel_k[i] = a.nb[0] * d - a.nb[1] * nvel[i] - a.nb[2] * naccel[i];
    }
}

// ------------------------------------------------------------- assembly
// Material tangent of one particle in a factored form that the pair loop
// contracts with the scaled gradient a of the row node and the gradient b of
// the column node (K_ij = sum_kl a_k C_ikjl b_l of ComputeTangentModulus,
// solve_solid_implicit.cpp:34-63, written out for each model's C):
//   isotropic (models -1, 0, 1; C = lambda' I(x)I + 2 mu' I4sym):
//       K = lambda' a b^T + mu' b a^T + mu' (a.b) I
//   general (models 2, 3):
//       K = (G a) b^T + a (G' b)^T + alpha (a.b) I + gam b a^T
//           + eps (B a)(B b)^T + beta (a.B b) B + delta (B b)(B a)^T
// plus, with NR_flag, the geometric term ((sigma a).b) I.
template <typename R>
struct Tangent {
    bool general;
    R lam, mu;                    // isotropic
    R B[3][3], G[3][3], Gp[3][3];  // general
    R alpha, gam, eps, beta, delta;
};

// St.Venant-Kirchhoff (MatStVk's stif_mat, constitutive_model.cpp:160-183):
// C = lambda' b(x)b + mu' (b_ik b_jl + b_il b_jk), lambda' = lambda / J, mu' = mu / J, b = F F^T.
template <typename R>
__device__ __forceinline__ void tangent_stvk(Tangent<R> &t, const R F[3][3], R J, R E, R nu) {
    const R rd = (R)1 / (((R)1 + nu) * ((R)1 - (R)2 * nu));
    const R ij = (R)1 / J;
    t.general = true;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            t.B[i][j] = F[i][0] * F[j][0] + F[i][1] * F[j][1] + F[i][2] * F[j][2];
            t.G[i][j] = (R)0;
            t.Gp[i][j] = (R)0;
        }
    t.alpha = t.gam = (R)0;
    t.eps = nu * E * rd * ij;
    t.beta = t.delta = (R)0.5 * E * ((R)1 - (R)2 * nu) * rd * ij;
}

// Mooney-Rivlin (MatMooneyRivlin's stif_mat, constitutive_model.cpp:235-283)
// with B the isochoric b, I1, I2 its invariants, hp = bulk ln J / J, s the
// Cauchy stress, A = I1 B - B^2:
//   G  = (bulk / J - t1 / 3 + c4) I - 2/3 dev(s) - c3 A,  G' = -2/3 dev(s) - c3 A,
//   alpha = gam = t1 / 2 - hp,  eps = c2',  beta = delta = -c2' / 2,
// t1 = 4 (c1 I1 + 2 c2 I2) / (3 J), c2' = 4 c2 / J, c3 = 4 c2 / (3 J), c4 = 8 c2 I2 / (9 J).
template <typename R>
__device__ __forceinline__ void tangent_mooney_rivlin(Tangent<R> &t, const R F[3][3], R J, R lnJ, const R *s, R c1,
                                                      R c2, R bulk) {
    const R ij = (R)1 / J;
    const R k2 = exp((R)(-2.0 / 3.0) * lnJ);   // J^(-2/3)
    R B2[3][3];
    t.general = true;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) t.B[i][j] = k2 * (F[i][0] * F[j][0] + F[i][1] * F[j][1] + F[i][2] * F[j][2]);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) B2[i][j] = t.B[i][0] * t.B[0][j] + t.B[i][1] * t.B[1][j] + t.B[i][2] * t.B[2][j];
    const R i1 = t.B[0][0] + t.B[1][1] + t.B[2][2];
    const R i2 = (R)0.5 * (i1 * i1 - (B2[0][0] + B2[1][1] + B2[2][2]));
    const R hp = bulk * lnJ * ij;
    const R t1 = (R)4 * (c1 * i1 + (R)2 * c2 * i2) * ij / (R)3;
    const R c2p = (R)4 * c2 * ij, c3 = c2p / (R)3, c4 = (R)8 * c2 * i2 * ij / (R)9;
    const R sg[3][3] = {{s[0], s[5], s[4]}, {s[5], s[1], s[3]}, {s[4], s[3], s[2]}};
    const R tr3 = (s[0] + s[1] + s[2]) / (R)3;
    const R g0 = bulk * ij - t1 / (R)3 + c4;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const R dev = sg[i][j] - (i == j ? tr3 : (R)0);
            const R Aij = i1 * t.B[i][j] - B2[i][j];
            t.Gp[i][j] = (R)(-2.0 / 3.0) * dev - c3 * Aij;
            t.G[i][j] = t.Gp[i][j] + (i == j ? g0 : (R)0);
        }
    t.alpha = t.gam = (R)0.5 * t1 - hp;
    t.eps = c2p;
    t.beta = t.delta = (R)(-0.5) * c2p;
}

// A particle's part of AssembleSystem (solve_solid_implicit.cpp:123-189):
// UpdateDefGrad with alpha_f, the stress of the Newton iterate (written to
// stress_k), the gradient correction dN <- dN dF^-1 and the tangent of its model.
template <typename R, int OX, int OY, int OZ>
__device__ __forceinline__ void imp_particle(const ImpArgs &a, const PView<R> &P, const R *ndispl, R *stress_k,
                                             int p, int *nid, R *Nw, R (*dN)[3], R *sk, R &vol, Tangent<R> &t) {
    constexpr int NE = (OX + 1) * (OY + 1) * (OZ + 1);
    const size_t N = (size_t)a.nodec, NP = (size_t)a.num;
    const KGeom<R> g = kgeom<R>(a);
    const R x[3] = {P.x[0][p], P.x[1][p], P.x[2][p]};
    bool oob = false;
    shape_nodes<R, OX, OY, OZ>(a, g, x, Nw, dN, nid, oob);
    // ComputeDeltaDefGrad with alpha_f (material_point.cpp:127-151): d = I + Dm
    R Dm[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    for (int q = 0; q < NE; q++)
        for (int r = 0; r < 3; r++) {
            const R u = (R)ndispl[r * N + nid[q]];
            for (int c = 0; c < 3; c++) Dm[r][c] += dN[q][c] * u;
        }
    const R af = (R)a.af;
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++) Dm[r][c] *= af;
    R d[3][3];
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++) d[r][c] = Dm[r][c] + (r == c ? (R)1 : (R)0);
    // UpdateDefGrad: Fn = d F.  FP32 stores H = F - I and forms
    // Hn = Dm + H + Dm H, J - 1 = det(I + Hn) - 1 without the rounding of numbers near 1.
    R Fn[3][3], Hn[3][3], J, jm1;
    if constexpr (sizeof(R) == 8) {
        R F[3][3];
        for (int r = 0; r < 3; r++)
            for (int c = 0; c < 3; c++) F[r][c] = P.F[3 * r + c][p];
        for (int r = 0; r < 3; r++)
            for (int c = 0; c < 3; c++) {
                R sum = 0.0;
                for (int k = 0; k < 3; k++) sum += d[r][k] * F[k][c];
                Fn[r][c] = sum;
            }
        J = det3(Fn);
        jm1 = J - (R)1;
    } else {
        R H[3][3];
        for (int r = 0; r < 3; r++)
            for (int c = 0; c < 3; c++) H[r][c] = P.F[3 * r + c][p];
        for (int r = 0; r < 3; r++)
            for (int c = 0; c < 3; c++) {
                R sum = Dm[r][c] + H[r][c];
                for (int k = 0; k < 3; k++) sum += Dm[r][k] * H[k][c];
                Hn[r][c] = sum;
            }
        jm1 = det_ipm1(Hn);
        J = (R)1 + jm1;
        for (int r = 0; r < 3; r++)
            for (int c = 0; c < 3; c++) Fn[r][c] = Hn[r][c] + (r == c ? (R)1 : (R)0);
    }
    vol = J * P.vol0[p];
    // UpdateConstitutiveModel on the Newton stress (constitutive_model.cpp:16-305)
    for (int k = 0; k < 6; k++) sk[k] = stress_k[k * NP + p];
    const int mid = P.matid[p];
    const int model = a.iprop[mid];
    const R E = (R)a.matprop[3 * mid], nu = (R)a.matprop[3 * mid + 1], m3 = (R)a.matprop[3 * mid + 2];
    t.general = false;
    t.lam = t.mu = (R)0;
    if (model == 0) {
        // the strain increment: FP64 takes d - I as the reference does, FP32 the exact Dm
        R De[3][3];
        for (int r = 0; r < 3; r++)
            for (int c = 0; c < 3; c++)
                De[r][c] = sizeof(R) == 8 ? (r == c ? d[r][c] - (R)1 : d[r][c]) : Dm[r][c];
        lin_elast_update(sk, De, E, nu);
        t.lam = E * nu / (((R)1 - (R)2 * nu) * ((R)1 + nu));
        t.mu = E / ((R)2 * ((R)1 + nu));
    } else if (model == 1) {
        R lnj;
        if constexpr (sizeof(R) == 8) {
            lnj = neo_hookean_stress(sk, Fn, J, E, nu);
        } else {
            neo_hookean_stress_h(sk, Hn, jm1, E, nu);
            lnj = log1pf(jm1);
        }
        const R rd = (R)1 / (((R)1 + nu) * ((R)1 - (R)2 * nu));
        const R lmd = nu * E * rd;
        const R mu0 = (R)0.5 * E * ((R)1 - (R)2 * nu) * rd;
        const R ij = (R)1 / J;
        t.lam = lmd * ij;
        t.mu = (mu0 - lmd * lnj) * ij;
    } else if (model == 2) {
        if constexpr (sizeof(R) == 8) {
            stvk_stress(sk, Fn, J, E, nu);
        } else {
            stvk_stress_h(sk, Hn, jm1, E, nu);
        }
        tangent_stvk(t, Fn, J, E, nu);
    } else if (model == 3) {   // mat_prop = {c1, c2, bulk}
        R lnj;
        if constexpr (sizeof(R) == 8) {
            mooney_rivlin_stress(sk, Fn, J, E, nu, m3);
            lnj = log(J);
        } else {
            mooney_rivlin_stress_h(sk, Hn, jm1, E, nu, m3);
            lnj = log1pf(jm1);
        }
        tangent_mooney_rivlin(t, Fn, J, lnj, sk, E, nu, m3);
    } else {
        for (int k = 0; k < 6; k++) sk[k] = (R)0;
    }
    for (int k = 0; k < 6; k++) stress_k[k * NP + p] = sk[k];
    // ImplicitDsfCorr: dN <- dN d^-1 (material_point.cpp:153-172)
    R di[3][3];
    {
        const R det = (R)1 / det3(d);
        di[0][0] = (d[1][1] * d[2][2] - d[1][2] * d[2][1]) * det;
        di[0][1] = (d[0][2] * d[2][1] - d[0][1] * d[2][2]) * det;
        di[0][2] = (d[0][1] * d[1][2] - d[0][2] * d[1][1]) * det;
        di[1][0] = (d[1][2] * d[2][0] - d[1][0] * d[2][2]) * det;
        di[1][1] = (d[0][0] * d[2][2] - d[0][2] * d[2][0]) * det;
        di[1][2] = (d[0][2] * d[1][0] - d[0][0] * d[1][2]) * det;
        di[2][0] = (d[1][0] * d[2][1] - d[1][1] * d[2][0]) * det;
        di[2][1] = (d[0][1] * d[2][0] - d[0][0] * d[2][1]) * det;
        di[2][2] = (d[0][0] * d[1][1] - d[0][1] * d[1][0]) * det;
    }
    for (int q = 0; q < NE; q++) {
        R tq[3];
        for (int c = 0; c < 3; c++) tq[c] = dN[q][0] * di[0][c] + dN[q][1] * di[1][c] + dN[q][2] * di[2][c];
        for (int c = 0; c < 3; c++) dN[q][c] = tq[c];
    }
}

// The tangent blocks of each unordered node pair of one particle once (K_ba =
// K_ab^T: every C here has the major symmetry) + lumped mass, and the
// internal/external force into the RHS, with atomics; the RHS is summed in FP64.
template <typename R, int OX, int OY, int OZ>
__device__ __forceinline__ void imp_scatter(const ImpArgs &a, const PView<R> &P, int p, const int *nid, const R *Nw,
                                            const R (*dN)[3], const R *sk, R vol, const Tangent<R> &t, R *A,
                                            double *b) {
    constexpr int NX = OX + 1, NY = OY + 1, NZ = OZ + 1, NE = NX * NY * NZ;
    constexpr int SX = 2 * OX + 1, SY = 2 * OY + 1, NS = SX * SY * (2 * OZ + 1);
    const size_t N = (size_t)a.nodec;
    const R af = (R)a.af;
    const R sg[3][3] = {{sk[0], sk[5], sk[4]}, {sk[5], sk[1], sk[3]}, {sk[4], sk[3], sk[2]}};
    const R m = P.m[p];
    const R fx = (R)(a.grav[0] * a.facl), fy = (R)(a.grav[1] * a.facl), fz = (R)(a.grav[2] * a.facl);
    const R afv = af * vol;
    const R am = (R)a.am, nb3 = (R)a.nb[3];
    for (int qa = 0; qa < NE; qa++) {
        const int na = nid[qa];
        const int ia = qa % NX, ja = (qa / NX) % NY, ka = qa / (NX * NY);
        const R emd = nb3 * Nw[qa] * m;   // ComputeNRLumpedMat (material_point.h:144)
        R ah[3], Sa[3];
#pragma unroll
        for (int k = 0; k < 3; k++) ah[k] = afv * dN[qa][k];
#pragma unroll
        for (int k = 0; k < 3; k++)
            Sa[k] = a.nr_flag ? sg[k][0] * ah[0] + sg[k][1] * ah[1] + sg[k][2] * ah[2] : (R)0;
        // isotropic: L = lambda' a, M = mu' a, T = M + sigma a;  general: G a, B a
        R L[3], M[3], T[3], Ga[3], Ba[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            L[k] = t.lam * ah[k];
            M[k] = t.mu * ah[k];
            T[k] = M[k] + Sa[k];
        }
        if (t.general) {
#pragma unroll
            for (int k = 0; k < 3; k++) {
                Ga[k] = t.G[k][0] * ah[0] + t.G[k][1] * ah[1] + t.G[k][2] * ah[2];
                Ba[k] = t.B[k][0] * ah[0] + t.B[k][1] * ah[1] + t.B[k][2] * ah[2];
            }
        }
#pragma unroll 1
        for (int qb = qa; qb < NE; qb++) {
            const int nbn = nid[qb];
            const int dxo = qb % NX - ia, dyo = (qb / NX) % NY - ja, dzo = qb / (NX * NY) - ka;
            const int sl = (dxo + OX) + SX * ((dyo + OY) + SY * (dzo + OZ));
            const R db[3] = {dN[qb][0], dN[qb][1], dN[qb][2]};
            R K[3][3];
            if (!t.general) {
                const R dg = T[0] * db[0] + T[1] * db[1] + T[2] * db[2];
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = 0; j < 3; j++) K[i][j] = L[i] * db[j] + M[j] * db[i] + (i == j ? dg : (R)0);
            } else {
                R Bb[3], Gb[3];
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    Bb[k] = t.B[k][0] * db[0] + t.B[k][1] * db[1] + t.B[k][2] * db[2];
                    Gb[k] = t.Gp[k][0] * db[0] + t.Gp[k][1] * db[1] + t.Gp[k][2] * db[2];
                }
                const R ab = ah[0] * db[0] + ah[1] * db[1] + ah[2] * db[2];
                const R aBb = ah[0] * Bb[0] + ah[1] * Bb[1] + ah[2] * Bb[2];
                const R sab = Sa[0] * db[0] + Sa[1] * db[1] + Sa[2] * db[2];
                const R dg = t.alpha * ab + sab;
                const R bsc = t.beta * aBb;
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = 0; j < 3; j++)
                        K[i][j] = Ga[i] * db[j] + ah[i] * Gb[j] + t.gam * db[i] * ah[j] + t.eps * Ba[i] * Bb[j] +
                                  t.delta * Bb[i] * Ba[j] + bsc * t.B[i][j] + (i == j ? dg : (R)0);
            }
            if (qa == qb) {
#pragma unroll
                for (int i = 0; i < 3; i++) K[i][i] += am * emd;
            }
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    atomicAdd(&A[aidx(sl * 9 + 3 * i + j, na, a.qp)], K[i][j]);
                    if (qb != qa) atomicAdd(&A[aidx((NS - 1 - sl) * 9 + 3 * j + i, nbn, a.qp)], K[i][j]);
                }
        }
        const R f0 = -vol * (sk[0] * dN[qa][0] + sk[5] * dN[qa][1] + sk[4] * dN[qa][2]) + Nw[qa] * (m * fx);
        const R f1 = -vol * (sk[5] * dN[qa][0] + sk[1] * dN[qa][1] + sk[3] * dN[qa][2]) + Nw[qa] * (m * fy);
        const R f2 = -vol * (sk[4] * dN[qa][0] + sk[3] * dN[qa][1] + sk[2] * dN[qa][2]) + Nw[qa] * (m * fz);
        atomicAdd(&b[na], (double)f0);
        atomicAdd(&b[N + na], (double)f1);
        atomicAdd(&b[2 * N + na], (double)f2);
    }
}

// One thread per particle: its part, then its pairs with atomics.  R is the
// particle precision and the precision of the arithmetic and of A.
template <typename R, int OX, int OY, int OZ>
__global__ void __launch_bounds__(128) k_imp_assemble(ImpArgs a, PView<R> P, const R *ndispl, R *stress_k,
                                                      R *A, double *b) {
    constexpr int NE = (OX + 1) * (OY + 1) * (OZ + 1);
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.num) return;
    int nid[NE];
    R Nw[NE], dN[NE][3], sk[6], vol;
    Tangent<R> t;
    imp_particle<R, OX, OY, OZ>(a, P, ndispl, stress_k, p, nid, Nw, dN, sk, vol, t);
    imp_scatter<R, OX, OY, OZ>(a, P, p, nid, Nw, dN, sk, vol, t, A, b);
}

// The assembly of an FP32 operator whose materials are isotropic (models -1, 0,
// 1), cell by cell.  A particle adds 576 numbers to the matrix (8 nodes) and its
// cell's other particles add to the same ones: with an atomic each, the assembly
// waited for the memory system (1,728,000 particles: 1.1e9 atomics, 2.07 ms).
// Here a CTA takes CELLS cells of a brick: its threads form their particles'
// parts in shared memory, then BG threads per cell and row node sum that node's
// blocks with NB column nodes over the cell's particles in registers and add
// each once, two entries per reduction.  What is left is bound by registers and
// latency (72 sums a thread): 16 cells and 128 particles per CTA, three CTAs per
// SM held to 168 registers, beat 32 cells in one CTA (592 to 741 us) and two or
// four threads per row node (790 to 1018).  The class with scaling and RHS, per
// Newton iteration: 1,728,000 particles 2217 -> 592 us, 232,320 372 -> 150, quadratic
// B-splines (87,808) 870 -> 439.  A round's particles are neighbours in the sorted
// order, so crowded cells take turns: at 216 particles per linear cell the class takes
// 1060 us for 216,000 particles, as the atomics do, and 813 in place of 248 for 27,000
// (a whole step of theirs still 2.5 ms in place of 3.6).
// A particle outside its sorted cell scatters with atomics of its own.
template <int OX, int OY, int OZ>
struct AsmShape {
    static constexpr int NX = OX + 1, NY = OY + 1, NZ = OZ + 1, NE = NX * NY * NZ;
    static constexpr int SX = 2 * OX + 1, SY = 2 * OY + 1, NS = SX * SY * (2 * OZ + 1);
    static constexpr int BG = NE == 8 ? 1 : 3, NB = NE / BG;
    static constexpr int CELLS = NE == 8 ? 16 : NE == 18 ? 8 : 4;
    static constexpr int THREADS = CELLS * NE * BG;
    static constexpr int CH = NE == 8 ? 128 : 64, ST = CH + 1;          // particles per round; row stride
    static constexpr int F_N = 3 * NE, F_L = 4 * NE, F_M = F_L + 1, F_S = F_L + 2, F_MASS = F_L + 8, NFLD = F_L + 9;
    static constexpr size_t SMEM = sizeof(float) * NFLD * ST;
    static_assert((CELLS & (CELLS - 1)) == 0, "binary search");
    static_assert(NE % BG == 0 && THREADS >= CH, "one particle per thread and round");
};

__device__ __forceinline__ void red2(float *p, float x, float y) {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(x), "f"(y) : "memory");
}
// a double sum as an unevaluated pair of FP32 numbers (two-sum)
__device__ __forceinline__ void pair_add(float &s, float &e, float q) {
    const float t = __fadd_rn(s, q), u = __fsub_rn(t, s);
    e += __fadd_rn(__fsub_rn(s, __fsub_rn(t, u)), __fsub_rn(q, u));
    s = t;
}

template <int OX, int OY, int OZ>
__global__ void __launch_bounds__(AsmShape<OX, OY, OZ>::THREADS, (OX == 1 ? 3 : 1))
    k_imp_assemble_cells(ImpArgs a, PView<float> P, const float *ndispl, float *stress_k, float *A, double *b,
                         const int *cstart, const int *blist, const int *nblist, int nbx, int nby) {
    using C = AsmShape<OX, OY, OZ>;
    constexpr int NX = C::NX, NY = C::NY, NE = C::NE, NB = C::NB, ST = C::ST;
    extern __shared__ float sm[];   // [NFLD][ST]
    constexpr int SLABS = BRC / C::CELLS;
    const int item = blockIdx.x;
    if (item >= *nblist * SLABS) return;
    const int br = blist[item / SLABS], c0 = (item % SLABS) * C::CELLS;
    const int *cs = cstart + (size_t)br * (BRC + 1) + c0;
    const int P0 = cs[0], P1 = cs[C::CELLS];
    if (P0 == P1) return;
    const int lc = threadIdx.x / (NE * C::BG), rem = threadIdx.x % (NE * C::BG), na = rem % NE, b0 = (rem / NE) * NB;
    const int cell = c0 + lc;
    const int cx = (br % nbx) * BRX + cell % BRX, cy = ((br / nbx) % nby) * BRY + (cell / BRX) % BRY,
              cz = (br / (nbx * nby)) * BRZ + cell / (BRX * BRY);
    const int p0 = cs[lc], p1 = cs[lc + 1];
    const float afg = a.nr_flag ? (float)a.af : 0.0f, amb = (float)(a.am * a.nb[3]);
    const float gv[3] = {(float)(a.grav[0] * a.facl), (float)(a.grav[1] * a.facl), (float)(a.grav[2] * a.facl)};
    float K[NB][3][3], f[3] = {0.0f, 0.0f, 0.0f}, fe[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int q = 0; q < NB; q++)
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) K[q][i][j] = 0.0f;
    for (int r0 = P0; r0 < P1; r0 += C::CH) {
        const int l = threadIdx.x, p = r0 + l;
        if (l < C::CH && p < P1) {
            int nid[NE];
            float Nw[NE], dN[NE][3], sk[6], vol;
            Tangent<float> t;
            imp_particle<float, OX, OY, OZ>(a, P, ndispl, stress_k, p, nid, Nw, dN, sk, vol, t);
            // its sorted cell is the one whose range holds p; its own cell's first node is nid[0]
            int q = 0;
#pragma unroll
            for (int h = C::CELLS / 2; h >= 1; h /= 2)
                if (cs[q + h] <= p) q += h;
            const int oc = c0 + q;
            const int ox = (br % nbx) * BRX + oc % BRX, oy = ((br / nbx) % nby) * BRY + (oc / BRX) % BRY,
                      oz = (br / (nbx * nby)) * BRZ + oc / (BRX * BRY);
            const bool mine = nid[0] == ox + a.nnc[0] * (oy + a.nnc[1] * oz);
            if (!mine) imp_scatter<float, OX, OY, OZ>(a, P, p, nid, Nw, dN, sk, vol, t, A, b);
            const float on = mine ? 1.0f : 0.0f, afv = (float)a.af * vol;
#pragma unroll
            for (int e = 0; e < NE; e++) {
#pragma unroll
                for (int c = 0; c < 3; c++) sm[(3 * e + c) * ST + l] = mine ? dN[e][c] : 0.0f;
                sm[(C::F_N + e) * ST + l] = mine ? Nw[e] : 0.0f;
            }
            sm[C::F_L * ST + l] = mine ? t.lam * afv : 0.0f;
            sm[C::F_M * ST + l] = mine ? t.mu * afv : 0.0f;
#pragma unroll
            for (int e = 0; e < 6; e++) sm[(C::F_S + e) * ST + l] = mine ? vol * sk[e] : 0.0f;
            sm[C::F_MASS * ST + l] = on * P.m[p];
        }
        __syncthreads();
        const int q1 = min(p1, r0 + C::CH);
        for (int pp = max(p0, r0); pp < q1; pp++) {
            const float *s = sm + (pp - r0);
            const float av[3] = {s[(3 * na) * ST], s[(3 * na + 1) * ST], s[(3 * na + 2) * ST]};
            const float lam = s[C::F_L * ST], mu = s[C::F_M * ST], m = s[C::F_MASS * ST], N_ = s[(C::F_N + na) * ST];
            const float S[6] = {s[C::F_S * ST], s[(C::F_S + 1) * ST], s[(C::F_S + 2) * ST],
                                s[(C::F_S + 3) * ST], s[(C::F_S + 4) * ST], s[(C::F_S + 5) * ST]};
            // vol sigma a: the force of node a and, times alpha_f, the geometric term
            const float Sa[3] = {S[0] * av[0] + S[5] * av[1] + S[4] * av[2], S[5] * av[0] + S[1] * av[1] + S[3] * av[2],
                                 S[4] * av[0] + S[3] * av[1] + S[2] * av[2]};
            float L[3], M[3], T[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                L[c] = lam * av[c];
                M[c] = mu * av[c];
                T[c] = fmaf(afg, Sa[c], M[c]);
            }
#pragma unroll
            for (int q = 0; q < NB; q++) {
                const float bv[3] = {s[(3 * (b0 + q)) * ST], s[(3 * (b0 + q) + 1) * ST], s[(3 * (b0 + q) + 2) * ST]};
                const float dg = T[0] * bv[0] + T[1] * bv[1] + T[2] * bv[2];
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        float v = fmaf(L[i], bv[j], K[q][i][j]);
                        if (i == j) v += dg;
                        K[q][i][j] = fmaf(M[j], bv[i], v);
                    }
            }
            const float emd = amb * N_ * m;
#pragma unroll
            for (int q = 0; q < NB; q++)
                if (b0 + q == na) K[q][0][0] += emd, K[q][1][1] += emd, K[q][2][2] += emd;
            if (b0 == 0) {
                const float Nm = N_ * m;
#pragma unroll
                for (int c = 0; c < 3; c++) pair_add(f[c], fe[c], fmaf(Nm, gv[c], -Sa[c]));
            }
        }
        __syncthreads();   // shared memory is reused by the next round
    }
    if (p0 == p1) return;
    const int ia = na % NX, ja = (na / NX) % NY, ka = na / (NX * NY);
    const int node = (cx + ia) + a.nnc[0] * ((cy + ja) + a.nnc[1] * (cz + ka));
#pragma unroll
    for (int q = 0; q < NB; q++) {
        const int nb = b0 + q;
        const int sl = (nb % NX - ia + OX) + C::SX * (((nb / NX) % NY - ja + OY) + C::SY * (nb / (NX * NY) - ka + OZ));
        const float *v = &K[q][0][0];
        float *row = A + aidx(9 * sl, node, a.qp);   // entry 9 sl: the first of a pair when sl is even
        const bool odd = sl & 1;
        // the other half of a pair is the next address, the next pair 64 on
        float *pr = odd ? row + 63 : row;
        atomicAdd(odd ? row : pr + 4 * 64, odd ? v[0] : v[8]);
#pragma unroll
        for (int u = 0; u < 4; u++)
            red2(pr + 64 * u, odd ? v[2 * u + 1] : v[2 * u], odd ? v[2 * u + 2] : v[2 * u + 1]);
    }
    if (b0 == 0) {
        const size_t N = (size_t)a.nodec;
#pragma unroll
        for (int c = 0; c < 3; c++) atomicAdd(&b[c * N + node], (double)f[c] + (double)fe[c]);
    }
}

// AddInertialForceToRHS (material_point.h:151-161) and the diagonal of the
// scaling D^-1/2 (crsmat.cpp:87-146, FEM_flag false)
template <typename R>
__global__ void k_imp_rhs_diag(ImpArgs a, const R *A, const double *nmass, const double *naccel_k,
                               const double *naccel, double *b, double *adiag) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= a.nodec) return;
    const size_t N = (size_t)a.nodec;
    const int dslot = (a.ns - 1) / 2;
    for (int c = 0; c < 3; c++) {
        const double aam = a.am * naccel_k[c * N + n] + (1.0 - a.am) * naccel[c * N + n];
        b[c * N + n] -= nmass[n] * aam;
        const double dg = fabs((double)A[aidx(dslot * 9 + 4 * c, n, a.qp)]);
        adiag[c * N + n] = dg < a.mtol ? 0.0 : 1.0 / sqrt(dg);
    }
}

// ApplyDiagonalScaling (crsmat.cpp:152-172)
template <typename R>
__global__ void k_imp_scale(ImpArgs a, R *A, const double *adiag) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= a.nodec) return;
    const size_t N = (size_t)a.nodec;
    int i, j, k;
    node_ijk(n, a.nnc, i, j, k);
    const int sx = 2 * a.rad[0] + 1, sy = 2 * a.rad[1] + 1;
    for (int s = 0; s < a.ns; s++) {
        const int ii = i + s % sx - a.rad[0], jj = j + (s / sx) % sy - a.rad[1], kk = k + s / (sx * sy) - a.rad[2];
        if (ii < 0 || jj < 0 || kk < 0 || ii >= a.nnc[0] || jj >= a.nnc[1] || kk >= a.nnc[2]) continue;
        const size_t col = ii + (size_t)a.nnc[0] * (jj + (size_t)a.nnc[1] * kk);
        if constexpr (sizeof(R) == 8) {
            for (int r = 0; r < 3; r++)
                for (int c = 0; c < 3; c++) A[aidx(s * 9 + 3 * r + c, n, a.qp)] *= adiag[r * N + n] * adiag[c * N + col];
        } else {
            // the FP32 matrix is scaled in FP32 (one FP64 operation per entry
            // would make this pass FP64-pipe bound)
            const float dr[3] = {(float)adiag[n], (float)adiag[N + n], (float)adiag[2 * N + n]};
            const float dc[3] = {(float)adiag[col], (float)adiag[N + col], (float)adiag[2 * N + col]};
            for (int r = 0; r < 3; r++)
                for (int c = 0; c < 3; c++) A[aidx(s * 9 + 3 * r + c, n, a.qp)] *= dr[r] * dc[c];
        }
    }
}

// ----------------------------------------------------------- reductions
// Per-block partial sums in fixed order; k_finish adds the partials in index order.
__device__ __forceinline__ double block_sum(double v, double *sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) r += sh[w];
    return r;
}

// Warp sums of V values (V a power of two <= 32) with the values spread over
// the lanes as the butterfly goes: at each of the first log2(V) steps a lane
// keeps half of its values and adds its partner's copy of that half, so a
// lane adds 2V - 1 + log2(32 / V) numbers instead of 5 V.  FP64 adds are the
// scarce resource on this part.  Returns the value index whose warp total the
// lane holds in v[0] (every lane of a group of 32 / V lanes holds it).
template <int V, typename T>
__device__ __forceinline__ int warp_sums(T (&v)[V]) {
    const int lane = threadIdx.x & 31;
    int j = 0, o = 16;
#pragma unroll
    for (int h = V / 2; h >= 1; h /= 2, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < h; i++) {
            const T send = up ? v[i] : v[i + h];
            const T keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
        if (up) j += h;
    }
    for (; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return j;
}

template <int V>
__device__ __forceinline__ bool partials_last(const double (&vin)[V], int nv, double *part, unsigned *cnt) {
    __shared__ double sh[V][8];   // CTAs of at most 8 warps
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double v[V];
#pragma unroll
    for (int j = 0; j < V; j++) v[j] = vin[j];
    const int j = warp_sums<V>(v);
    if ((lane & (32 / V - 1)) == 0) sh[j][wid] = v[0];
    __syncthreads();
    if ((int)threadIdx.x < nv) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[threadIdx.x][w];
        part[threadIdx.x * gridDim.x + blockIdx.x] = t;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(cnt, 1u) == gridDim.x - 1;
    __syncthreads();
    if (s_last) __threadfence();
    return s_last;
}

// in the last block: thread j < nv gets the total of value j over all blocks.  All
// values are read at once (a reduction per value waited for memory once each).
template <int V>
__device__ __forceinline__ double last_sums(const double *part, int nv) {
    __shared__ double sh[V][8];   // CTAs of at most 8 warps
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double t[V];
#pragma unroll
    for (int j = 0; j < V; j++) t[j] = 0.0;
#pragma unroll 4
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x)
#pragma unroll
        for (int j = 0; j < V; j++)
            if (j < nv) t[j] += __ldcg(part + (size_t)j * gridDim.x + i);
    const int jv = warp_sums<V>(t);
    if ((lane & (32 / V - 1)) == 0) sh[jv][wid] = t[0];
    __syncthreads();
    double s = 0.0;
    if ((int)threadIdx.x < nv)
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += sh[threadIdx.x][w];
    return s;
}

__global__ void k_finish(const double *part, int nblk, double *out, int slot) {
    __shared__ double sh[32];
    double acc = 0.0;
    for (int i = threadIdx.x; i < nblk; i += blockDim.x) acc += part[i];
    const double t = block_sum(acc, sh);
    if (threadIdx.x == 0) out[slot] = t;
}

// y = A x with BC rows zeroed (MatVecMult + BCResidualSet), optionally the block
// sums of dot(x, y) in part.  TA: storage of A; TC: arithmetic.  RX, RY, RZ: the
// stencil radius per axis.
template <typename TA, typename TC, int RX, int RY, int RZ>
__global__ void __launch_bounds__(256) k_imp_matvec(ImpArgs a, const TA *A, const double *x, double *y,
                                                    double *part) {
    using TA2 = typename std::conditional<sizeof(TA) == 8, double2, float2>::type;
    constexpr int SX = 2 * RX + 1, SY = 2 * RY + 1, NS = SX * SY * (2 * RZ + 1);
    __shared__ double sh[32];
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    double dot = 0.0;
    if (n < a.nodec) {
        const size_t N = (size_t)a.nodec;
        int i, j, k;
        node_ijk(n, a.nnc, i, j, k);
        TC acc[3] = {(TC)0, (TC)0, (TC)0};
#pragma unroll
        for (int s = 0; s < NS; s++) {
            const int ii = i + s % SX - RX, jj = j + (s / SX) % SY - RY, kk = k + s / (SX * SY) - RZ;
            if (ii < 0 || jj < 0 || kk < 0 || ii >= a.nnc[0] || jj >= a.nnc[1] || kk >= a.nnc[2]) continue;
            const size_t col = ii + (size_t)a.nnc[0] * (jj + (size_t)a.nnc[1] * kk);
            const TC x0 = (TC)x[col], x1 = (TC)x[N + col], x2 = (TC)x[2 * N + col];
            // the block's 9 entries: 4 aligned pairs and 1 single (which end depends on the parity of 9 s)
            TC e[9];
            if ((s & 1) == 0) {
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const TA2 v = __ldg(reinterpret_cast<const TA2 *>(A + aidx(s * 9 + 2 * t, n, a.qp)));
                    e[2 * t] = (TC)v.x;
                    e[2 * t + 1] = (TC)v.y;
                }
                e[8] = (TC)__ldg(A + aidx(s * 9 + 8, n, a.qp));
            } else {
                e[0] = (TC)__ldg(A + aidx(s * 9, n, a.qp));
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const TA2 v = __ldg(reinterpret_cast<const TA2 *>(A + aidx(s * 9 + 1 + 2 * t, n, a.qp)));
                    e[1 + 2 * t] = (TC)v.x;
                    e[2 + 2 * t] = (TC)v.y;
                }
            }
            // chained FMAs: in FP64 the FP64 pipe is this kernel's limit, and a
            // separate product and add per entry would cost a third more
#pragma unroll
            for (int r = 0; r < 3; r++) acc[r] = fma(e[3 * r + 2], x2, fma(e[3 * r + 1], x1, fma(e[3 * r], x0, acc[r])));
        }
        const unsigned char bf = a.bcflag[n];
        for (int c = 0; c < 3; c++) {
            const double v = (bf & (1 << c)) ? 0.0 : (double)acc[c];
            y[c * N + n] = v;
            if (part) dot += x[c * N + n] * v;
        }
    }
    if (part) {
        const double t = block_sum(dot, sh);
        if (threadIdx.x == 0) part[blockIdx.x] = t;
    }
}

// The same product with MV_G threads per control point, each of SL neighbouring
// slots (an even number, so that its entries start on a pair), added in order
// through shared memory.
// x in the precision TV of the arithmetic's input, y in TY; with `part`, the dot
// product of xd (FP64) and y goes to scal[slot] and scal[num] divided by it to
// S_ALPHA (num >= 0).  `done`: nothing to do when set.
constexpr int MV_NODES = 32, MV_G = 7;
template <typename TA, typename TC, int RX, int RY, int RZ, typename TV, typename TY>
__global__ void __launch_bounds__(MV_NODES * MV_G)
    k_imp_matvec_split(ImpArgs a, const TA *__restrict__ A, const TV *__restrict__ x, TY *__restrict__ y,
                       const double *__restrict__ xd, double *part, unsigned *cnt, double *scal, int slot, int num,
                       const double *done) {
    using TA2 = typename std::conditional<sizeof(TA) == 8, double2, float2>::type;
    constexpr int SX = 2 * RX + 1, SY = 2 * RY + 1, NS = SX * SY * (2 * RZ + 1);
    constexpr int SL = 2 * ((NS + 2 * MV_G - 1) / (2 * MV_G));
    static_assert(SL * MV_G >= NS, "every slot has a thread");
    __shared__ TC sh[MV_G][3][MV_NODES];
    pdl_wait();
    if (done && *done != 0.0) return;   // uniform over the grid
    const int lane = threadIdx.x % MV_NODES, grp = threadIdx.x / MV_NODES;
    const size_t N = (size_t)a.nodec;
    double dot = 0.0;
    const int n = blockIdx.x * MV_NODES + lane;
    TC acc[3] = {(TC)0, (TC)0, (TC)0};
    if (n < a.nodec) {
        int i, j, k;
        node_ijk(n, a.nnc, i, j, k);
#pragma unroll
        for (int q = 0; q < SL; q++) {
            const int s = grp * SL + q;
            const int ii = i + s % SX - RX, jj = j + (s / SX) % SY - RY, kk = k + s / (SX * SY) - RZ;
            if (s >= NS || ii < 0 || jj < 0 || kk < 0 || ii >= a.nnc[0] || jj >= a.nnc[1] || kk >= a.nnc[2]) continue;
            const size_t col = ii + (size_t)a.nnc[0] * (jj + (size_t)a.nnc[1] * kk);
            const TC x0 = (TC)x[col], x1 = (TC)x[N + col], x2 = (TC)x[2 * N + col];
            TC e[9];
            if ((q & 1) == 0) {
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const TA2 v = __ldg(reinterpret_cast<const TA2 *>(A + aidx(s * 9 + 2 * t, n, a.qp)));
                    e[2 * t] = (TC)v.x;
                    e[2 * t + 1] = (TC)v.y;
                }
                e[8] = (TC)__ldg(A + aidx(s * 9 + 8, n, a.qp));
            } else {
                e[0] = (TC)__ldg(A + aidx(s * 9, n, a.qp));
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const TA2 v = __ldg(reinterpret_cast<const TA2 *>(A + aidx(s * 9 + 1 + 2 * t, n, a.qp)));
                    e[1 + 2 * t] = (TC)v.x;
                    e[2 + 2 * t] = (TC)v.y;
                }
            }
#pragma unroll
            for (int r = 0; r < 3; r++) acc[r] = fma(e[3 * r + 2], x2, fma(e[3 * r + 1], x1, fma(e[3 * r], x0, acc[r])));
        }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) sh[grp][c][lane] = acc[c];
    __syncthreads();
    if (grp < 3 && n < a.nodec) {
        TC v = sh[0][grp][lane];
#pragma unroll
        for (int q = 1; q < MV_G; q++) v += sh[q][grp][lane];
        const double r = (a.bcflag[n] & (1 << grp)) ? 0.0 : (double)v;
        y[grp * N + n] = (TY)r;
        if (part) dot = xd[grp * N + n] * r;
    }
    if (part) {
        const double v[1] = {dot};
        if (!partials_last<1>(v, 1, part, cnt)) return;
        const double t = last_sums<1>(part, 1);
        if (threadIdx.x == 0) {
            scal[slot] = t;
            if (num >= 0) scal[S_ALPHA] = t != 0.0 ? scal[num] / t : 0.0;
            *cnt = 0u;
        }
    }
}

// x = xh + xl with FP32 parts (xl the rounding error of xh): 48 bits of x
__global__ void k_split_df(const double *__restrict__ x, float *__restrict__ xh, float *__restrict__ xl, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = x[i];
    const float h = (float)v;
    xh[i] = h;
    xl[i] = (float)(v - (double)h);
}

// y = A x for the FP32-stored stencil of the FP32 operator, in double-float
// arithmetic instead of FP64 (the true residual and the Newton check): each
// product e x = e (xh + xl) is e xh exactly (an FMA gives its rounding error)
// plus e xl, and the row sums are carried as an unevaluated FP32 pair
// (Knuth's two-sum for the high part).  About 44 bits of the sum, on the FP32
// pipe (GB300 executes 2 FP64 FMAs per SM and clock, against 128 FP32 lanes).
// The points' slots are split over MV_G threads as in k_imp_matvec_split, in the same
// pair arithmetic (one thread per point: 90 us at 274,625 points; the learned step,
// with five or six of them, 8.00 -> 7.81 ms).
template <int RX, int RY, int RZ>
__global__ void __launch_bounds__(MV_NODES * MV_G) k_imp_matvec_df(ImpArgs a, const float *__restrict__ A,
                                                                   const float *__restrict__ xh,
                                                                   const float *__restrict__ xl, double *y) {
    constexpr int SX = 2 * RX + 1, SY = 2 * RY + 1, NS = SX * SY * (2 * RZ + 1);
    constexpr int SL = 2 * ((NS + 2 * MV_G - 1) / (2 * MV_G));
    __shared__ float ph[MV_G][3][MV_NODES], pl[MV_G][3][MV_NODES];
    const int lane = threadIdx.x % MV_NODES, grp = threadIdx.x / MV_NODES;
    const int n = blockIdx.x * MV_NODES + lane;
    const size_t N = (size_t)a.nodec;
    float sh[3] = {0.0f, 0.0f, 0.0f}, sl[3] = {0.0f, 0.0f, 0.0f};
    int i = 0, j = 0, k = 0;
    if (n < a.nodec) node_ijk(n, a.nnc, i, j, k);
#pragma unroll
    for (int q = 0; q < SL; q++) {
        const int s = grp * SL + q;
        if (s >= NS || n >= a.nodec) continue;
        const int ii = i + s % SX - RX, jj = j + (s / SX) % SY - RY, kk = k + s / (SX * SY) - RZ;
        if (ii < 0 || jj < 0 || kk < 0 || ii >= a.nnc[0] || jj >= a.nnc[1] || kk >= a.nnc[2]) continue;
        const size_t col = ii + (size_t)a.nnc[0] * (jj + (size_t)a.nnc[1] * kk);
        const float h[3] = {__ldg(xh + col), __ldg(xh + N + col), __ldg(xh + 2 * N + col)};
        const float l[3] = {__ldg(xl + col), __ldg(xl + N + col), __ldg(xl + 2 * N + col)};
        float e[9];
        if ((q & 1) == 0) {   // SL is even
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const float2 v = __ldg(reinterpret_cast<const float2 *>(A + aidx(s * 9 + 2 * t, n, a.qp)));
                e[2 * t] = v.x;
                e[2 * t + 1] = v.y;
            }
            e[8] = __ldg(A + aidx(s * 9 + 8, n, a.qp));
        } else {
            e[0] = __ldg(A + aidx(s * 9, n, a.qp));
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const float2 v = __ldg(reinterpret_cast<const float2 *>(A + aidx(s * 9 + 1 + 2 * t, n, a.qp)));
                e[1 + 2 * t] = v.x;
                e[2 + 2 * t] = v.y;
            }
        }
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                // round-to-nearest intrinsics: the compiler may not fuse or
                // reorder them, which the error-free transformations rely on
                const float ev = e[3 * r + c];
                const float p = __fmul_rn(ev, h[c]);
                const float pe = fmaf(ev, h[c], -p);   // e xh - p, exactly
                const float sum = __fadd_rn(sh[r], p);   // two-sum of sh and p
                const float bp = __fsub_rn(sum, sh[r]);
                const float err = __fadd_rn(__fsub_rn(sh[r], __fsub_rn(sum, bp)), __fsub_rn(p, bp));
                sh[r] = sum;
                sl[r] += err + fmaf(ev, l[c], pe);
            }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
        ph[grp][c][lane] = sh[c];
        pl[grp][c][lane] = sl[c];
    }
    __syncthreads();
    if (grp >= 3 || n >= a.nodec) return;
    float s = ph[0][grp][lane], e = pl[0][grp][lane];
#pragma unroll
    for (int q = 1; q < MV_G; q++) {
        pair_add(s, e, ph[q][grp][lane]);
        e += pl[q][grp][lane];
    }
    y[grp * N + n] = (a.bcflag[n] & (1 << grp)) ? 0.0 : (double)s + (double)e;
}

// ScaleSolution + BCResidualSet: xs = x / D, r = b D (crsmat.cpp:190-209)
__global__ void k_cg_scale_in(ImpArgs a, const double *x, const double *b, const double *adiag, double *xs,
                              double *rr) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= a.nodec) return;
    const size_t N = (size_t)a.nodec;
    const unsigned char bf = a.bcflag[n];
    for (int c = 0; c < 3; c++) {
        const size_t i = c * N + n;
        const double dg = adiag[i];
        if (dg < a.mtol) {
            xs[i] = 0.0;
            rr[i] = 0.0;
        } else {
            xs[i] = x[i] / dg;
            rr[i] = b[i] * dg;
        }
        if (bf & (1 << c)) rr[i] = 0.0;
    }
}

// r = rr - Ax, p = r, partial r.r
__global__ void k_cg_init(ImpArgs a, const double *Ax, double *r, double *p, double *part) {
    __shared__ double sh[32];
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    double dot = 0.0;
    if (n < a.nodec) {
        const size_t N = (size_t)a.nodec;
        for (int c = 0; c < 3; c++) {
            const size_t i = c * N + n;
            const double v = r[i] - Ax[i];
            r[i] = v;
            p[i] = v;
            dot += v * v;
        }
    }
    const double t = block_sum(dot, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// num / den (0 when den is 0 or `zero`) evaluated by one thread of the block
// and shared: an FP64 division costs tens of FP64-pipe operations on this
// part, too many to repeat in every thread.  Every thread of the block must
// call it (it synchronises the block), at most once per kernel.
__device__ __forceinline__ double block_div(double num, double den, bool zero = false) {
    __shared__ double s_q;
    if (threadIdx.x == 0) s_q = (zero || den == 0.0) ? 0.0 : num / den;
    __syncthreads();
    return s_q;
}

// Four neighbouring values of a vector of m (a direction's slot starts on 16 bytes),
// zero past its end.
__device__ __forceinline__ void ld4(float (&v)[4], const float *p, int i, int m) {
    if (i + 4 <= m) {
        const float4 q = *reinterpret_cast<const float4 *>(p + i);
        v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++) v[e] = i + e < m ? p[i + e] : 0.0f;
    }
}
__device__ __forceinline__ void ld4(double (&v)[4], const double *p, int i, int m) {
    if (i + 4 <= m) {
        const double2 a = *reinterpret_cast<const double2 *>(p + i), b = *reinterpret_cast<const double2 *>(p + i + 2);
        v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++) v[e] = i + e < m ? p[i + e] : 0.0;
    }
}
__device__ __forceinline__ void st4(float *p, const float (&v)[4], int i, int m) {
    if (i + 4 <= m) {
        *reinterpret_cast<float4 *>(p + i) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (i + e < m) p[i + e] = v[e];
    }
}
__device__ __forceinline__ void st4(double *p, const double (&v)[4], int i, int m) {
    if (i + 4 <= m) {
        *reinterpret_cast<double2 *>(p + i) = make_double2(v[0], v[1]);
        *reinterpret_cast<double2 *>(p + i + 2) = make_double2(v[2], v[3]);
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (i + e < m) p[i + e] = v[e];
    }
}

// p.Ap to S_PAP and alpha = scal[cur] / p.Ap to S_ALPHA, where the product does not
// form it (mv_dot)
__global__ void __launch_bounds__(256) k_cg_dot(const double *p, const double *Ap, int m, double *part, unsigned *cnt,
                                                double *scal, int cur, const double *done) {
    pdl_wait();
    if (done && *done != 0.0) return;   // uniform over the grid
    const int i = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    double v[1] = {0.0};
    if (i < m) {
        double x[4], y[4];
        ld4(x, p, i, m);
        ld4(y, Ap, i, m);
#pragma unroll
        for (int e = 0; e < 4; e++) v[0] = fma(x[e], y[e], v[0]);
    }
    if (!partials_last<1>(v, 1, part, cnt)) return;
    const double t = last_sums<1>(part, 1);
    if (threadIdx.x == 0) {
        scal[S_PAP] = t;
        scal[S_ALPHA] = t != 0.0 ? scal[cur] / t : 0.0;
        *cnt = 0u;
    }
}

// x += alpha p, r -= alpha Ap, then (last block) r.r and beta;  alpha = rr_cur / pAp
// and beta = rr_new / rr_cur are divided once, by the block that reduced them.
// stop: the pass belongs to a solve that ends itself: nothing to do once S_DONE is
// set, and the last block sets it when r.r is below S_THR (or not a number) and
// counts the iteration.  Every load is issued before the first store.
__global__ void __launch_bounds__(256) k_cg_update(ImpArgs a, double *scal, int cur, double *x, double *r,
                                                   const double *p, const double *Ap, double *part, unsigned *cnt,
                                                   int stop) {
    pdl_wait();
    if (stop && scal[S_DONE] != 0.0) return;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    const size_t N = (size_t)a.nodec;
    double xv[3], rv[3], pv[3], qv[3];
    if (n < a.nodec) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const size_t i = c * N + n;
            xv[c] = x[i], rv[c] = r[i], pv[c] = p[i], qv[c] = Ap[i];
        }
    }
    const double alpha = scal[S_ALPHA];
    double dot = 0.0;
    if (n < a.nodec) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const size_t i = c * N + n;
            x[i] = xv[c] + alpha * pv[c];
            const double v = rv[c] - alpha * qv[c];
            r[i] = v;
            dot += v * v;
        }
    }
    const double v[1] = {dot};
    if (!partials_last<1>(v, 1, part, cnt)) return;
    const double t = last_sums<1>(part, 1);
    if (threadIdx.x == 0) {
        scal[cur ^ 1] = t;
        scal[S_BETA] = scal[cur] != 0.0 ? t / scal[cur] : 0.0;
        *cnt = 0u;
        if (stop) {
            scal[S_ITER] += 1.0;
            if (!(t >= scal[S_THR])) scal[S_DONE] = 1.0;
        }
    }
}

// p = r + beta p; p32: the copy of p that the FP32 operator multiplies (null: none)
__global__ void __launch_bounds__(256) k_cg_dir(ImpArgs a, const double *scal, const double *r, double *p, float *p32,
                                                int stop) {
    pdl_wait();
    if (stop && scal[S_DONE] != 0.0) return;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    const size_t N = (size_t)a.nodec;
    if (n >= a.nodec) return;
    double rv[3], pv[3];
#pragma unroll
    for (int c = 0; c < 3; c++) rv[c] = r[c * N + n], pv[c] = p[c * N + n];
    const double beta = scal[S_BETA];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const size_t i = c * N + n;
        const double v = rv[c] + beta * pv[c];
        p[i] = v;
        if (p32) p32[i] = (float)v;
    }
}

// (re)starts a solve from the residual r: p = r, the iteration count `it` and the
// threshold that ends it
__global__ void k_cg_start(ImpArgs a, double *scal, double thr, int it, const double *r, double *p, float *p32) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        scal[S_THR] = thr;
        scal[S_ITER] = (double)it;
        scal[S_DONE] = 0.0;
    }
    if (i >= 3 * a.nodec) return;
    const double v = r[i];
    p[i] = v;
    if (p32) p32[i] = (float)v;
}

// RestorSolution: x = xs D (crsmat.cpp:214-230)
__global__ void k_cg_scale_out(ImpArgs a, const double *xs, const double *adiag, double *x) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= 3 * a.nodec) return;
    x[n] = adiag[n] > a.mtol ? xs[n] * adiag[n] : 0.0;
}

// Newton residual of the linear system (ComputeRefResidual / ComputeAbsResidual,
// solver.cpp:484-555): b with BC rows zeroed, r = b - (A (x / D)) / D
__global__ void k_imp_prepare_residual(ImpArgs a, const double *x, const double *adiag, double *b, double *xs) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= a.nodec) return;
    const size_t N = (size_t)a.nodec;
    const unsigned char bf = a.bcflag[n];
    for (int c = 0; c < 3; c++) {
        const size_t i = c * N + n;
        if (bf & (1 << c)) b[i] = 0.0;
        xs[i] = adiag[i] > a.mtol ? x[i] / adiag[i] : 0.0;
    }
}

__global__ void k_imp_residual(ImpArgs a, const double *Ax, const double *adiag, const double *b, double *part) {
    __shared__ double sh[32];
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    double rr = 0.0, cnt = 0.0;
    if (n < a.nodec) {
        const size_t N = (size_t)a.nodec;
        for (int c = 0; c < 3; c++) {
            const size_t i = c * N + n;
            const double axp = adiag[i] > a.mtol ? Ax[i] / adiag[i] : 0.0;
            const double r = b[i] - axp;
            rr += r * r;
            if (adiag[i] > a.mtol) cnt += 1.0;
        }
    }
    const double t = block_sum(rr, sh);
    const double u = block_sum(cnt, sh);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = t;
        part[gridDim.x + blockIdx.x] = u;
    }
}

// ---------------------------------------------------------------- G2P
// nei = max(0, nvof - nvol) and sum nei^2 (material_point.cpp:175-185)
__global__ void k_imp_nei(ImpArgs a, const double *nvof, double *nei, double *part) {
    __shared__ double sh[32];
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    double e2 = 0.0;
    if (n < a.nodec) {
        const double e = fmax(0.0, -a.nvol[n] + nvof[n]);
        nei[n] = e;
        e2 = e * e;
    }
    const double t = block_sum(e2, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// Node2Particle (var_trans_solid_implicit.cpp:202-255) with the nodal kinematics
// already committed: F, J, vol, stress, displacement/acceleration/velocity
// gathers and the shifting gradient; CommitParticleKinematics without the shift.
template <typename R, int OX, int OY, int OZ>
__global__ void __launch_bounds__(128) k_imp_g2p(ImpArgs a, PView<R> P, const R *__restrict__ ndispl,
                                                 const R *__restrict__ nvel, const R *__restrict__ naccel,
                                                 const R *__restrict__ nei, R *geup, double *part, DevCtl *ctl,
                                                 int parity) {
    constexpr int NE = (OX + 1) * (OY + 1) * (OZ + 1);
    __shared__ double sh[32];
    __shared__ float sh_m[4][4];   // the four bounds of the block's warps
    float bnd[4] = {0.0f, 0.0f, 0.0f, 0.0f};   // |a|, |v|, vol, vol |sigma|
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    double gd = 0.0;
    if (p < a.num) {
        const size_t N = (size_t)a.nodec, NP = (size_t)a.num;
        const KGeom<R> g = kgeom<R>(a);
        const R x[3] = {P.x[0][p], P.x[1][p], P.x[2][p]};
        int nid[NE];
        R Nw[NE], dN[NE][3];
        bool oob = false;
        shape_nodes<R, OX, OY, OZ>(a, g, x, Nw, dN, nid, oob);
        R Dm[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
        for (int q = 0; q < NE; q++)
            for (int r = 0; r < 3; r++) {
                const R u = (R)ndispl[r * N + nid[q]];
                for (int c = 0; c < 3; c++) Dm[r][c] += dN[q][c] * (R)1 * u;
            }
        R d[3][3];
        for (int r = 0; r < 3; r++)
            for (int c = 0; c < 3; c++) d[r][c] = Dm[r][c] + (r == c ? (R)1 : (R)0);
        R Fn[3][3], Hn[3][3], J, jm1;
        if constexpr (sizeof(R) == 8) {
            R F[3][3];
            for (int r = 0; r < 3; r++)
                for (int c = 0; c < 3; c++) F[r][c] = P.F[3 * r + c][p];
            for (int r = 0; r < 3; r++)
                for (int c = 0; c < 3; c++) {
                    R sum = 0.0;
                    for (int k = 0; k < 3; k++) sum += d[r][k] * F[k][c];
                    Fn[r][c] = sum;
                }
            J = det3(Fn);
            jm1 = J - (R)1;
            for (int r = 0; r < 3; r++)
                for (int c = 0; c < 3; c++) P.F[3 * r + c][p] = Fn[r][c];
        } else {
            for (int r = 0; r < 3; r++)
                for (int c = 0; c < 3; c++) {
                    R sum = Dm[r][c] + P.F[3 * r + c][p];
                    for (int k = 0; k < 3; k++) sum += Dm[r][k] * P.F[3 * k + c][p];
                    Hn[r][c] = sum;
                }
            jm1 = det_ipm1(Hn);
            J = (R)1 + jm1;
            for (int r = 0; r < 3; r++)
                for (int c = 0; c < 3; c++) {
                    Fn[r][c] = Hn[r][c] + (r == c ? (R)1 : (R)0);
                    P.F[3 * r + c][p] = Hn[r][c];
                }
        }
        const R vol = J * P.vol0[p];
        P.vol[p] = vol;
        R sk[6];
        for (int k = 0; k < 6; k++) sk[k] = P.s[k][p];
        const int mid = P.matid[p];
        const int model = a.iprop[mid];
        const R E = (R)a.matprop[3 * mid], nu = (R)a.matprop[3 * mid + 1], m3 = (R)a.matprop[3 * mid + 2];
        if (model == 0) {
            R De[3][3];
            for (int r = 0; r < 3; r++)
                for (int c = 0; c < 3; c++)
                    De[r][c] = sizeof(R) == 8 ? (r == c ? d[r][c] - (R)1 : d[r][c]) : Dm[r][c];
            lin_elast_update(sk, De, E, nu);
        } else if (model == 1) {
            if constexpr (sizeof(R) == 8) neo_hookean_stress(sk, Fn, J, E, nu);
            else neo_hookean_stress_h(sk, Hn, jm1, E, nu);
        } else if (model == 2) {
            if constexpr (sizeof(R) == 8) stvk_stress(sk, Fn, J, E, nu);
            else stvk_stress_h(sk, Hn, jm1, E, nu);
        } else if (model == 3) {
            if constexpr (sizeof(R) == 8) mooney_rivlin_stress(sk, Fn, J, E, nu, m3);
            else mooney_rivlin_stress_h(sk, Hn, jm1, E, nu, m3);
        } else {
            for (int k = 0; k < 6; k++) sk[k] = (R)0;
        }
        for (int k = 0; k < 6; k++) P.s[k][p] = sk[k];
        const bool flip = (a.scheme == MPM_FLIP);
        // gathers in the particle precision (FP64 arithmetic for FP32
        // particles would make this pass FP64-pipe bound)
        R disp[3] = {0, 0, 0}, acc[3] = {0, 0, 0}, vel[3] = {0, 0, 0};
        const R aold[3] = {P.acc[0][p], P.acc[1][p], P.acc[2][p]};
        if (model != -1) {
            for (int q = 0; q < NE; q++)
                for (int c = 0; c < 3; c++) {
                    disp[c] += Nw[q] * (R)ndispl[c * N + nid[q]];
                    acc[c] += Nw[q] * (R)naccel[c * N + nid[q]];
                    if (!flip) vel[c] += Nw[q] * (R)nvel[c * N + nid[q]];
                }
        }
        // shifting gradient at the old position with the new volume (material_point.cpp:192-216)
        R gv[3] = {0, 0, 0};
        for (int q = 0; q < NE; q++)
            for (int c = 0; c < 3; c++) gv[c] += dN[q][c] * (R)nei[nid[q]];
        for (int c = 0; c < 3; c++) {
            gv[c] *= (R)2 * vol;
            geup[c * NP + p] = gv[c];
            gd += (double)gv[c] * (double)gv[c];
        }
        // CommitParticleKinematics (nonlinear_time_integration.cpp:83-96), shift added by k_imp_shift
        float amax = 0.0f, vmax = 0.0f;
        const R dtr = (R)a.dt, gam = (R)a.gamma;
        for (int c = 0; c < 3; c++) {
            const R vc = flip ? P.v[c][p] + dtr * (((R)1 - gam) * aold[c] + gam * acc[c]) : vel[c];
            P.v[c][p] = vc;
            P.acc[c][p] = acc[c];
            P.x[c][p] = x[c] + disp[c];
            amax = fmaxf(amax, (float)fabs(acc[c]));
            vmax = fmaxf(vmax, (float)fabs(vc));
        }
        const float f0 = fabsf((float)sk[0]), f1 = fabsf((float)sk[1]), f2 = fabsf((float)sk[2]),
                    f3 = fabsf((float)sk[3]), f4 = fabsf((float)sk[4]), f5 = fabsf((float)sk[5]);
        bnd[0] = amax;
        bnd[1] = vmax;
        bnd[2] = fabsf((float)vol);
        bnd[3] = bnd[2] * fmaxf(f0 + f5 + f4, fmaxf(f5 + f1 + f3, f4 + f3 + f2));
    }
    // the block's bounds: one atomic each (one per particle took half of this pass)
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 4; k++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float v = __shfl_xor_sync(0xffffffffu, bnd[k], o);
            bnd[k] = (v > bnd[k] || v != v) ? v : bnd[k];   // keeps a NaN, which atomic_max_pos turns into the largest bound
        }
        if (lane == 0) sh_m[k][wid] = bnd[k];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        constexpr int slot[4] = {B_AMAX, B_VMAX, B_VOLMAX, B_VOLSMAX};
        float v = 0.0f;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
            const float u = sh_m[threadIdx.x][w];
            v = (u > v || u != u) ? u : v;
            if (u != u) break;
        }
        int sl = slot[0];
#pragma unroll
        for (int k = 1; k < 4; k++)
            if ((int)threadIdx.x == k) sl = slot[k];
        atomic_max_pos(&ctl->nxt[parity ^ 1][sl], v * 1.000001f);
    }
    const double t = block_sum(gd, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// x += -b0 geup, b0 = eu / gd unless gd < mtol (material_point.cpp:219-225)
template <typename R>
__global__ void k_imp_shift(ImpArgs a, PView<R> P, const R *geup, const double *scal) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const double gd = scal[S_GD];
    const double b0 = block_div(scal[S_EU], gd, gd < a.mtol);
    if (p >= a.num || !a.shifting || b0 == 0.0) return;
    const size_t NP = (size_t)a.num;
    for (int c = 0; c < 3; c++) P.x[c][p] = (R)((double)P.x[c][p] + -b0 * (double)geup[c * NP + p]);
}

// ------------------------------------------------ flexible CG (Notay's FCG(1))
// partial dot u.w over the 3 * nodec vector (node-blocked like the matvec)
__global__ void k_dot3(ImpArgs a, const double *u, const double *w, double *part) {
    __shared__ double sh[32];
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    double d = 0.0;
    if (n < a.nodec) {
        const size_t N = (size_t)a.nodec;
        for (int c = 0; c < 3; c++) d += u[c * N + n] * w[c * N + n];
    }
    const double t = block_sum(d, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// p = z - (z.q_prev / p_prev.q_prev) p_prev (p = z on a restart); partial p.r
__global__ void k_fcg_dir(ImpArgs a, const double *scal, int restart, const double *z, const double *r, double *p,
                          double *part) {
    __shared__ double sh[32];
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    const double beta = block_div(-scal[S_ZQ], scal[S_PAP], restart != 0);
    double d = 0.0;
    if (n < a.nodec) {
        const size_t N = (size_t)a.nodec;
        for (int c = 0; c < 3; c++) {
            const size_t i = c * N + n;
            const double v = z[i] + beta * p[i];
            p[i] = v;
            d += v * r[i];
        }
    }
    const double t = block_sum(d, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// alpha = p.r / p.q; x += alpha p; r -= alpha q; partial r.r
__global__ void k_fcg_update(ImpArgs a, const double *scal, double *x, double *r, const double *p, const double *q,
                             double *part) {
    __shared__ double sh[32];
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    const double alpha = block_div(scal[S_PR], scal[S_PAP]);
    double d = 0.0;
    if (n < a.nodec) {
        const size_t N = (size_t)a.nodec;
        for (int c = 0; c < 3; c++) {
            const size_t i = c * N + n;
            x[i] += alpha * p[i];
            const double v = r[i] - alpha * q[i];
            r[i] = v;
            d += v * v;
        }
    }
    const double t = block_sum(d, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// true residual r = bs - Ax (scaled system, BC rows already zero in Ax and bs); partial r.r
__global__ void k_true_residual(ImpArgs a, const double *bs, const double *Ax, double *r, double *part) {
    __shared__ double sh[32];
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    double d = 0.0;
    if (n < a.nodec) {
        const size_t N = (size_t)a.nodec;
        for (int c = 0; c < 3; c++) {
            const size_t i = c * N + n;
            const double v = bs[i] - Ax[i];
            r[i] = v;
            d += v * v;
        }
    }
    const double t = block_sum(d, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// network feature channels: the mass term's share of each diagonal entry,
// phi = alpha_m nb3 nmass / diag (diag = 1 / adiag^2), clamped to [0, 1]
__global__ void k_phi(ImpArgs a, const double *nmass, const double *adiag, double *phi) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= a.nodec) return;
    const size_t N = (size_t)a.nodec;
    for (int c = 0; c < 3; c++) {
        const double d = adiag[c * N + n];
        const double v = a.am * a.nb[3] * nmass[n] * d * d;
        phi[c * N + n] = v < 0.0 ? 0.0 : (v > 1.0 ? 1.0 : v);
    }
}

// e = xstar - x
__global__ void k_sub3(const double *xstar, const double *x, double *e, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) e[i] = xstar[i] - x[i];
}

// seeded random right-hand side of the scaled system for training-pair
// harvesting: a few random low-wavenumber cosine modes per component
// (wavenumber 0, a uniform load, included) plus white noise, zero on
// inactive and boundary rows
__device__ __forceinline__ uint64_t hash64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ double hash_unit(uint64_t k) { return ((hash64(k) >> 11) + 0.5) * (1.0 / 9007199254740992.0); }

__global__ void k_random_rhs(ImpArgs a, const double *adiag, uint64_t seed, double smooth_amp, double noise_amp,
                             double *bs) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= a.nodec) return;
    int i, j, k;
    node_ijk(n, a.nnc, i, j, k);
    const size_t N = (size_t)a.nodec;
    const unsigned char bf = a.bcflag[n];
    for (int c = 0; c < 3; c++) {
        double v = 0.0;
        for (int m = 0; m < 4; m++) {
            const uint64_t key = seed * 1315423911ull + (uint64_t)(c * 4 + m) * 97;
            const double kx = floor(4.0 * hash_unit(key + 1)), ky = floor(4.0 * hash_unit(key + 2));
            const double kz = floor(4.0 * hash_unit(key + 3));
            const double ph = 6.283185307179586 * hash_unit(key + 4);
            const double amp = 2.0 * hash_unit(key + 5) - 1.0;
            v += amp * cos(3.141592653589793 * (kx * i / a.nnc[0] + ky * j / a.nnc[1] + kz * k / a.nnc[2]) + ph);
        }
        const uint64_t nk = seed * 2654435761ull + (uint64_t)n * 3 + c;
        const double u1 = hash_unit(nk * 2 + 11), u2 = hash_unit(nk * 2 + 12);
        const double g = sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2);
        const size_t idx = c * N + n;
        const bool off = (bf & (1 << c)) || !(adiag[idx] >= a.mtol);
        bs[idx] = off ? 0.0 : smooth_amp * v + noise_amp * g;
    }
}

__global__ void k_set_modulus(double *matprop, int nmat, double E) {
    const int m = threadIdx.x;
    if (m < nmat) matprop[3 * m] = E;
}

// ------------------------------------------------ flexible GCR(GM)
// slot of the direction kept j + 1 iterations before the one in `slot` (ring of w)
__device__ __forceinline__ int gcr_prev(int slot, int j, int w) { return (slot - 1 - j + 2 * w) % w; }

// The three passes of a flexible GCR iteration after the product q = A p.  Each is
// a pass over vectors that mostly sit in L2 (17, 46 and 42 MB at 274,625 nodes, FP32)
// and a reduction that its last block finishes; what they took was the chain of
// loads per thread and the last block's one reduction per value.  So a thread
// takes four neighbouring values with every load issued before the first use, the
// last block reads all partials at once, and each pass is launched while its
// predecessor drains.  Dots, axpy and update, 1,728,000 particles: 18.4 + 24.4 + 19.8 ->
// 11.0 + 21.4 + 15.8 us (the last with the network's input pass, 8.0 before).
//
// beta_j = (q . Q_j) / (Q_j . Q_j) with the `used` previous images (j = 0 the
// newest; W >= the window w).  beta only has to be close: the same beta_j update
// both the direction and its image (k_gcr_axpy), so A p = q holds whatever their
// accuracy and only the orthogonality of the kept images is at FP32 level.  So the
// dots run in FP32 on FP32 copies of the kept images (the FP64 pipe is this part's
// scarce resource), and the block partials are summed in FP64.
template <typename T, int W>
__global__ void __launch_bounds__(256) k_gcr_dots(const T *Q, const float *Qf, size_t st, int m, int slot, int used,
                                                  int w, double *part, unsigned *cnt, const double *qq,
                                                  double *beta) {
    __shared__ double shw[W][8];
    __shared__ bool s_last;
    pdl_wait();
    const int i = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    float d[W];
#pragma unroll
    for (int j = 0; j < W; j++) d[j] = 0.0f;
    if (i < m) {
        T q[4];
        float qj[W][4];
        ld4(q, Q + (size_t)slot * st, i, m);
#pragma unroll
        for (int j = 0; j < W; j++)   // past `used`: any slot, the dot is not used
            ld4(qj[j], Qf + (size_t)(j < used ? gcr_prev(slot, j, w) : slot) * st, i, m);
#pragma unroll
        for (int j = 0; j < W; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) d[j] += (float)q[e] * qj[j][e];
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int jv = warp_sums<W>(d);
    if ((lane & (32 / W - 1)) == 0) shw[jv][wid] = (double)d[0];
    __syncthreads();
    if ((int)threadIdx.x < used) {
        double t = 0.0;
        for (int q = 0; q < (int)(blockDim.x >> 5); q++) t += shw[threadIdx.x][q];
        part[threadIdx.x * gridDim.x + blockIdx.x] = t;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(cnt, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const double t = last_sums<W>(part, used);
    if ((int)threadIdx.x < used) {
        const double dq = qq[gcr_prev(slot, threadIdx.x, w)];
        beta[threadIdx.x] = dq > 0.0 ? t / dq : 0.0;
    }
    if (threadIdx.x == 0) *cnt = 0u;
}

// p -= sum beta_j P_j, q -= sum beta_j Q_j in the precision T of the directions
// (FP64: an FP32 copy of q is kept for the dots; FP32: the images themselves are
// what the dots read, Qf is null); then (last block) q.r, q.q (kept as the slot's)
// and alpha = q.r / q.q.
// rr: r.r after the coming update, r.r - (q.r)^2 / q.q, goes to S_RRC (the update
// then needs no reduction and can feed the network).  It is used where r is
// replaced by the true residual every few iterations (the FP32 operator): within
// those r.r falls by far less than the 2^52 that the difference could lose.
template <typename T, int W>
__global__ void __launch_bounds__(256) k_gcr_axpy(T *P, T *Q, float *Qf, size_t st, int m, int slot, int used, int w,
                                                  const double *beta, const double *r, double *qqs, double *part,
                                                  unsigned *cnt, double *scal, int rr) {
    pdl_wait();
    const int i = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    double v[2] = {0.0, 0.0};
    if (i < m) {
        T *p = P + (size_t)slot * st, *q = Q + (size_t)slot * st;
        T pv[4], qv[4], pj[W][4], qj[W][4], bj[W];
        double rv[4];
        ld4(pv, p, i, m);
        ld4(qv, q, i, m);
        ld4(rv, r, i, m);
#pragma unroll
        for (int j = 0; j < W; j++) {
            const size_t o = (size_t)(j < used ? gcr_prev(slot, j, w) : slot) * st;
            ld4(pj[j], P + o, i, m);
            ld4(qj[j], Q + o, i, m);
            bj[j] = j < used ? (T)beta[j] : (T)0;
        }
#pragma unroll
        for (int j = 0; j < W; j++)
            if (j < used)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    pv[e] -= bj[j] * pj[j][e];
                    qv[e] -= bj[j] * qj[j][e];
                }
        st4(p, pv, i, m);
        st4(q, qv, i, m);
        if (Qf) {   // the copy k_gcr_dots reads
            float qf[4];
#pragma unroll
            for (int e = 0; e < 4; e++) qf[e] = (float)qv[e];
            st4(Qf + (size_t)slot * st, qf, i, m);
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const double qd = (double)qv[e];
            v[0] = fma(qd, rv[e], v[0]);
            v[1] = fma(qd, qd, v[1]);
        }
    }
    if (!partials_last<2>(v, 2, part, cnt)) return;
    __shared__ double s_t[2];
    const double t = last_sums<2>(part, 2);
    if (threadIdx.x < 2) s_t[threadIdx.x] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        const double qr = s_t[0], qq = s_t[1], alpha = qq > 0.0 ? qr / qq : 0.0;
        scal[S_ALPHA] = alpha;
        qqs[slot] = qq;
        if (rr) {
            const double left = scal[S_RRC] - alpha * qr;
            scal[S_RRC] = left < 0.0 ? 0.0 : left;   // keeps a NaN
        }
        *cnt = 0u;
    }
}

// x += alpha p; r -= alpha q; then (last block) r.r
template <typename T>
__global__ void __launch_bounds__(256) k_gcr_update(double *scal, double *x, double *r, const T *P, const T *Q,
                                                    size_t st, int m, int slot, double *part, unsigned *cnt) {
    pdl_wait();
    const int i = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    const double alpha = scal[S_ALPHA];
    double v[1] = {0.0};
    if (i < m) {
        T p[4], q[4];
        double xv[4], rv[4];
        ld4(p, P + (size_t)slot * st, i, m);
        ld4(q, Q + (size_t)slot * st, i, m);
        ld4(xv, x, i, m);
        ld4(rv, r, i, m);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            xv[e] += alpha * (double)p[e];
            rv[e] -= alpha * (double)q[e];
            v[0] += rv[e] * rv[e];
        }
        st4(x, xv, i, m);
        st4(r, rv, i, m);
    }
    if (!partials_last<1>(v, 1, part, cnt)) return;
    const double rr = last_sums<1>(part, 1);
    if (threadIdx.x == 0) {
        scal[S_RRC] = rr;
        *cnt = 0u;
    }
}

// The same for the FP32 operator, whose r.r k_gcr_axpy left: no reduction, and the
// new residual goes straight into the network's input (feed; the next iteration's
// first pass, k_input_r, is then not needed).
__global__ void __launch_bounds__(256) k_gcr_update_feed(const double *scal, double *x, double *r,
                                                         const float *__restrict__ P, const float *__restrict__ Q,
                                                         size_t st, int nodec, int slot, int feed, nn::Input in) {
    __shared__ double s_inv;
    pdl_wait();
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    const size_t N = (size_t)nodec;
    if (threadIdx.x == 0) s_inv = nn::inv_rms(scal[S_RRC], nodec);
    __syncthreads();
    if (n >= nodec) return;
    const double alpha = scal[S_ALPHA], inv = s_inv;
    const float *p = P + (size_t)slot * st + n, *q = Q + (size_t)slot * st + n;
    double xv[3], rv[3];
    float pv[3], qv[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        pv[c] = p[c * N];
        qv[c] = q[c * N];
        xv[c] = x[c * N + n];
        rv[c] = r[c * N + n];
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
        x[c * N + n] = xv[c] + alpha * (double)pv[c];
        rv[c] -= alpha * (double)qv[c];
        r[c * N + n] = rv[c];
    }
    if (feed) nn::store_input(in, n, (float)(rv[0] * inv), (float)(rv[1] * inv), (float)(rv[2] * inv));
}

__global__ void k_imp_reset_next(DevCtl *ctl, int parity) {
    for (int k = 0; k < B_NB; k++) ctl->nxt[parity ^ 1][k] = 0u;
}

}  // namespace mpm

using namespace mpm;

#define CKI(call)                                                                                                      \
    do {                                                                                                               \
        cudaError_t _e = (call);                                                                                       \
        if (_e != cudaSuccess) {                                                                                       \
            fprintf(stderr, "mpm_gb300: %s failed: %s\n", #call, cudaGetErrorString(_e));                              \
            return _e == cudaErrorMemoryAllocation ? MPM_ERR_OOM : MPM_ERR_CUDA;                                       \
        }                                                                                                              \
    } while (0)

namespace mpm {
void implicit_free(mpm_ctx *c) {
    ImpState *s = c->imp;
    if (!s) return;
    void *bufs[] = {s->A, s->bcval64, s->adiag, s->b, s->x, s->r, s->p, s->Ap, s->xs, s->ndispl, s->nvel, s->naccel,
                      s->naccel_k, s->nmass, s->nvof, s->nei, s->stress_k, s->geup, s->part, s->scal,
                      s->z, s->bs, s->xstar, s->ev, s->gp, s->gq, s->gqq, s->gbeta};
    for (void *b : bufs)
        if (b) cudaFree(b);
    if (s->cnt) cudaFree(s->cnt);
    if (s->gqf) cudaFree(s->gqf);
    if (s->gp32) cudaFree(s->gp32);
    if (s->p32) cudaFree(s->p32);
    if (s->nf32) cudaFree(s->nf32);
    if (s->dfx) cudaFree(s->dfx);
    if (s->gq32) cudaFree(s->gq32);
    if (s->h_scal) cudaFreeHost(s->h_scal);
    for (cudaGraphExec_t g : {s->g_cg, s->g_fcg_nn, s->g_fcg_jac, s->g_gcr})
        if (g) cudaGraphExecDestroy(g);
    delete s;
    c->imp = nullptr;
}
}  // namespace mpm

namespace mpm {
// The FP64 copy of the BC values the implicit kernels read, from the host
// lists of mpm_gpu_set_bc (later entries win, as there).
mpm_status implicit_bc_changed(mpm_ctx *c) {
    ImpState *s = c->imp;
    if (!s || !s->bcval64) return MPM_OK;
    const size_t N = (size_t)c->g.nodec;
    std::vector<double> val(3 * N, 0.0);
    for (int k = 0; k < 3; k++)
        for (size_t i = 0; i < c->bc_nodes[k].size(); i++) val[k * N + c->bc_nodes[k][i]] = c->bc_vals[k][i];
    CKI(cudaStreamSynchronize(c->stream));
    CKI(cudaMemcpy(s->bcval64, val.data(), sizeof(double) * 3 * N, cudaMemcpyHostToDevice));
    return MPM_OK;
}
}  // namespace mpm

static mpm_status ensure_particle_scratch(mpm_ctx *c) {
    ImpState *s = c->imp;
    if (s->num_alloc == c->num && s->stress_k) return MPM_OK;
    if (s->stress_k) cudaFree(s->stress_k);
    if (s->geup) cudaFree(s->geup);
    s->stress_k = s->geup = nullptr;
    size_t n = (size_t)(c->num > 0 ? c->num : 1);
    CKI(cudaMalloc((void **)&s->stress_k, c->rsize * 6 * n));
    CKI(cudaMalloc((void **)&s->geup, c->rsize * 3 * n));
    s->num_alloc = c->num;
    return MPM_OK;
}

mpm_status mpm_gpu_implicit_setup(mpm_ctx *c, int nr_flag, double spec_rad) {
    if (!c) return MPM_ERR_BAD_ARG;
    if (c->nreal != 27) return MPM_ERR_UNSUPPORTED;
    {
        // the shape orders mpm_gpu_create takes: linear, quadratic, or quadratic in x and z
        const int *o = c->g.order;
        const bool ok = (o[0] == 1 && o[1] == 1 && o[2] == 1) || (o[0] == 2 && o[1] == 2 && o[2] == 2) ||
                        (o[0] == 2 && o[1] == 1 && o[2] == 2);
        if (!ok) return MPM_ERR_UNSUPPORTED;
    }
    bool isotropic = true;
    {
        std::vector<int> ip(c->nmat);
        CKI(cudaMemcpy(ip.data(), c->d_iprop, sizeof(int) * c->nmat, cudaMemcpyDeviceToHost));
        for (int m : ip) {
            if (m > 3) return MPM_ERR_UNSUPPORTED;   // no tangent for the fluid model
            isotropic = isotropic && m <= 1;
        }
    }
    implicit_free(c);
    ImpState *s = new ImpState();
    c->imp = s;
    s->isotropic = isotropic;
    s->debug = getenv("MPM_GB300_KRYLOV_TRACE") != nullptr;
    s->gcr = getenv("MPM_GB300_FCG_ONLY") == nullptr;
    if (const char *w = getenv("MPM_GB300_GCR_WINDOW")) {
        const int v = atoi(w);
        if (v == 1 || v == 2 || v == 4 || v == 8) s->gm = v;   // divides the 8 iterations of a graph launch
    }
    s->nr_flag = nr_flag ? 1 : 0;
    s->prec = c->precision;
    s->qp = imp_args(c).qp;
    // GeneralizedAlphaParaSet + NewmarkBetaParaSet (nonlinear_time_integration.cpp:10-56), second order
    double t = 1.0 + spec_rad;
    s->alpha_f = 1.0 / t;
    s->alpha_m = (2.0 - spec_rad) / t;
    t = 1.0 - s->alpha_f + s->alpha_m;
    s->gamma = t - 0.5;
    s->beta = 0.25 * t * t;
    const double g = s->gamma, b = s->beta, dt = c->dt;
    s->nb[0] = g / (b * dt);
    s->nb[1] = g / b - 1.0;
    s->nb[2] = dt / 2.0 * (g / b - 2.0);
    s->nb[3] = 1.0 / (b * dt * dt);
    s->nb[4] = 1.0 / (b * dt);
    s->nb[5] = 1.0 / (2.0 * b) - 1.0;
    const size_t N = (size_t)c->g.nodec;
    CKI(cudaMalloc((void **)&s->A, (s->prec == 64 ? sizeof(double) : sizeof(float)) * a_size((int)N, s->qp)));
    CKI(cudaMalloc((void **)&s->bcval64, sizeof(double) * 3 * N));
    {
        const mpm_status q = implicit_bc_changed(c);
        if (q != MPM_OK) return q;
    }
    double **vec3[] = {&s->adiag, &s->b,    &s->x,       &s->r, &s->p,  &s->Ap,    &s->xs, &s->ndispl,
                       &s->nvel,  &s->naccel, &s->naccel_k, &s->z, &s->bs, &s->xstar, &s->ev};
    for (double **v : vec3) CKI(cudaMalloc((void **)v, sizeof(double) * 3 * N));
    s->gst = (3 * N + 3) & ~(size_t)3;
    CKI(cudaMalloc((void **)&s->gp, sizeof(double) * GM * s->gst));
    CKI(cudaMalloc((void **)&s->gq, sizeof(double) * GM * s->gst));
    CKI(cudaMalloc((void **)&s->gqq, sizeof(double) * GM));
    CKI(cudaMalloc((void **)&s->gbeta, sizeof(double) * GM));
    CKI(cudaMalloc((void **)&s->gqf, sizeof(float) * GM * s->gst));
    if (s->prec == 32) {
        CKI(cudaMalloc((void **)&s->gp32, sizeof(float) * GM * s->gst));
        CKI(cudaMalloc((void **)&s->gq32, sizeof(float) * GM * s->gst));
        CKI(cudaMalloc((void **)&s->p32, sizeof(float) * 3 * N));
        CKI(cudaMalloc((void **)&s->nf32, sizeof(float) * 10 * N));
        if (!getenv("MPM_GB300_TRUE_RESIDUAL_FP64")) CKI(cudaMalloc((void **)&s->dfx, sizeof(float) * 2 * 3 * N));
    }
    CKI(cudaMalloc((void **)&s->cnt, sizeof(unsigned) * 8));
    CKI(cudaMemset(s->cnt, 0, sizeof(unsigned) * 8));
    CKI(cudaMalloc((void **)&s->nmass, sizeof(double) * N));
    CKI(cudaMalloc((void **)&s->nvof, sizeof(double) * N));
    CKI(cudaMalloc((void **)&s->nei, sizeof(double) * N));
    s->nblk = (int)((N + 255) / 256);
    int pblk = (int)((c->num + 127) / 128);
    int nparts = 2 * (s->nblk > pblk ? s->nblk : pblk) + 2 * ((3 * (int)N + 255) / 256) + (GM + 2) * s->nblk + (int)((N + MV_NODES - 1) / MV_NODES) + 64;
    CKI(cudaMalloc((void **)&s->part, sizeof(double) * (size_t)nparts));
    CKI(cudaMalloc((void **)&s->scal, sizeof(double) * S_NSCAL));
    CKI(cudaMallocHost((void **)&s->h_scal, sizeof(double) * S_NSCAL));
    CKI(cudaMemset(s->ndispl, 0, sizeof(double) * 3 * N));
    CKI(cudaMemset(s->x, 0, sizeof(double) * 3 * N));
    CKI(cudaMemset(s->scal, 0, sizeof(double) * S_NSCAL));
    return ensure_particle_scratch(c);
}

static int nb_nodes(mpm_ctx *c) { return (c->g.nodec + 255) / 256; }

// y = A x on the context's stream (k_imp_matvec for the context's matrix
// precision and stencil); hi: FP64 arithmetic whatever the storage (the
// true residual and the Newton check of the FP32 operator).
static void launch_matvec(mpm_ctx *c, const ImpArgs &a, int nb, const double *x, double *y,
                          double *part = nullptr, bool hi = false) {
    ImpState *s = c->imp;
    const int *o = c->g.order;
    auto go = [&](auto ta, auto tc) {
        using TA = decltype(ta);
        using TC = decltype(tc);
        const TA *A = (const TA *)s->A;
        if (o[0] == 1 && o[1] == 1 && o[2] == 1)
            k_imp_matvec<TA, TC, 1, 1, 1><<<nb, 256, 0, c->stream>>>(a, A, x, y, part);
        else if (o[1] == 2)
            k_imp_matvec<TA, TC, 2, 2, 2><<<nb, 256, 0, c->stream>>>(a, A, x, y, part);
        else
            k_imp_matvec<TA, TC, 2, 1, 2><<<nb, 256, 0, c->stream>>>(a, A, x, y, part);
    };
    if (s->prec == 64) {
        go(double(), double());
    } else if (hi && !part && s->dfx) {
        // FP32 operator, true residual / Newton check: double-float arithmetic
        const int n3 = 3 * c->g.nodec;
        k_split_df<<<(n3 + 255) / 256, 256, 0, c->stream>>>(x, s->dfx, s->dfx + n3, n3);
        const int nbs = (c->g.nodec + MV_NODES - 1) / MV_NODES;
        const float *A = (const float *)s->A;
        if (o[0] == 1 && o[1] == 1 && o[2] == 1)
            k_imp_matvec_df<1, 1, 1><<<nbs, MV_NODES * MV_G, 0, c->stream>>>(a, A, s->dfx, s->dfx + n3, y);
        else if (o[1] == 2)
            k_imp_matvec_df<2, 2, 2><<<nbs, MV_NODES * MV_G, 0, c->stream>>>(a, A, s->dfx, s->dfx + n3, y);
        else
            k_imp_matvec_df<2, 1, 2><<<nbs, MV_NODES * MV_G, 0, c->stream>>>(a, A, s->dfx, s->dfx + n3, y);
    } else if (hi) {
        go(float(), double());
    } else {
        go(float(), float());
    }
}

// Whether a CG product forms p.Ap itself.  MV_G threads per control point give it
// eight times as many CTAs as a pass over vectors has, and on a large grid their
// partials cost more than a pass of its own over p and Ap: per product, with its own dot
// against a separate one, 18.8 against 17.1 us (FP32) and 38.1 against 35.3 (FP64) at
// 46,305 points, 86 against 59 to 63 (FP32) at 274,625; but 10.9 against 12.6 at 1,690 and
// 18.8 against 19.6 at 24,000 (B-spline stencil).
// (One thread per point: 19.6 us FP32 at 1,690 points, 22.1 at 46,305, 65 at
// 274,625; FP64 50.8 and 153 where the split takes 35.3 and 143.)
static bool mv_dot(const mpm_ctx *c) { return c->g.nodec <= 32768; }

template <typename TA, typename TC, typename TV, typename TY>
static void launch_split(mpm_ctx *c, const ImpArgs &a, const TV *x, TY *y, const double *xd, double *part,
                         unsigned *cnt, double *scal, int slot, int num, const double *done) {
    const int *o = c->g.order;
    const unsigned nb = (unsigned)((c->g.nodec + MV_NODES - 1) / MV_NODES);
    const TA *A = (const TA *)c->imp->A;
    auto go = [&](auto k) {
        launch(c->pdl != 0, k, nb, MV_NODES * MV_G, 0, c->stream, a, A, x, y, xd, part, cnt, scal, slot, num, done);
    };
    if (o[0] == 1 && o[1] == 1 && o[2] == 1) go(k_imp_matvec_split<TA, TC, 1, 1, 1, TV, TY>);
    else if (o[1] == 2) go(k_imp_matvec_split<TA, TC, 2, 2, 2, TV, TY>);
    else go(k_imp_matvec_split<TA, TC, 2, 1, 2, TV, TY>);
}

// y = A x with FP32 vectors and FP32 arithmetic (FP32 operator only): the
// matvec of the flexible GCR directions.  Without a dot product the split form is
// the faster one on every grid (52.6 against 57.0 us at 274,625 points).
static void launch_matvec_f32(mpm_ctx *c, const ImpArgs &a, const float *x, float *y) {
    launch_split<float, float>(c, a, x, y, nullptr, nullptr, nullptr, nullptr, 0, -1, nullptr);
}

// Ap = A p and p.Ap (into S_PAP) of one CG iteration; the FP32 operator
// multiplies the FP32 copy of p that k_cg_dir left
static void launch_matvec_cg(mpm_ctx *c, const ImpArgs &a, int nb, int cur, const double *done) {
    ImpState *s = c->imp;
    const int *o = c->g.order;
    const bool dot = mv_dot(c);
    double *part = dot ? s->part : nullptr;
    if (s->prec == 64)
        launch_split<double, double>(c, a, (const double *)s->p, s->Ap, s->p, part, s->cnt + 3, s->scal, S_PAP, cur, done);
    else
        launch_split<float, float>(c, a, (const float *)s->p32, s->Ap, s->p, part, s->cnt + 3, s->scal, S_PAP, cur, done);
    if (!dot) {
        const int m = 3 * c->g.nodec;
        launch(c->pdl != 0, k_cg_dot, (m + 1023) / 1024, 256, 0, c->stream, (const double *)s->p, (const double *)s->Ap, m,
               s->part, s->cnt + 3, s->scal, cur, done);
        c->launches++;
    }
}

// FP32 copies of nodal fields, so that the FP32 particles' gathers convert each
// node's value once instead of once per particle and node (a conversion takes a
// slot of the FP64 pipe)
__global__ void k_to_f32(const double *__restrict__ x, float *__restrict__ y, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = (float)x[i];
}
// `n` values of a nodal field in the particle precision: the field itself, or its
// copy at `at` of the FP32 copies
template <typename R>
static const R *nodal_of(mpm_ctx *c, const double *x, size_t at, size_t n) {
    if constexpr (sizeof(R) == 8) {
        return x;
    } else {
        float *y = c->imp->nf32 + at;
        k_to_f32<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(x, y, (int)n);
        c->launches++;
        return y;
    }
}

// AssembleSystem: k_imp_assemble (per particle), k_imp_rhs_diag, k_imp_scale
template <typename R>
static void launch_assemble(mpm_ctx *c, const ImpArgs &a) {
    ImpState *s = c->imp;
    const PView<R> P = pview<R>(c);
    R *A = (R *)s->A, *sk = (R *)s->stress_k;
    const R *nd = nodal_of<R>(c, s->ndispl, 0, 3 * (size_t)c->g.nodec);
    const int pb = (int)((c->num + 127) / 128);
    const int *o = c->g.order;
    bool cells = false;
    if constexpr (sizeof(R) == 4) {
        cells = s->isotropic && c->cell_scatter;
        auto go = [&](auto shape, auto k) {
            using C = decltype(shape);
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
            k<<<c->g.nbricks * (BRC / C::CELLS), C::THREADS, C::SMEM, c->stream>>>(
                a, P, nd, sk, A, s->b, c->d_cstart, c->d_blist, c->d_nblist, c->g.nbrick[0], c->g.nbrick[1]);
        };
        if (cells && o[0] == 1) go(AsmShape<1, 1, 1>(), k_imp_assemble_cells<1, 1, 1>);
        else if (cells && o[1] == 2) go(AsmShape<2, 2, 2>(), k_imp_assemble_cells<2, 2, 2>);
        else if (cells) go(AsmShape<2, 1, 2>(), k_imp_assemble_cells<2, 1, 2>);
    }
    if (cells) {
    } else if (o[0] == 1 && o[1] == 1 && o[2] == 1)
        k_imp_assemble<R, 1, 1, 1><<<pb, 128, 0, c->stream>>>(a, P, nd, sk, A, s->b);
    else if (o[1] == 2)
        k_imp_assemble<R, 2, 2, 2><<<pb, 128, 0, c->stream>>>(a, P, nd, sk, A, s->b);
    else
        k_imp_assemble<R, 2, 1, 2><<<pb, 128, 0, c->stream>>>(a, P, nd, sk, A, s->b);
    k_imp_rhs_diag<R><<<nb_nodes(c), 256, 0, c->stream>>>(a, A, s->nmass, s->naccel_k, s->naccel, s->b, s->adiag);
    k_imp_scale<R><<<nb_nodes(c), 256, 0, c->stream>>>(a, A, s->adiag);
}

// Node2Particle's particle pass (k_imp_g2p) and the shift (k_imp_shift)
template <typename R>
static void launch_g2p(mpm_ctx *c, const ImpArgs &a, int parity, int pb) {
    ImpState *s = c->imp;
    const PView<R> P = pview<R>(c);
    R *geup = (R *)s->geup;
    const size_t N = (size_t)c->g.nodec;
    const R *nd = nodal_of<R>(c, s->ndispl, 0, 3 * N), *nv = nodal_of<R>(c, s->nvel, 3 * N, 3 * N),
            *na = nodal_of<R>(c, s->naccel, 6 * N, 3 * N), *ne = nodal_of<R>(c, s->nei, 9 * N, N);
    const int *o = c->g.order;
    if (o[0] == 1 && o[1] == 1 && o[2] == 1)
        k_imp_g2p<R, 1, 1, 1><<<pb, 128, 0, c->stream>>>(a, P, nd, nv, na, ne, geup, s->part,
                                                          c->d_ctl, parity);
    else if (o[1] == 2)
        k_imp_g2p<R, 2, 2, 2><<<pb, 128, 0, c->stream>>>(a, P, nd, nv, na, ne, geup, s->part,
                                                          c->d_ctl, parity);
    else
        k_imp_g2p<R, 2, 1, 2><<<pb, 128, 0, c->stream>>>(a, P, nd, nv, na, ne, geup, s->part,
                                                          c->d_ctl, parity);
    k_finish<<<1, 256, 0, c->stream>>>(s->part, pb, s->scal, S_GD);
    k_imp_shift<R><<<pb, 128, 0, c->stream>>>(a, P, geup, s->scal);
}

// stress_k <- the particles' stress (InitializeNRStress)
static mpm_status copy_stress_k(mpm_ctx *c) {
    ImpState *s = c->imp;
    const size_t rs = c->rsize, n = (size_t)c->num;
    const char *f = (const char *)c->pbuf[c->cur];
    for (int k = 0; k < 6; k++)
        CKI(cudaMemcpyAsync((char *)s->stress_k + k * n * rs, f + (15 + k) * c->pstride * rs, rs * n,
                            cudaMemcpyDeviceToDevice, c->stream));
    return MPM_OK;
}

// P2G of the implicit solid: AccelP2G mode of the scatter + k_imp_grid
static mpm_status imp_p2g(mpm_ctx *c, double facl) {
    ImpState *s = c->imp;
    c->facl = facl;
    const size_t N = (size_t)c->g.nodec;
    if (c->steps_since_sort >= c->resort_period) {
        mpm_status st = sort_particles(c);
        if (st != MPM_OK) return st;
    }
    CKI(cudaMemsetAsync(c->d_acc, 0, sizeof(unsigned long long) * NACC * N, c->stream));
    c->write_nodal_dl = false;
    mpm_status st = run_p2g(c, facl);
    if (st != MPM_OK) return st;
    ImpArgs a = imp_args(c);
    k_imp_grid<<<nb_nodes(c), 256, 0, c->stream>>>(a, c->d_acc, c->d_ctl->p2g_inv, s->nmass, s->nvof, s->nvel,
                                                   s->naccel);
    c->launches++;
    return check_launch(c);
}

// one linear solve of the assembled, scaled system; s->x holds the initial
// guess (physical) and receives the physical solution.  Returns iterations.
static constexpr int KCHECK = 8;   // Krylov iterations between residual checks (and per graph)
// Within this factor of the tolerance (squared norms, 100x in the norm) the
// flexible GCR leaves the 8-iteration graphs and checks after every iteration, so
// that a solve stops at the iteration that reaches the tolerance instead of at
// the end of the next block of 8.  (CG stops itself on the device.)
static constexpr double FINE_FACTOR = 1.0e4;

static bool graphs_on(mpm_ctx *c) { return c->use_graph && c->stream != nullptr && !c->timer.on && !c->imp->no_graph; }

template <typename F>
static mpm_status capture_iters(mpm_ctx *c, cudaGraphExec_t *exec, F body) {
    CKI(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
    body();
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(c->stream, &g);
    if (e != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        cudaGetLastError();
        return MPM_ERR_CUDA;
    }
    e = cudaGraphInstantiate(exec, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
        *exec = nullptr;
        cudaGetLastError();
        return MPM_ERR_CUDA;
    }
    return MPM_OK;
}

// one CG iteration on the scaled system; `it` fixes the residual-norm slot parity
static void cg_iteration(mpm_ctx *c, const ImpArgs &a, int nb, int it, int stop) {
    ImpState *s = c->imp;
    const int cur = (it & 1) ? S_RR1 : S_RR0;
    timer_begin(c, K_MATVEC);
    launch_matvec_cg(c, a, nb, cur, stop ? s->scal + S_DONE : nullptr);
    timer_end(c, K_MATVEC);
    timer_begin(c, K_KRYLOV);
    launch(c->pdl != 0, k_cg_update, nb, 256, 0, c->stream, a, s->scal, cur, s->xs, s->r, (const double *)s->p,
           (const double *)s->Ap, s->part, s->cnt + 4, stop);
    launch(c->pdl != 0, k_cg_dir, nb, 256, 0, c->stream, a, (const double *)s->scal, (const double *)s->r, s->p, s->p32, stop);
    timer_end(c, K_KRYLOV);
    c->launches += 3;
}

static mpm_status imp_cg(mpm_ctx *c, double eps, int kmax, int *iters) {
    ImpState *s = c->imp;
    ImpArgs a = imp_args(c);
    const int nb = nb_nodes(c), nb3 = (3 * c->g.nodec + 255) / 256;
    k_cg_scale_in<<<nb, 256, 0, c->stream>>>(a, s->x, s->b, s->adiag, s->xs, s->r);
    if (s->prec == 32)   // the scaled RHS, for the true residual of the FP32 operator
        CKI(cudaMemcpyAsync(s->bs, s->r, sizeof(double) * 3 * c->g.nodec, cudaMemcpyDeviceToDevice, c->stream));
    launch_matvec(c, a, nb, s->xs, s->Ap, nullptr, true);
    k_cg_init<<<nb, 256, 0, c->stream>>>(a, s->Ap, s->r, s->p, s->part);
    k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_RR0);
    c->launches += 4;
    CKI(cudaMemcpyAsync(s->h_scal, s->scal, sizeof(double) * S_NSCAL, cudaMemcpyDeviceToHost, c->stream));
    CKI(cudaStreamSynchronize(c->stream));
    const double rr0 = s->h_scal[S_RR0];
    int it = 0;
    bool done = !(rr0 > 1.0e-300);
    // the device ends the solve at the iteration that reaches the tolerance; what
    // is left of the launched block then does nothing.  (Checked by the host, the
    // last decades of the residual went one iteration and one wait at a time.)
    if (!done) {
        k_cg_start<<<nb3, 256, 0, c->stream>>>(a, s->scal, eps * rr0, 0, s->r, s->p, s->p32);
        c->launches++;
    }
    while (!done && it < kmax) {
        bool ran = false;
        if (graphs_on(c) && it % KCHECK == 0 && it + KCHECK <= kmax) {
            const int64_t l0 = c->launches;
            if (!s->g_cg && capture_iters(c, &s->g_cg, [&] {
                    for (int k = 0; k < KCHECK; k++) cg_iteration(c, a, nb, k, 1);
                    s->cg_launches = c->launches - l0;
                }) != MPM_OK)
                s->no_graph = true;
            if (s->g_cg) {
                CKI(cudaGraphLaunch(s->g_cg, c->stream));
                if (c->launches == l0) c->launches += s->cg_launches;   // the capture counted the first block
                ran = true;
            }
        }
        if (!ran) {
            const int end = std::min(kmax, it + KCHECK - it % KCHECK);
            for (int k = it; k < end; k++) cg_iteration(c, a, nb, k, 1);
        }
        CKI(cudaMemcpyAsync(s->h_scal, s->scal, sizeof(double) * S_NSCAL, cudaMemcpyDeviceToHost, c->stream));
        CKI(cudaStreamSynchronize(c->stream));
        it = (int)s->h_scal[S_ITER];
        const int cur = (it & 1) ? S_RR1 : S_RR0;
        const double rr = s->h_scal[cur];
        if (rr != rr) {
            *iters = it;
            return MPM_ERR_NONFINITE;
        }
        if (s->debug) fprintf(stderr, "mpm_gb300 cg: it %d |r|/|r0| %.3e\n", it, sqrt(rr / rr0));
        if (rr < eps * rr0 && s->prec == 32) {
            // FP32 operator: the recursive residual carries the rounding of
            // the FP32 matvecs, so convergence is judged on the true
            // residual bs - A x (FP64 arithmetic); if it is not below the
            // tolerance, CG restarts from it (r, and p = r).  Keeping the
            // old direction instead diverged: at this point the recursive
            // residual, and with it p, has fallen far below the true
            // residual, so alpha = r.r / p.Ap overshoots.
            launch_matvec(c, a, nb, s->xs, s->z, nullptr, true);
            k_true_residual<<<nb, 256, 0, c->stream>>>(a, s->bs, s->z, s->r, s->part);
            k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, cur);
            k_cg_start<<<nb3, 256, 0, c->stream>>>(a, s->scal, eps * rr0, it, s->r, s->p, s->p32);
            c->launches += 4;
            CKI(cudaMemcpyAsync(s->h_scal, s->scal, sizeof(double) * 2, cudaMemcpyDeviceToHost, c->stream));
            CKI(cudaStreamSynchronize(c->stream));
            const double rrt = s->h_scal[cur];
            if (s->debug) fprintf(stderr, "mpm_gb300 cg: it %d true |r|/|r0| %.3e\n", it, sqrt(rrt / rr0));
            if (rrt < eps * rr0) done = true;
            s->last_rel = sqrt(rrt / rr0);
        } else {
            if (rr < eps * rr0) done = true;
            s->last_rel = sqrt(rr / rr0);
        }
    }
    k_cg_scale_out<<<nb3, 256, 0, c->stream>>>(a, s->xs, s->adiag, s->x);
    c->launches++;
    *iters = it;
    if (!done) return MPM_ERR_KRYLOV_MAXIT;
    return check_launch(c);
}

// One flexible GCR iteration on the scaled system: z = M(r) into direction
// slot `sl`, q = A z, orthogonalised against the `u` previous images, then
// x += alpha z, r -= alpha q with alpha = q.r / q.q.
// fed: the network's input already holds r; feed: leave the new r there.
static mpm_status gcr_iter(mpm_ctx *c, const ImpArgs &a, int nb, int u, int sl, bool fed = false, bool feed = false) {
    ImpState *s = c->imp;
    const size_t st = s->gst;
    const int m = 3 * c->g.nodec, nq = (m + 1023) / 1024;
    const bool pdl = c->pdl != 0 && !c->timer.on;
    auto dots = [&](auto k, auto *Q, const float *Qf) {
        launch(pdl, k, nq, 256, 0, c->stream, Q, Qf, st, m, sl, u, s->gm, s->part, s->cnt, (const double *)s->gqq,
               s->gbeta);
    };
    auto axpy = [&](auto k, auto *P, auto *Q, float *Qf, int rr) {
        launch(pdl, k, nq, 256, 0, c->stream, P, Q, Qf, st, m, sl, u, s->gm, (const double *)s->gbeta,
               (const double *)s->r, s->gqq, s->part, s->cnt + 1, s->scal, rr);
    };
    if (s->gp32 && mpm_nn_fp32_output(s->net)) {
        // FP32 operator: directions and images in FP32 (the FP32 matvec computes
        // them in FP32 anyway; x, r and the true residual stay FP64)
        float *p = s->gp32 + (size_t)sl * st, *q = s->gq32 + (size_t)sl * st;
        timer_begin(c, K_PRECOND);
        mpm_status e = mpm_nn_apply_precond_f32(s->net, c->stream, s->r, s->scal + S_RRC, s->adiag, a.bcflag, a.mtol,
                                                p, fed, pdl);
        timer_end(c, K_PRECOND);
        if (e != MPM_OK) return e;
        timer_begin(c, K_MATVEC);
        launch_matvec_f32(c, a, p, q);
        timer_end(c, K_MATVEC);
        timer_begin(c, K_KRYLOV);
        const float *Q = s->gq32;
        if (s->gm <= 4) {
            if (u > 0) dots(k_gcr_dots<float, 4>, Q, Q);
            axpy(k_gcr_axpy<float, 4>, s->gp32, s->gq32, nullptr, 1);
        } else {
            if (u > 0) dots(k_gcr_dots<float, GM>, Q, Q);
            axpy(k_gcr_axpy<float, GM>, s->gp32, s->gq32, nullptr, 1);
        }
        launch(pdl, k_gcr_update_feed, nb, 256, 0, c->stream, (const double *)s->scal, s->xs, s->r,
               (const float *)s->gp32, (const float *)s->gq32, st, c->g.nodec, sl, feed ? 1 : 0,
               mpm_nn_input(s->net));
        timer_end(c, K_KRYLOV);
        c->launches += 7 + (fed ? 0 : 1) + 3 + (u > 0 ? 1 : 0);
        return MPM_OK;
    }
    timer_begin(c, K_PRECOND);
    mpm_status e = mpm_nn_apply_precond(s->net, c->stream, s->r, s->scal + S_RRC, s->adiag, a.bcflag, a.mtol,
                                        s->gp + (size_t)sl * st);
    timer_end(c, K_PRECOND);
    if (e != MPM_OK) return e;
    timer_begin(c, K_MATVEC);
    launch_matvec(c, a, nb, s->gp + (size_t)sl * st, s->gq + (size_t)sl * st);
    timer_end(c, K_MATVEC);
    timer_begin(c, K_KRYLOV);
    const double *Q = s->gq;
    if (s->gm <= 4) {
        if (u > 0) dots(k_gcr_dots<double, 4>, Q, s->gqf);
        axpy(k_gcr_axpy<double, 4>, s->gp, s->gq, s->gqf, 0);
    } else {
        if (u > 0) dots(k_gcr_dots<double, GM>, Q, s->gqf);
        axpy(k_gcr_axpy<double, GM>, s->gp, s->gq, s->gqf, 0);
    }
    launch(pdl, k_gcr_update<double>, nq, 256, 0, c->stream, s->scal, s->xs, s->r, (const double *)s->gp,
           (const double *)s->gq, st, m, sl, s->part, s->cnt + 2);
    timer_end(c, K_KRYLOV);
    c->launches += 9 + 3 + (u > 0 ? 1 : 0);
    return MPM_OK;
}

// One solve of the assembled, scaled system by flexible CG with the learned
// preconditioner z = net(r) (Notay's FCG(1): p = z - (z.q'/p'.q') p',
// alpha = p.r / p.q).  The residual is checked every 8 iterations; when two
// checks in a row find no new minimum the solve continues with the Jacobi
// preconditioner (z = r in the scaled system).  Convergence is accepted only
// on the true residual bs - A x, recomputed in FP64.
static mpm_status imp_fcg(mpm_ctx *c, double eps, int kmax, int *iters) {
    ImpState *s = c->imp;
    ImpArgs a = imp_args(c);
    const int nb = nb_nodes(c);
    const size_t N = (size_t)c->g.nodec;
    k_cg_scale_in<<<nb, 256, 0, c->stream>>>(a, s->x, s->b, s->adiag, s->xs, s->r);
    CKI(cudaMemcpyAsync(s->bs, s->r, sizeof(double) * 3 * N, cudaMemcpyDeviceToDevice, c->stream));
    launch_matvec(c, a, nb, s->xs, s->Ap, nullptr, true);
    k_true_residual<<<nb, 256, 0, c->stream>>>(a, s->bs, s->Ap, s->r, s->part);
    k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_RR0);
    k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_RRC);
    c->launches += 5;
    CKI(cudaMemcpyAsync(s->h_scal, s->scal, sizeof(double) * S_NSCAL, cudaMemcpyDeviceToHost, c->stream));
    CKI(cudaStreamSynchronize(c->stream));
    const double rr0 = s->h_scal[S_RR0];
    int it = 0;
    bool done = !(rr0 > 1.0e-300);
    bool use_nn = s->net != nullptr;
    if (use_nn) {
        k_phi<<<nb, 256, 0, c->stream>>>(a, s->nmass, s->adiag, s->ev);
        mpm_status st = mpm_nn_set_feature(s->net, c->stream, s->ev);
        if (st != MPM_OK) return st;
    }
    int restart = 1;
    double rr_window = rr0;   // smallest residual norm seen at a check
    int stall = 0;
    const int check = KCHECK;
    // one FCG iteration: z = M(r), p = z - (z.q'/p'.q') p', q = A p, x, r update
    auto iteration = [&](bool nn, int rs) -> mpm_status {
        if (nn) {
            timer_begin(c, K_PRECOND);
            mpm_status st = mpm_nn_apply_precond(s->net, c->stream, s->r, s->scal + S_RRC, s->adiag, a.bcflag, a.mtol,
                                                 s->z);
            timer_end(c, K_PRECOND);
            if (st != MPM_OK) return st;
            c->launches += 9;
        } else {
            CKI(cudaMemcpyAsync(s->z, s->r, sizeof(double) * 3 * N, cudaMemcpyDeviceToDevice, c->stream));
        }
        if (!rs) {
            k_dot3<<<nb, 256, 0, c->stream>>>(a, s->z, s->Ap, s->part);
            k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_ZQ);
            c->launches += 2;
        }
        timer_begin(c, K_KRYLOV);
        k_fcg_dir<<<nb, 256, 0, c->stream>>>(a, s->scal, rs, s->z, s->r, s->p, s->part);
        k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_PR);
        timer_end(c, K_KRYLOV);
        timer_begin(c, K_MATVEC);
        launch_matvec(c, a, nb, s->p, s->Ap, s->part);
        timer_end(c, K_MATVEC);
        timer_begin(c, K_KRYLOV);
        k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_PAP);
        k_fcg_update<<<nb, 256, 0, c->stream>>>(a, s->scal, s->xs, s->r, s->p, s->Ap, s->part);
        k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_RRC);
        timer_end(c, K_KRYLOV);
        c->launches += 6;
        return MPM_OK;
    };
    if (s->g_fcg_nn && s->g_net != s->net) {
        cudaGraphExecDestroy(s->g_fcg_nn);
        s->g_fcg_nn = nullptr;
    }
    if (s->g_gcr && s->g_net != s->net) {
        cudaGraphExecDestroy(s->g_gcr);
        s->g_gcr = nullptr;
    }
    // Phase 1: flexible GCR(GM) with the network as right preconditioner.  It
    // minimises the residual over the kept directions, so it needs no
    // symmetry of the (learned, non-symmetric) preconditioner.  It runs while
    // every window of `check` iterations at least halves the residual norm.
    if (use_nn && s->gcr) {
        int used = 0, slot = 0;
        double rr_win = rr0;
        bool fine = false;   // close to the tolerance: one iteration at a time, checked after each
        bool fed = false;    // the network's input holds the current residual
        while (!done && use_nn && it < kmax) {
            if (graphs_on(c) && !fine && used == s->gm && slot == 0 && it % check == 0 && it + check <= kmax) {
                const int64_t l0 = c->launches;
                if (!s->g_gcr && capture_iters(c, &s->g_gcr, [&] {
                        for (int k = 0; k < check; k++)
                            gcr_iter(c, a, nb, s->gm, k % s->gm, k > 0, k + 1 < check);
                        s->gcr_launches = c->launches - l0;
                    }) != MPM_OK)
                    s->no_graph = true;
                if (!s->g_gcr) continue;
                s->g_net = s->net;
                CKI(cudaGraphLaunch(s->g_gcr, c->stream));
                if (c->launches == l0) c->launches += s->gcr_launches;
                fed = false;
                s->nn_applications += check;
                it += check;
            } else {
                mpm_status st = gcr_iter(c, a, nb, used, slot, fed, true);
                if (st != MPM_OK) return st;
                fed = s->gp32 && mpm_nn_fp32_output(s->net);
                s->nn_applications++;
                used = used < s->gm ? used + 1 : s->gm;
                slot = (slot + 1) % s->gm;
                it++;
            }
            if (it % check == 0 || it == kmax || fine) {
                // between the checks the recursive residual tells whether the true one
                // (a double-float product) is worth forming: within a window they
                // differ by the rounding of a few FP32 products
                bool form = s->prec == 32;
                if (form && it % check != 0 && it != kmax) {
                    CKI(cudaMemcpyAsync(s->h_scal, s->scal, sizeof(double) * S_NSCAL, cudaMemcpyDeviceToHost,
                                        c->stream));
                    CKI(cudaStreamSynchronize(c->stream));
                    if (s->h_scal[S_RRC] >= 1.1 * eps * rr0) continue;
                }
                fed = false;
                if (form) {
                    // FP32 operator: the recursive residual drifts from the true one
                    // by the rounding of the FP32 matvecs, so at every check it is
                    // replaced by the true residual bs - A x (FP64 arithmetic); the
                    // kept directions and their images stay valid
                    launch_matvec(c, a, nb, s->xs, s->z, nullptr, true);
                    k_true_residual<<<nb, 256, 0, c->stream>>>(a, s->bs, s->z, s->r, s->part);
                    k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_RRC);
                    c->launches += 3;
                }
                CKI(cudaMemcpyAsync(s->h_scal, s->scal, sizeof(double) * S_NSCAL, cudaMemcpyDeviceToHost, c->stream));
                CKI(cudaStreamSynchronize(c->stream));
                double rr = s->h_scal[S_RRC];
                if (rr != rr) {
                    *iters = it;
                    return MPM_ERR_NONFINITE;
                }
                if (s->debug) fprintf(stderr, "mpm_gb300 gcr: it %d |r|/|r0| %.3e\n", it, sqrt(rr / rr0));
                if (rr < eps * rr0 && s->prec == 32) {
                    done = true;   // rr is the true residual
                } else if (rr < eps * rr0) {
                    launch_matvec(c, a, nb, s->xs, s->z, nullptr, true);
                    k_true_residual<<<nb, 256, 0, c->stream>>>(a, s->bs, s->z, s->r, s->part);
                    k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_RRC);
                    c->launches += 3;
                    CKI(cudaMemcpyAsync(s->h_scal, s->scal, sizeof(double) * S_NSCAL, cudaMemcpyDeviceToHost,
                                        c->stream));
                    CKI(cudaStreamSynchronize(c->stream));
                    rr = s->h_scal[S_RRC];
                    if (rr < eps * rr0) done = true;
                    used = 0;   // the residual was replaced: the kept directions no longer apply
                    slot = 0;
                }
                if (!done && rr < FINE_FACTOR * eps * rr0) fine = true;
                if (it % check == 0 || it == kmax) {   // the window test, at window ends only
                    if (!done && !(rr < 0.25 * rr_win)) {
                        use_nn = false;   // less than a halving of |r| per window: Jacobi does better
                        s->fallbacks++;
                    }
                    rr_win = rr;
                }
                s->last_rel = sqrt(rr / rr0);
            }
        }
        restart = 1;
    }
    while (!done && it < kmax) {
        cudaGraphExec_t *gx = use_nn ? &s->g_fcg_nn : &s->g_fcg_jac;
        if (s->debug && use_nn) {
            // diagnostics: |z| / |r| and cos(z, r) of the preconditioned residual
            mpm_nn_apply_precond(s->net, c->stream, s->r, s->scal + S_RRC, s->adiag, a.bcflag, a.mtol, s->z);
            k_dot3<<<nb, 256, 0, c->stream>>>(a, s->z, s->z, s->part);
            k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_DZZ);
            k_dot3<<<nb, 256, 0, c->stream>>>(a, s->z, s->r, s->part);
            k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_DZR);
            CKI(cudaMemcpyAsync(s->h_scal, s->scal, sizeof(double) * S_NSCAL, cudaMemcpyDeviceToHost, c->stream));
            CKI(cudaStreamSynchronize(c->stream));
            const double zz = s->h_scal[S_DZZ], zr = s->h_scal[S_DZR], rr = s->h_scal[S_RRC];
            fprintf(stderr, "mpm_gb300 fcg: it %d |z|/|r| %.3e cos(z,r) %.3e\n", it, sqrt(zz / rr),
                    zr / sqrt(zz * rr + 1e-300));
        }
        if (graphs_on(c) && !restart && it % check == 0 && it + check <= kmax) {
            const int64_t l0 = c->launches;
            if (!*gx && capture_iters(c, gx, [&] {
                    for (int k = 0; k < check; k++) iteration(use_nn, 0);
                }) != MPM_OK)
                s->no_graph = true;
            if (*gx) {
                if (use_nn) s->g_net = s->net;
                CKI(cudaGraphLaunch(*gx, c->stream));
                if (c->launches == l0) c->launches += (use_nn ? 17 : 8) * check;
                if (use_nn) s->nn_applications += check;
                it += check;
            } else {
                continue;
            }
        } else {
            mpm_status st = iteration(use_nn, restart);
            if (st != MPM_OK) return st;
            if (use_nn) s->nn_applications++;
            restart = 0;
            it++;
        }
        if (it % check == 0 || it == kmax) {
            CKI(cudaMemcpyAsync(s->h_scal, s->scal, sizeof(double) * S_NSCAL, cudaMemcpyDeviceToHost, c->stream));
            CKI(cudaStreamSynchronize(c->stream));
            double rr = s->h_scal[S_RRC];
            if (rr != rr) {
                *iters = it;
                return MPM_ERR_NONFINITE;
            }
            if (s->debug)
                fprintf(stderr, "mpm_gb300 fcg: it %d |r|/|r0| %.3e (%s)\n", it, sqrt(rr / rr0),
                        use_nn ? "network" : "jacobi");
            if (rr < eps * rr0) {
                // confirm on the true residual
                launch_matvec(c, a, nb, s->xs, s->z, nullptr, true);
                k_true_residual<<<nb, 256, 0, c->stream>>>(a, s->bs, s->z, s->r, s->part);
                k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_RRC);
                c->launches += 3;
                CKI(cudaMemcpyAsync(s->h_scal, s->scal, sizeof(double) * S_NSCAL, cudaMemcpyDeviceToHost, c->stream));
                CKI(cudaStreamSynchronize(c->stream));
                rr = s->h_scal[S_RRC];
                if (rr < eps * rr0) done = true;
                else restart = 1;
            }
            // the residual norm of a preconditioned solve need not fall at every
            // check: fall back only after two windows without a new minimum
            if (rr < rr_window) {
                rr_window = rr;
                stall = 0;
            } else {
                stall++;
            }
            if (!done && use_nn && stall >= 2) {
                use_nn = false;   // the network stopped reducing the residual
                restart = 1;
                s->fallbacks++;
            }
            s->last_rel = sqrt(rr / rr0);
        }
    }
    k_cg_scale_out<<<(3 * c->g.nodec + 255) / 256, 256, 0, c->stream>>>(a, s->xs, s->adiag, s->x);
    c->launches++;
    *iters = it;
    if (!done) return MPM_ERR_KRYLOV_MAXIT;
    return check_launch(c);
}

static mpm_status imp_assemble(mpm_ctx *c) {
    ImpState *s = c->imp;
    ImpArgs a = imp_args(c);
    const size_t N = (size_t)c->g.nodec;
    CKI(cudaMemsetAsync(s->A, 0, (s->prec == 64 ? sizeof(double) : sizeof(float)) * a_size((int)N, s->qp),
                        c->stream));
    CKI(cudaMemsetAsync(s->b, 0, sizeof(double) * 3 * N, c->stream));
    timer_begin(c, K_ASSEMBLE);
    if (s->prec == 64) launch_assemble<double>(c, a);
    else launch_assemble<float>(c, a);
    timer_end(c, K_ASSEMBLE);
    c->launches += 3;
    return check_launch(c);
}

// CheckNRConvergence's two residual measures of the last linear solve
static mpm_status imp_residuals(mpm_ctx *c, double *ref, double *absr) {
    ImpState *s = c->imp;
    ImpArgs a = imp_args(c);
    const int nb = nb_nodes(c);
    k_imp_prepare_residual<<<nb, 256, 0, c->stream>>>(a, s->x, s->adiag, s->b, s->xs);
    launch_matvec(c, a, nb, s->xs, s->Ap, nullptr, true);
    k_imp_residual<<<nb, 256, 0, c->stream>>>(a, s->Ap, s->adiag, s->b, s->part);
    k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_RES);
    k_finish<<<1, 256, 0, c->stream>>>(s->part + nb, nb, s->scal, S_IDOF);
    c->launches += 5;
    CKI(cudaMemcpyAsync(s->h_scal, s->scal, sizeof(double) * S_NSCAL, cudaMemcpyDeviceToHost, c->stream));
    CKI(cudaStreamSynchronize(c->stream));
    const double rtr = s->h_scal[S_RES], idof = s->h_scal[S_IDOF];
    *ref = sqrt(rtr);
    *absr = idof <= 1.0e-30 ? 0.0 : sqrt(rtr / idof);
    return MPM_OK;
}

__global__ void k_add(double *y, const double *x, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] += x[i];
}

// SolidMaterialPoint::SolveSolid (solve_solid_implicit.cpp:65-103)
static mpm_status imp_newton(mpm_ctx *c, double eps, int kmax, int *krylov, int *newton) {
    ImpState *s = c->imp;
    ImpArgs a = imp_args(c);
    const size_t N = (size_t)c->g.nodec;
    if (copy_stress_k(c) != MPM_OK) return MPM_ERR_CUDA;
    CKI(cudaMemsetAsync(s->ndispl, 0, sizeof(double) * 3 * N, c->stream));
    CKI(cudaMemsetAsync(s->x, 0, sizeof(double) * 3 * N, c->stream));
    const int iter_max = s->nr_flag ? 1000 : 0;
    double r0r = 0.0;
    int ktot = 0, it;
    mpm_status st = MPM_OK;
    for (it = 0; it <= iter_max; it++) {
        k_imp_predict<<<nb_nodes(c), 256, 0, c->stream>>>(a, s->ndispl, s->nvel, s->naccel, s->naccel_k, nullptr, 1);
        c->launches++;
        st = imp_assemble(c);
        if (st != MPM_OK) return st;
        int k = 0;
        st = s->net ? imp_fcg(c, eps, kmax, &k) : imp_cg(c, eps, kmax, &k);
        ktot += k;
        if (st != MPM_OK) break;
        k_add<<<(3 * c->g.nodec + 255) / 256, 256, 0, c->stream>>>(s->ndispl, s->x, 3 * c->g.nodec);
        c->launches++;
        if (s->nr_flag) {
            double rkr, ra;
            st = imp_residuals(c, &rkr, &ra);
            if (st != MPM_OK) break;
            if (it == 0) r0r = rkr;
            const double rref = r0r > 1.0e-30 ? rkr / r0r : 0.0;
            if (rref < 1.0e-6 || r0r < 1.0e-6 || ra < 1.0e-8) break;
        }
    }
    *krylov = ktot;
    *newton = (it > iter_max ? iter_max : it) + 1;
    if (st == MPM_OK && s->nr_flag && it > iter_max) st = MPM_ERR_NEWTON_MAXIT;
    return st;
}

// Node2Particle (var_trans_solid_implicit.cpp:106-167)
static mpm_status imp_g2p(mpm_ctx *c) {
    ImpState *s = c->imp;
    ImpArgs a = imp_args(c);
    const int nb = nb_nodes(c);
    const int parity = (int)(c->step & 1);
    // PredictNewmarkBetaVelAndAccel + CommitNodalKinematics: nvel, naccel <- predicted
    k_imp_predict<<<nb, 256, 0, c->stream>>>(a, s->ndispl, s->nvel, s->naccel, s->naccel_k, s->Ap, 0);
    CKI(cudaMemcpyAsync(s->nvel, s->Ap, sizeof(double) * 3 * c->g.nodec, cudaMemcpyDeviceToDevice, c->stream));
    CKI(cudaMemcpyAsync(s->naccel, s->naccel_k, sizeof(double) * 3 * c->g.nodec, cudaMemcpyDeviceToDevice,
                        c->stream));
    k_imp_nei<<<nb, 256, 0, c->stream>>>(a, s->nvof, s->nei, s->part);
    k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_EU);
    k_imp_reset_next<<<1, 1, 0, c->stream>>>(c->d_ctl, parity);
    const int pb = (int)((c->num + 127) / 128);
    if (s->prec == 64) launch_g2p<double>(c, a, parity, pb);
    else launch_g2p<float>(c, a, parity, pb);
    c->launches += 7;
    return check_launch(c);
}

mpm_status mpm_gpu_implicit_step(mpm_ctx *c, int nsteps, double facl, double eps, int kmax, mpm_solve_stats *stats) {
    if (!c || !c->imp || nsteps < 0 || !(eps > 0.0) || kmax <= 0) return MPM_ERR_BAD_ARG;
    if (c->num == 0) return MPM_ERR_STATE;
    mpm_status st = ensure_particle_scratch(c);
    if (st != MPM_OK) return st;
    int kt = 0, nt = 0;
    const int fb0 = c->imp->fallbacks, na0 = c->imp->nn_applications;
    for (int i = 0; i < nsteps; i++) {
        st = imp_p2g(c, facl);
        if (st != MPM_OK) break;
        int k = 0, n = 0;
        st = imp_newton(c, eps, kmax, &k, &n);
        kt += k;
        nt += n;
        if (st != MPM_OK) break;
        st = imp_g2p(c);
        if (st != MPM_OK) break;
        c->step++;
        c->steps_since_sort++;
    }
    c->imp->krylov_total += kt;
    c->imp->newton_total += nt;
    if (stats) {
        stats->krylov_iters = kt;
        stats->newton_iters = nt;
        stats->last_rel_residual = c->imp->last_rel;
        stats->precond_fallbacks = c->imp->fallbacks - fb0;
        stats->nn_applications = c->imp->nn_applications - na0;
    }
    if (st != MPM_OK) return st;
    CKI(cudaStreamSynchronize(c->stream));
    return check_launch(c);
}

// ------------------------------------------------------------- test hooks
mpm_status mpm_gpu_implicit_assemble(mpm_ctx *c, double facl) {
    if (!c || !c->imp) return MPM_ERR_BAD_ARG;
    if (c->num == 0) return MPM_ERR_STATE;
    mpm_status st = ensure_particle_scratch(c);
    if (st != MPM_OK) return st;
    st = imp_p2g(c, facl);
    if (st != MPM_OK) return st;
    ImpState *s = c->imp;
    ImpArgs a = imp_args(c);
    if (copy_stress_k(c) != MPM_OK) return MPM_ERR_CUDA;
    CKI(cudaMemsetAsync(s->ndispl, 0, sizeof(double) * 3 * c->g.nodec, c->stream));
    CKI(cudaMemsetAsync(s->x, 0, sizeof(double) * 3 * c->g.nodec, c->stream));
    k_imp_predict<<<nb_nodes(c), 256, 0, c->stream>>>(a, s->ndispl, s->nvel, s->naccel, s->naccel_k, nullptr, 1);
    c->launches++;
    st = imp_assemble(c);
    if (st != MPM_OK) return st;
    CKI(cudaStreamSynchronize(c->stream));
    return MPM_OK;
}

mpm_status mpm_gpu_implicit_get_system(mpm_ctx *c, double *stencil, double *adiag, double *b_rhs) {
    if (!c || !c->imp) return MPM_ERR_BAD_ARG;
    ImpState *s = c->imp;
    const size_t N = (size_t)c->g.nodec;
    CKI(cudaStreamSynchronize(c->stream));
    if (stencil) {
        const int nq = 9 * imp_args(c).ns;
        if (s->prec == 64) {
            std::vector<double> t(a_size((int)N, s->qp));
            CKI(cudaMemcpy(t.data(), s->A, sizeof(double) * t.size(), cudaMemcpyDeviceToHost));
            for (int q = 0; q < nq; q++)
                for (size_t n = 0; n < N; n++) stencil[(size_t)q * N + n] = t[aidx(q, (int)n, s->qp)];
        } else {
            std::vector<float> t(a_size((int)N, s->qp));
            CKI(cudaMemcpy(t.data(), s->A, sizeof(float) * t.size(), cudaMemcpyDeviceToHost));
            for (int q = 0; q < nq; q++)
                for (size_t n = 0; n < N; n++) stencil[(size_t)q * N + n] = (double)t[aidx(q, (int)n, s->qp)];
        }
    }
    if (adiag) CKI(cudaMemcpy(adiag, s->adiag, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost));
    if (b_rhs) CKI(cudaMemcpy(b_rhs, s->b, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost));
    return MPM_OK;
}

mpm_status mpm_gpu_implicit_matvec(mpm_ctx *c, const double *x, double *y) {
    if (!c || !c->imp || !x || !y) return MPM_ERR_BAD_ARG;
    ImpState *s = c->imp;
    const size_t N = (size_t)c->g.nodec;
    CKI(cudaMemcpyAsync(s->xs, x, sizeof(double) * 3 * N, cudaMemcpyHostToDevice, c->stream));
    ImpArgs a = imp_args(c);
    timer_begin(c, K_MATVEC);
    launch_matvec(c, a, nb_nodes(c), s->xs, s->Ap, nullptr, true);
    timer_end(c, K_MATVEC);
    c->launches++;
    CKI(cudaMemcpyAsync(y, s->Ap, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost, c->stream));
    CKI(cudaStreamSynchronize(c->stream));
    return check_launch(c);
}

mpm_status mpm_gpu_implicit_solve(mpm_ctx *c, double eps, int kmax, double *x, int *iters) {
    if (!c || !c->imp || !(eps > 0.0) || kmax <= 0) return MPM_ERR_BAD_ARG;
    ImpState *s = c->imp;
    const size_t N = (size_t)c->g.nodec;
    CKI(cudaMemsetAsync(s->x, 0, sizeof(double) * 3 * N, c->stream));
    int it = 0;
    mpm_status st = s->net ? imp_fcg(c, eps, kmax, &it) : imp_cg(c, eps, kmax, &it);
    if (iters) *iters = it;
    if (x) CKI(cudaMemcpy(x, s->x, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost));
    return st;
}

// ------------------------------------------------ learned preconditioner hooks
mpm_status mpm_gpu_implicit_set_precond(mpm_ctx *c, mpm_nn *net) {
    if (!c || !c->imp) return MPM_ERR_BAD_ARG;
    if (net && !mpm_nn_grid_matches(net, c->g.nnc)) return MPM_ERR_BAD_ARG;
    c->imp->net = net;
    return MPM_OK;
}

// CG on the scaled system from x = 0 with right-hand side s->bs.  With a
// network, every `stride`-th iterate appends the pair (r_k, xstar - x_k).
static mpm_status cg_scaled(mpm_ctx *c, double eps, int kmax, mpm_nn *net, int stride, int max_pairs, int *iters) {
    ImpState *s = c->imp;
    ImpArgs a = imp_args(c);
    const int nb = nb_nodes(c);
    const size_t N = (size_t)c->g.nodec;
    CKI(cudaMemsetAsync(s->xs, 0, sizeof(double) * 3 * N, c->stream));
    CKI(cudaMemsetAsync(s->Ap, 0, sizeof(double) * 3 * N, c->stream));
    CKI(cudaMemcpyAsync(s->r, s->bs, sizeof(double) * 3 * N, cudaMemcpyDeviceToDevice, c->stream));
    k_cg_init<<<nb, 256, 0, c->stream>>>(a, s->Ap, s->r, s->p, s->part);
    k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_RR0);
    CKI(cudaMemcpyAsync(s->h_scal, s->scal, sizeof(double) * S_NSCAL, cudaMemcpyDeviceToHost, c->stream));
    CKI(cudaStreamSynchronize(c->stream));
    const double rr0 = s->h_scal[S_RR0];
    int it = 0, pairs = 0;
    bool done = !(rr0 > 1.0e-300);
    k_cg_start<<<(3 * c->g.nodec + 255) / 256, 256, 0, c->stream>>>(a, s->scal, 0.0, 0, s->r, s->p, s->p32);
    while (!done && it < kmax) {
        const int cur = (it & 1) ? S_RR1 : S_RR0;
        if (net && it % stride == 0 && pairs < max_pairs) {
            k_sub3<<<(3 * c->g.nodec + 255) / 256, 256, 0, c->stream>>>(s->xstar, s->xs, s->ev, 3 * c->g.nodec);
            mpm_status st = mpm_nn_append_pair(net, c->stream, s->r, s->scal + cur, s->ev);
            if (st != MPM_OK) return st;
            pairs++;
        }
        cg_iteration(c, a, nb, it, 0);
        it++;
        if (it % 8 == 0 || it == kmax) {
            CKI(cudaMemcpyAsync(s->h_scal, s->scal, sizeof(double) * 2, cudaMemcpyDeviceToHost, c->stream));
            CKI(cudaStreamSynchronize(c->stream));
            const double rr = s->h_scal[(it & 1) ? S_RR1 : S_RR0];
            if (rr != rr) return MPM_ERR_NONFINITE;
            if (rr < eps * rr0) done = true;
        }
    }
    *iters = it;
    return check_launch(c);
}

// Flexible GCR with the context's preconditioner from x = 0 for the RHS s->bs,
// storing (r_k, xstar - x_k) before each of its first `npairs` iterations.
static mpm_status gcr_record(mpm_ctx *c, mpm_nn *rec, int npairs) {
    ImpState *s = c->imp;
    ImpArgs a = imp_args(c);
    const int nb = nb_nodes(c);
    const size_t N = (size_t)c->g.nodec;
    CKI(cudaMemsetAsync(s->xs, 0, sizeof(double) * 3 * N, c->stream));
    CKI(cudaMemcpyAsync(s->r, s->bs, sizeof(double) * 3 * N, cudaMemcpyDeviceToDevice, c->stream));
    k_dot3<<<nb, 256, 0, c->stream>>>(a, s->r, s->r, s->part);
    k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_RRC);
    int used = 0, slot = 0;
    for (int k = 0; k < npairs; k++) {
        k_sub3<<<(3 * c->g.nodec + 255) / 256, 256, 0, c->stream>>>(s->xstar, s->xs, s->ev, 3 * c->g.nodec);
        mpm_status st = mpm_nn_append_pair(rec, c->stream, s->r, s->scal + S_RRC, s->ev);
        if (st != MPM_OK) return st;
        st = gcr_iter(c, a, nb, used, slot);
        if (st != MPM_OK) return st;
        // the pairs are scaled by the residual's own norm
        k_dot3<<<nb, 256, 0, c->stream>>>(a, s->r, s->r, s->part);
        k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_RRC);
        used = used < s->gm ? used + 1 : s->gm;
        slot = (slot + 1) % s->gm;
    }
    return check_launch(c);
}

mpm_status mpm_gpu_implicit_harvest(mpm_ctx *c, mpm_nn *net, int nsystems, int loads_per_system, int pairs_per_load,
                                    double e_min, double e_max, uint64_t seed, double eps, int kmax) {
    if (!c || !c->imp || !net || nsystems < 1 || loads_per_system < 1 || pairs_per_load < 1 || !(e_min > 0.0) ||
        !(e_max >= e_min) || !(eps > 0.0) || kmax < 1)
        return MPM_ERR_BAD_ARG;
    if (!mpm_nn_grid_matches(net, c->g.nnc)) return MPM_ERR_BAD_ARG;
    if (c->num == 0) return MPM_ERR_STATE;
    ImpState *s = c->imp;
    ImpArgs a = imp_args(c);
    const int nb = nb_nodes(c);
    const size_t N = (size_t)c->g.nodec;
    std::vector<double> saved(3 * (size_t)c->nmat);
    CKI(cudaMemcpy(saved.data(), c->d_matprop, sizeof(double) * saved.size(), cudaMemcpyDeviceToHost));
    mpm_status st = MPM_OK;
    uint64_t z = seed;
    auto next_unit = [&z]() {
        z += 0x9E3779B97F4A7C15ull;
        uint64_t t = z;
        t = (t ^ (t >> 30)) * 0xBF58476D1CE4E5B9ull;
        t = (t ^ (t >> 27)) * 0x94D049BB133111EBull;
        t ^= t >> 31;
        return ((t >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    };
    for (int sys = 0; sys < nsystems && st == MPM_OK; sys++) {
        const double E = exp(log(e_min) + next_unit() * (log(e_max) - log(e_min)));
        k_set_modulus<<<1, 32, 0, c->stream>>>(c->d_matprop, c->nmat, E);
        st = mpm_gpu_implicit_assemble(c, 1.0);
        if (st == MPM_OK) {
            k_phi<<<nb, 256, 0, c->stream>>>(a, s->nmass, s->adiag, s->ev);
            st = mpm_nn_begin_system(net, c->stream, s->ev);
            if (st == MPM_OK && s->net) st = mpm_nn_set_feature(s->net, c->stream, s->ev);
        }
        for (int ld = 0; ld < loads_per_system && st == MPM_OK; ld++) {
            const uint64_t key = seed * 1000003ull + (uint64_t)sys * 1009ull + (uint64_t)ld;
            if (ld == 0) {
                // the assembled system's own right-hand side (body force and inertia)
                k_cg_scale_in<<<nb, 256, 0, c->stream>>>(a, s->x, s->b, s->adiag, s->xs, s->bs);
            } else {
                // alternate smooth-dominated and noise-dominated loads
                const double smooth = (ld & 1) ? 0.2 : 1.0, noise = (ld & 1) ? 1.0 : 0.2;
                k_random_rhs<<<nb, 256, 0, c->stream>>>(a, s->adiag, key, smooth, noise, s->bs);
            }
            int K = 0;
            st = cg_scaled(c, eps, kmax, nullptr, 1, 0, &K);
            if (st != MPM_OK) break;
            CKI(cudaMemcpyAsync(s->xstar, s->xs, sizeof(double) * 3 * N, cudaMemcpyDeviceToDevice, c->stream));
            if (s->net) {
                // pairs along the learned solve itself: the residuals the
                // preconditioner meets once it has removed what it can
                st = gcr_record(c, net, pairs_per_load);
            } else {
                const int stride = K / pairs_per_load > 1 ? K / pairs_per_load : 1;
                int K2 = 0;
                st = cg_scaled(c, eps, K, net, stride, pairs_per_load, &K2);
            }
        }
    }
    cudaMemcpy(c->d_matprop, saved.data(), sizeof(double) * saved.size(), cudaMemcpyHostToDevice);
    if (st != MPM_OK) return st;
    CKI(cudaStreamSynchronize(c->stream));
    return check_launch(c);
}

// Test hook: z = M(r) for host arrays r, z (3 * nodec, scaled system) with the
// preconditioner set on ctx and the features of the assembled system.
mpm_status mpm_gpu_implicit_apply_precond(mpm_ctx *c, const double *r, double *z) {
    if (!c || !c->imp || !c->imp->net || !r || !z) return MPM_ERR_BAD_ARG;
    ImpState *s = c->imp;
    ImpArgs a = imp_args(c);
    const int nb = nb_nodes(c);
    const size_t N = (size_t)c->g.nodec;
    CKI(cudaMemcpyAsync(s->r, r, sizeof(double) * 3 * N, cudaMemcpyHostToDevice, c->stream));
    k_phi<<<nb, 256, 0, c->stream>>>(a, s->nmass, s->adiag, s->ev);
    mpm_status st = mpm_nn_set_feature(s->net, c->stream, s->ev);
    if (st != MPM_OK) return st;
    k_dot3<<<nb, 256, 0, c->stream>>>(a, s->r, s->r, s->part);
    k_finish<<<1, 256, 0, c->stream>>>(s->part, nb, s->scal, S_RRC);
    st = mpm_nn_apply_precond(s->net, c->stream, s->r, s->scal + S_RRC, s->adiag, a.bcflag, a.mtol, s->z);
    if (st != MPM_OK) return st;
    CKI(cudaMemcpyAsync(z, s->z, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost, c->stream));
    CKI(cudaStreamSynchronize(c->stream));
    return check_launch(c);
}
