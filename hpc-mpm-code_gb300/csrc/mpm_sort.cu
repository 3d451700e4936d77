// Particle binning and sorting.
//
// MeshPointLinklist (module/material_point.cpp:52-78) rebuilds a per-cell
// linked list every step; here every kernel recomputes a particle's cell from
// its position (the per-step binning), and every resort_period steps the
// particles are physically reordered by
//     (4x4x8-cell brick, cell inside the brick, load index)
// so that one CTA owns a brick and one thread owns a cell.  The order inside
// a cell is the load order (the reference visits a cell's particles in index
// order too), which makes the reordering deterministic.
//
//   k_bin         brick key + brick histogram
//   k_scan_up / k_scan_down
//                 brick starts, work-item list (chunks of <= CHUNK particles),
//                 list of non-empty bricks: a scan over segments
//   k_scatter     particles grouped by brick (order within a brick arbitrary)
//   k_cell_sort   per brick: cell histogram and starts, then each particle's
//                 rank inside its cell by load index; a crowded brick's shares
//   k_permute     the particle fields moved into the sorted order
#include <algorithm>

#include "mpm_device.cuh"

namespace mpm {

template <typename R>
__global__ void k_bin(KGeom<R> g, int nbx, int nby, const R *x0, const R *x1, const R *x2, int n, int *key,
                      int *bcount, unsigned *oob_count) {
    pdl_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool oob = false;
    int k = -1;
    if (i < n) {
        int cx = cell_of(x0[i], g, 0, oob), cy = cell_of(x1[i], g, 1, oob), cz = cell_of(x2[i], g, 2, oob);
        int b = cx / BRX + nbx * (cy / BRY + nby * (cz / BRZ));
        int lc = (cx % BRX) + BRX * ((cy % BRY) + BRY * (cz % BRZ));
        k = b;
        key[i] = b * BRC + lc;
    }
    unsigned act = __ballot_sync(0xffffffffu, i < n);
    if (i < n) {
        unsigned peers = __match_any_sync(act, k);
        int leader = __ffs(peers) - 1;
        if ((int)(threadIdx.x & 31) == leader) atomicAdd(&bcount[k], __popc(peers));
    }
    unsigned bad = __ballot_sync(0xffffffffu, oob);
    if ((threadIdx.x & 31) == 0 && bad) atomicAdd(oob_count, __popc(bad));
}

// Exclusive scan of the brick counts over segments of SCAN_SEG bricks: (1) each CTA
// sums its segment's particles, work items (chunks of <= CHUNK particles) and
// non-empty bricks (not launched for one segment); (2) each CTA adds the segments
// before its own, scans its segment again in brick order from there and writes
// the brick starts, the work list, the list of non-empty bricks and an empty
// brick's (equal) cell bounds, and resets the counters for the next sort.  Every
// load and store of the brick arrays is coalesced.
constexpr int SCAN_T = 1024;                 // threads per CTA
constexpr int SCAN_ITEMS = SCAN_SEG / SCAN_T;  // bricks per thread and segment
static_assert(SCAN_ITEMS * SCAN_T == SCAN_SEG, "scan segment");

struct Tri {
    int c, k, a;   // particles, work items, non-empty bricks
};
__device__ __forceinline__ Tri tri_of(int c) { return Tri{c, (c + CHUNK - 1) / CHUNK, c > 0 ? 1 : 0}; }

// inclusive block-wide scan of (c, k, a) over SCAN_T threads; the block total in *tot
__device__ __forceinline__ Tri block_scan(Tri v, Tri *sh, Tri *tot) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int c = __shfl_up_sync(0xffffffffu, v.c, o), k = __shfl_up_sync(0xffffffffu, v.k, o),
                  a = __shfl_up_sync(0xffffffffu, v.a, o);
        if (lane >= o) {
            v.c += c;
            v.k += k;
            v.a += a;
        }
    }
    if (lane == 31) sh[wid] = v;
    __syncthreads();
    if (wid == 0) {
        Tri w = lane < (SCAN_T >> 5) ? sh[lane] : Tri{0, 0, 0};
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int c = __shfl_up_sync(0xffffffffu, w.c, o), k = __shfl_up_sync(0xffffffffu, w.k, o),
                      a = __shfl_up_sync(0xffffffffu, w.a, o);
            if (lane >= o) {
                w.c += c;
                w.k += k;
                w.a += a;
            }
        }
        if (lane < (SCAN_T >> 5)) sh[lane] = w;   // inclusive warp offsets
    }
    __syncthreads();
    if (wid > 0) {
        const Tri b = sh[wid - 1];
        v.c += b.c;
        v.k += b.k;
        v.a += b.a;
    }
    *tot = sh[(SCAN_T >> 5) - 1];
    __syncthreads();   // sh is reused by the next call
    return v;
}

__global__ void __launch_bounds__(SCAN_T) k_scan_up(int nb, const int *__restrict__ bcount, int *part) {
    __shared__ Tri sh[32];
    pdl_wait();
    const int base = blockIdx.x * SCAN_SEG;
    Tri v{0, 0, 0};
#pragma unroll
    for (int r = 0; r < SCAN_ITEMS; r++) {
        const int t = base + r * SCAN_T + threadIdx.x;
        if (t < nb) {
            const Tri q = tri_of(bcount[t]);
            v.c += q.c;
            v.k += q.k;
            v.a += q.a;
        }
    }
    Tri tot;
    block_scan(v, sh, &tot);
    if (threadIdx.x == 0) {
        part[3 * blockIdx.x] = tot.c;
        part[3 * blockIdx.x + 1] = tot.k;
        part[3 * blockIdx.x + 2] = tot.a;
    }
}

__global__ void __launch_bounds__(SCAN_T) k_scan_down(int nb, int nseg, int *bcount, int *bstart, int *bcursor,
                                                      WorkItem *work, int *nwork, int cap, int *blist, int *nblist,
                                                      int *nshares, const int *part, int *cstart) {
    __shared__ Tri sh[32];
    pdl_wait();
    const int base = blockIdx.x * SCAN_SEG;
    Tri carry{0, 0, 0};
    if (blockIdx.x > 0) {
        Tri v{0, 0, 0};
        for (int i = threadIdx.x; i < (int)blockIdx.x; i += SCAN_T) {
            v.c += part[3 * i];
            v.k += part[3 * i + 1];
            v.a += part[3 * i + 2];
        }
        block_scan(v, sh, &carry);
    }
    for (int r = 0; r < SCAN_ITEMS; r++) {
        const int t = base + r * SCAN_T + threadIdx.x;
        const int c = t < nb ? bcount[t] : 0;
        const Tri v = tri_of(c);
        Tri tot;
        const Tri inc = block_scan(v, sh, &tot);
        if (t < nb) {
            const int pbase = carry.c + inc.c - v.c;
            int wbase = carry.k + inc.k - v.k;
            if (c > 0) blist[carry.a + inc.a - v.a] = t;
            else {
                // no kernel reads more of an empty brick's cell starts
                int *cs = cstart + (size_t)t * (BRC + 1);
                cs[0] = pbase;
                cs[BRC] = pbase;
            }
            bstart[t] = pbase;
            bcursor[t] = 0;
            bcount[t] = 0;
            for (int b = 0; b < c; b += CHUNK) {
                if (wbase < cap) {
                    WorkItem w;
                    w.tile = t;
                    w.begin = pbase + b;
                    w.end = pbase + min(c, b + CHUNK);
                    work[wbase] = w;
                }
                wbase++;
            }
        }
        carry.c += tot.c;
        carry.k += tot.k;
        carry.a += tot.a;
    }
    if ((int)blockIdx.x == nseg - 1 && threadIdx.x == 0) {
        *nwork = min(carry.k, cap);
        *nblist = carry.a;
        *nshares = carry.a;   // k_cell_sort adds to it
        bstart[nb] = carry.c;
    }
}

__global__ void k_scatter(const int *key, int n, const int *bstart, int *bcursor, int *tmp) {
    pdl_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned act = __ballot_sync(0xffffffffu, i < n);
    if (i >= n) return;
    int k = key[i] / BRC;
    unsigned peers = __match_any_sync(act, k);
    int lane = threadIdx.x & 31;
    int leader = __ffs(peers) - 1;
    int rank = __popc(peers & ((1u << lane) - 1));
    int base = 0;
    if (lane == leader) base = atomicAdd(&bcursor[k], __popc(peers));
    base = __shfl_sync(peers, base, leader);
    tmp[bstart[k] + base + rank] = i;
}

// Persistent CTAs over the non-empty bricks.  tmp holds a brick's particles in
// arbitrary order; writes perm (sorted by cell, then load index) and the brick's cell
// starts.  A particle's rank inside its cell is the number of the cell's particles
// with a smaller load index: these are compared in shared memory (a brick of more
// than CS_CAP particles takes tmp2), where the pass over global memory took two
// dependent loads per comparison, and empty bricks have no CTA (a CTA each wrote all
// their cell starts).  With k_scatter, per sort: 243,675 particles, 27 per cell, 44 -> 23
// us; 64 scenes in 118,000 bricks 76 -> 30; 4,096,000 84 -> 74.
constexpr int CS_T = 256, CS_CAP = 4096;
__global__ void __launch_bounds__(CS_T) k_cell_sort(const int *bstart, const int *key, const int *pid, const int *tmp,
                                                    int *tmp2, int *perm, int *cstart, const int *blist,
                                                    const int *nblist, int run, BrickShare *shares,
                                                    int *nshares) {
    static_assert(CS_T >= BRC && BRC % 32 == 0 && BRC <= 256, "cell scan layout");
    __shared__ int s_cnt[BRC];         // counts, then cursors
    __shared__ int s_start[BRC + 1];
    __shared__ int s_w[BRC / 32], s_max[BRC / 32];
    __shared__ int s_shares, s_base;
    __shared__ int s_pid[CS_CAP], s_idx[CS_CAP];
    __shared__ unsigned char s_cell[CS_CAP];
    pdl_wait();
    const int tid = threadIdx.x, n = *nblist;
    for (int it = blockIdx.x; it < n; it += gridDim.x) {
        const int b = blist[it];
        const int lo = bstart[b], num = bstart[b + 1] - lo;
        int *cs = cstart + (size_t)b * (BRC + 1);
        if (tid < BRC) s_cnt[tid] = 0;
        __syncthreads();
        for (int j = tid; j < num; j += CS_T) atomicAdd(&s_cnt[key[tmp[lo + j]] % BRC], 1);
        __syncthreads();
        // exclusive scan of the BRC cell counts: warp scans, then the warp offsets
        int v = 0;
        if (tid < BRC) {
            v = s_cnt[tid];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, o);
                if ((tid & 31) >= o) v += u;
            }
            if ((tid & 31) == 31) s_w[tid >> 5] = v;
            if (run > 0) {
                const int mx = __reduce_max_sync(0xffffffffu, s_cnt[tid]);
                if ((tid & 31) == 31) s_max[tid >> 5] = mx;
            }
        }
        __syncthreads();
        if (tid < BRC) {
            for (int w = 0; w < (tid >> 5); w++) v += s_w[w];
            const int first = v - s_cnt[tid];
            s_start[tid] = first;
            s_cnt[tid] = first;
            cs[tid] = lo + first;
            if (tid == BRC - 1) {
                s_start[BRC] = v;
                cs[BRC] = lo + v;
            }
            if (run > 0 && tid == 0) {
                int mx = s_max[0];
                for (int w = 1; w < BRC / 32; w++) mx = max(mx, s_max[w]);
                s_shares = max(1, (mx + run / 2) / run);
                shares[it] = BrickShare{b, 0, s_shares};
                if (s_shares > 1) s_base = atomicAdd(nshares, s_shares - 1) - 1;
            }
        }
        __syncthreads();
        if (run > 0)
            for (int q = 1 + tid; q < s_shares; q += CS_T) shares[s_base + q] = BrickShare{b, q, s_shares};
        const bool fits = num <= CS_CAP;
        for (int j = tid; j < num; j += CS_T) {
            const int i = tmp[lo + j], c = key[i] % BRC, q = atomicAdd(&s_cnt[c], 1);
            if (fits) {
                s_idx[q] = i;
                s_pid[q] = pid[i];
                s_cell[q] = (unsigned char)c;
            } else {
                tmp2[lo + q] = i;
            }
        }
        __syncthreads();
        for (int j = tid; j < num; j += CS_T) {
            const int i = fits ? s_idx[j] : tmp2[lo + j], c = fits ? (int)s_cell[j] : key[i] % BRC;
            const int me = fits ? s_pid[j] : pid[i], q0 = s_start[c], q1 = s_start[c + 1];
            int r = 0;
            if (fits)
                for (int q = q0; q < q1; q++) r += s_pid[q] < me;
            else
                for (int q = q0; q < q1; q++) r += pid[tmp2[lo + q]] < me;
            perm[lo + q0 + r] = i;
        }
        __syncthreads();   // shared memory is reused by the next brick
    }
}

// dst[j] = src[perm[j]] for all real fields and the two int fields.  The
// two buffers never overlap; eight fields are loaded before they are stored
// so that a thread keeps eight gathers in flight.
template <typename R>
__global__ void k_permute(const R *__restrict__ src, R *__restrict__ dst, const int *__restrict__ perm, int n,
                          int nreal, size_t N, int skip_lo, int skip_hi) {
    pdl_wait();
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const size_t i = (size_t)perm[j];
    // fields [skip_lo, skip_hi) are not moved (no kernel of the context reads them)
    const int nmove = nreal - (skip_hi - skip_lo);
    auto field = [&](int k) { return k < skip_lo ? k : k + (skip_hi - skip_lo); };
    int q = 0;
    for (; q + 8 <= nmove; q += 8) {
        R v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = __ldg(src + (size_t)field(q + k) * N + i);
#pragma unroll
        for (int k = 0; k < 8; k++) dst[(size_t)field(q + k) * N + j] = v[k];
    }
    for (; q < nmove; q++) dst[(size_t)field(q) * N + j] = __ldg(src + (size_t)field(q) * N + i);
    const int *si = (const int *)(src + (size_t)nreal * N);
    int *di = (int *)(dst + (size_t)nreal * N);
    const int a0 = __ldg(si + i), a1 = __ldg(si + N + i);
    di[j] = a0;
    di[N + j] = a1;
}

// Particles of a cell that one share takes.  The scatters of mpm_cells.cu give a
// cell to a few threads, which walk its particles one after another, and a brick to a
// CTA per slab: crowded cells in fewer bricks than the chip holds CTAs leave it idle.
// So a brick whose fullest cell holds 48 particles or more is cut into shares, each
// with a run of every cell's particles.  Where the bricks fill the chip (two CTAs per
// SM), only what is three times their average load is cut: another share costs
// another node pass (cut in two all the same, 970,299 FP64 particles at 27 per cell
// took 1563 us per step in place of 1380, 1,000,000 at 64 per cell with APIC 2963 in
// place of 2739).  Step without and with shares, and with the staging box: FP64 linear,
// 216,000 particles at 64 per cell 775, 489 and 1161 us, at 216 per cell 1800, 465 and
// 1262; FP64 APIC, 27,000 at 216 per cell 1775, 366 and 950; FP32 quadratic, 216,000 at
// 216 per cell 409, 247 and 2489; a 4^3-cell corner of 1,000,000 FP64 particles
// squeezed to 216 per cell 2315, 1638 and 2789.
static int share_run(int64_t n, int nsm) {
    const int64_t avg = n / ((int64_t)2 * nsm * BRC);
    return (int)std::max<int64_t>(SHARE_RUN, 3 * avg);
}

// FP32 linear explicit grids have kernels of their own, which take whole bricks.
static bool lists_shares(const mpm_ctx *c) {
    return c->cell_scatter && !(c->precision == 32 && c->g.order[0] == 1 && c->nreal != 27);
}

template <typename R>
static mpm_status sort_impl(mpm_ctx *c) {
    int n = (int)c->num;
    if (n == 0) return MPM_OK;
    KGeom<R> g;
    for (int d = 0; d < 3; d++) {
        g.xmin[d] = (R)c->g.xmin[d];
        g.dx[d] = (R)c->g.dx[d];
        g.inv_dx[d] = (R)(1.0 / c->g.dx[d]);
        g.nel[d] = c->g.nel[d];
        g.nnc[d] = c->g.nnc[d];
        g.ntile[d] = c->g.ntile[d];
    }
    g.nodec = c->g.nodec;
    const R *src = (const R *)c->pbuf[c->cur];
    R *dst = (R *)c->pbuf[c->cur ^ 1];
    size_t N = c->pstride;
    const int *pid = (const int *)(src + c->nreal * N) + N;
    int nb = (n + 255) / 256;
    timer_begin(c, K_BIN);
    const bool pdl = c->pdl != 0;
    launch(pdl, k_bin<R>, nb, 256, 0, c->stream, g, c->g.nbrick[0], c->g.nbrick[1], src, src + N, src + 2 * N, n, c->d_key,
           c->d_tcount, &c->d_ctl->err_oob);
    timer_end(c, K_BIN);
    timer_begin(c, K_SCAN);
    {
        const int nseg = (c->g.nbricks + SCAN_SEG - 1) / SCAN_SEG;
        if (nseg > 1) {
            launch(pdl, k_scan_up, nseg, SCAN_T, 0, c->stream, c->g.nbricks, (const int *)c->d_tcount, c->d_scanpart);
            c->launches++;
        }
        launch(pdl, k_scan_down, nseg, SCAN_T, 0, c->stream, c->g.nbricks, nseg, c->d_tcount, c->d_tstart, c->d_tcursor,
               c->d_work, c->d_nwork, c->nwork_cap, c->d_blist, c->d_nblist, c->d_nshares, (const int *)c->d_scanpart,
               c->d_cstart);
    }
    timer_end(c, K_SCAN);
    timer_begin(c, K_SCATTER);
    launch(pdl, k_scatter, nb, 256, 0, c->stream, (const int *)c->d_key, n, (const int *)c->d_tstart, c->d_tcursor,
           c->d_tmp);
    int nsm = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    launch(pdl, k_cell_sort, std::min(c->g.nbricks, 6 * nsm), CS_T, 0, c->stream, (const int *)c->d_tstart,
           (const int *)c->d_key, pid, (const int *)c->d_tmp, c->d_perm2, c->d_perm, c->d_cstart,
           (const int *)c->d_blist, (const int *)c->d_nblist, lists_shares(c) ? share_run(n, nsm) : 0,
           c->d_shares, c->d_nshares);
    timer_end(c, K_SCATTER);
    timer_begin(c, K_PERMUTE);
    // a Tait-fluid context keeps J - 1 in the first F field and never reads the other eight
    const int skip_lo = c->fluid_j ? 7 : 0, skip_hi = c->fluid_j ? 15 : 0;
    launch(pdl, k_permute<R>, nb, 256, 0, c->stream, src, dst, (const int *)c->d_perm, n, c->nreal, N, skip_lo, skip_hi);
    timer_end(c, K_PERMUTE);
    c->launches += 5;
    c->cur ^= 1;
    c->resorts++;
    c->steps_since_sort = 0;
    return check_launch(c);
}

mpm_status sort_particles(mpm_ctx *c) { return c->precision == 64 ? sort_impl<double>(c) : sort_impl<float>(c); }

}  // namespace mpm
