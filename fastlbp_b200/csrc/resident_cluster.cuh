// The cluster run kernel: a small graph's whole run inside the shared memory
// of one thread-block cluster.
//
// The resident kernel (resident.cuh) exchanges messages through L2 and
// separates the passes by grid barriers, about 4 us per sweep phase however
// small the graph is. A graph of up to some 150 k slots fits into the shared memory of
// one cluster: every block holds the incoming messages of its own items
// (factor items: vf, variable items: fv), and an item's outputs are stored
// straight into the receiving block's shared memory (st.shared::cluster), so
// that a phase costs its arithmetic and one hardware cluster barrier, and no
// scattered store ever reaches L2. Clusters take graphs from a queue one
// after the other: a batch of small graphs, or an engine's evidence sets, is
// solved with each graph at its own pace and no synchronisation between
// graphs.
//
// Positions are translated once per job: every block publishes the shared
// address of each run of four of its entries (slots) in a map in global
// memory, and after a cluster barrier replaces its items' positions by the
// receiving addresses. Cut entries of an evidence set become positions that
// nothing is stored to.
//
// What bounds it: the latency of one item per warp and of the cluster barrier
// (about 0.8 us with its fences) on the smallest graphs, on larger ones the
// remote stores, which an SM sends and takes in at about one in two cycles -
// no faster than L2 takes scattered stores, so that a graph spread over 16
// blocks gains nothing above some 40 k slots. Measured on one B200 in FP32,
// whole calls, the two launches a sweep against this kernel: 30 tolerance
// sweeps of 17 k slots 0.51 : 0.25 ms; 64 evidence sets of 12 k slots 2.2 :
// 0.86 ms; 64 graphs of 500 to 1,000 tuples 3.7 : 0.71 ms; 48 graphs of 1 k to
// 50 k tuples, the larger ones in the passes, 8.8 : 6.6 ms.
//
// Items are evaluated by the functions of the pass kernels in the same order
// per item, so a run gives the same bits as the other forms. Messages,
// damped messages and beliefs go back to global memory when a job ends, in
// the state the other forms leave. Groups that two graphs of a batch share
// are held by both jobs, each using and writing back its own lanes.
#pragma once

#include <type_traits>

#include "kernels.cuh"
#include "resident.cuh"

namespace flbp {

// One graph (or one evidence set's graph): its groups, large items and the
// range of its internal factors and variables; group: its index in the
// engine's per-group stop state.
struct ClusterJob {
    uint32_t fg0, fg1, f_lo, f_hi, fb0, fb1;
    uint32_t vg0, vg1, v_lo, v_hi, vb0, vb1;
    uint32_t group, pad[3];
};

template <typename T>
struct ClusterArgs {
    FactorArgs f;
    VarArgs v;
    T *vf, *fv, *fvd;
    T d;
    Ctl *ctl;
    const ClusterJob *jobs;  // in the order they are taken
    uint32_t n_jobs;
    int groups;              // jobs stop by themselves into v.gstate (else one job, the control block's run)
    int sets;                // jobs are evidence sets: per-set strides apply
    uint32_t *map;           // map_words words per cluster
    uint32_t map_words;
    uint32_t cap;            // sweeps of this launch at most, per job
    int final_beliefs;       // fixed runs: the last sweep also writes the beliefs
    uint32_t rows_f, rows_v; // items per block at most, over the jobs
    double *gdiff;           // groups: last belief change of every group
    const uint32_t *cut_ent; // sets: bits of the entries no message reaches, per set, or null
    uint32_t cut_words;
};

template <typename T>
constexpr int kClusterThreads = sizeof(T) == 4 ? 1024 : 512;

// Shared-memory layout of one item, in words (multiples of 4): messages,
// translated positions, then a factor's degrees and kinds (16 bits each item)
// and (p, q), or a variable's priors and (damping) its damped messages. A
// large item has one degree, (p, q) or prior, and its slots rounded up to 4.
__host__ __device__ __forceinline__ uint32_t cluster_slots(bool big, uint32_t w) {
    return big ? (w + 3u) & ~3u : 32u * w;
}
__host__ __device__ __forceinline__ uint32_t cluster_meta_words(bool big) { return big ? 4u : 16u; }
__host__ __device__ __forceinline__ uint32_t cluster_prior_words(bool big, uint32_t tsize) {
    return big ? 4u : 32u * (tsize == 4 ? 2u : 4u);
}
__host__ __device__ __forceinline__ uint32_t cluster_item_words(bool factor, bool big, uint32_t w, uint32_t tsize,
                                                                bool damp) {
    const uint32_t n = cluster_slots(big, w), tw = tsize / 4;
    return factor ? n * (tw + 1u) + cluster_meta_words(big) + (big ? 4u : 64u * tw)
                  : n * (tw + 1u + (damp ? tw : 0u)) + cluster_prior_words(big, tsize);
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ uint32_t cluster_size() {
    uint32_t n;
    asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
    return n;
}

// Address of this block's shared variable in block `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(const void *p, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}

__device__ __forceinline__ void cluster_st(uint32_t a, float x) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(x) : "memory");
}
__device__ __forceinline__ void cluster_st(uint32_t a, double x) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(x) : "memory");
}
__device__ __forceinline__ void cluster_st(uint32_t a, uint32_t x) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(x) : "memory");
}
__device__ __forceinline__ void cluster_st(uint32_t a, unsigned long long x) {
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(x) : "memory");
}

// An item's outputs into the receiving blocks' shared memory.
template <typename T>
struct ClusterOut {
    __device__ __forceinline__ void operator()(uint32_t a, T o) const {
        if (a != kSentinel) cluster_st(a, o);
    }
};

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

template <typename T, bool DAMP>
__global__ void __launch_bounds__(kClusterThreads<T>, 1) cluster_kernel(ClusterArgs<T> r) {
    extern __shared__ __align__(128) uint32_t sm[];
    constexpr int NT = kClusterThreads<T>, NW = NT / 32;
    constexpr uint32_t TW = sizeof(T) / 4, PSZ = sizeof(T) == 4 ? 2 : 4;
    __shared__ double s_max[NW];
    __shared__ unsigned long long s_cnt[NW];
    __shared__ double s_cmax[16];               // every block's residual of the sweep
    __shared__ unsigned long long s_ccnt[16];   // and count of changes above the tolerance
    __shared__ uint32_t s_over;                 // block 0: the run's time is over
    __shared__ uint32_t s_job;
    __shared__ double s_pscale;
    Ctl *ctl = r.ctl;
    if (!r.groups && *(volatile int *)&ctl->done) return;  // the same for every block
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t nb = cluster_size(), b = cluster_rank(), cid = blockIdx.x / nb;
    const int mode = ctl->mode;
    const double tol = ctl->tol, damping = ctl->damping, maxtime_ns = ctl->maxtime_ns, n_vars = (double)ctl->n_vars;
    const long long t0 = ctl->t, run00 = ctl->run_sweeps, iters0 = ctl->iters0, maxiter = ctl->maxiter;
    const long long min_iters = ctl->min_iters, max_iters = ctl->max_iters;
    unsigned long long t_start = ctl->t_start_ns;
    if (r.groups || run00 == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_start));
    ResRow *rows = reinterpret_cast<ResRow *>(sm);
    uint32_t *map = r.map + (size_t)cid * r.map_words;
    const T *pqg = reinterpret_cast<const T *>(r.f.f_pq);
    if (tid == 0) s_over = 0;
    // A block's shared memory may be written by the others only once it has
    // started: blocks of a cluster are scheduled together, not started
    // together. (One barrier per launch; it also orders s_over's first value
    // before any remote store to it.)
    cluster_sync_all();

    for (;;) {
        // ---- the next job of the queue, for the whole cluster
        if (b == 0 && tid == 0) {
            const uint32_t j = atomicAdd(&ctl->rs.arrive, 1u);
            for (uint32_t k = 0; k < nb; k++) cluster_st(cluster_addr(&s_job, k), j);
        }
        cluster_sync_all();
        const uint32_t ji = s_job;
        if (ji >= r.n_jobs) break;  // no block touches another's shared memory after this
        const ClusterJob J = r.jobs[ji];
        const uint32_t set = r.sets ? J.group : 0u, G = r.v.n_graphs;
        VarArgs va = r.v;
        const T *gvf = r.vf + (r.sets ? set * r.v.set_vf_stride : 0);
        const T *gfv = r.fv + (r.sets ? set * r.v.set_fv_stride : 0);
        T *gfvd = r.fvd + (DAMP && r.sets ? set * r.v.set_fv_stride : 0);
        const uint32_t *cut = r.sets && r.cut_ent ? r.cut_ent + (size_t)set * r.cut_words : nullptr;
        if (r.sets) {
            va.prior = reinterpret_cast<const unsigned char *>(r.v.prior) + set * r.v.set_prior_stride;
            va.belief = r.v.belief + set * r.v.set_belief_stride;
        }
        const uint32_t nfb = J.fb1 - J.fb0, nvb = J.vb1 - J.vb0;
        const uint32_t n_f = nfb + (J.fg1 - J.fg0), n_v = nvb + (J.vg1 - J.vg0);
        const bool skip = r.groups && r.v.gstate[J.group] != 0;  // stopped in an earlier launch

        // ---- its items: shared-memory offsets, then contents
        const uint32_t fs0 = r.f.fg_base[J.fg0], fsn = r.f.fg_base[J.fg1] - fs0, fb0 = nfb ? r.f.fb_off[J.fb0] : 0u;
        const uint32_t vs0 = va.vg_base[J.vg0], vsn = va.vg_base[J.vg1] - vs0, vb0 = nvb ? va.vb_off[J.vb0] : 0u;
        const uint32_t fs_end = r.f.fg_base[r.f.n_fgroups], vs_end = va.vg_base[va.n_vgroups];
        uint32_t *vmap = map;  // entries, then slots, four to a word
        uint32_t *fmap = map + (r.map_words >> 1);
        for (uint32_t j = tid; j < r.rows_f + r.rows_v; j += NT) {
            const bool fac = j < r.rows_f;
            const uint32_t it = res_item_of(fac ? j : j - r.rows_f, b, nb), big = fac ? nfb : nvb;
            ResRow x{0u, 0u, 0u};
            if (!skip && it < (fac ? n_f : n_v)) {
                if (it < big) {
                    const uint32_t k = (fac ? J.fb0 : J.vb0) + it;
                    x = ResRow{fac ? r.f.fb_off[k] : va.vb_off[k], fac ? r.f.fb_deg[k] : va.vb_deg[k], 0u};
                } else {
                    const uint32_t *gb = fac ? r.f.fg_base : va.vg_base;
                    const uint32_t g = (fac ? J.fg1 : J.vg1) - 1 - (it - big), b0 = gb[g];
                    x = ResRow{b0, (gb[g + 1] - b0) >> 5, 0u};
                }
                x.off = cluster_item_words(fac, it < big, x.w, sizeof(T), DAMP);
            }
            rows[j] = x;
        }
        __syncthreads();
        if (wid == 0) {  // sizes to offsets, behind the table
            uint32_t at = (3u * (r.rows_f + r.rows_v) + 31u) & ~31u;
            for (uint32_t j0 = 0; j0 < r.rows_f + r.rows_v; j0 += 32) {
                const uint32_t j = j0 + lane, n = j < r.rows_f + r.rows_v ? rows[j].off : 0u;
                uint32_t incl = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += y;
                }
                if (j < r.rows_f + r.rows_v) rows[j].off = at + incl - n;
                at += __shfl_sync(0xffffffffu, incl, 31);
            }
        }
        __syncthreads();
        auto f_index = [&](uint32_t it) { return it < nfb ? r.f.nf_sell + J.fb0 + it : 32u * (J.fg1 - 1 - (it - nfb)); };
        auto v_index = [&](uint32_t it) { return it < nvb ? va.nv_sell + J.vb0 + it : 32u * (J.vg1 - 1 - (it - nvb)); };
        if (!skip) {
            for (uint32_t j = wid; j < r.rows_f + r.rows_v; j += NW) {
                const bool fac = j < r.rows_f;
                const uint32_t it = res_item_of(fac ? j : j - r.rows_f, b, nb);
                if (it >= (fac ? n_f : n_v)) continue;
                const ResRow x = rows[j];
                const bool big = it < (fac ? nfb : nvb);
                const uint32_t n = big ? x.w : 32u * x.w;
                T *xs = reinterpret_cast<T *>(sm + x.off);
                const T *src = fac ? gvf : gfv;
                for (uint32_t k = lane; k < n; k += 32) {
                    T m = src[x.base + k];
                    if (!fac && cut && ((cut[(x.base + k) >> 5] >> ((x.base + k) & 31u)) & 1u)) m = T(0);
                    xs[k] = m;
                }
                uint32_t *mp = fac ? fmap + ((big ? fsn + (x.base - fb0) : x.base - fs0) >> 2)
                                   : vmap + ((big ? vsn + (x.base - vb0) : x.base - vs0) >> 2);
                const uint32_t a0 = cluster_addr(xs, b);
                for (uint32_t q = lane; q < (n + 3) / 4; q += 32) mp[q] = a0 + 4u * q * (uint32_t)sizeof(T);
                uint32_t *cst = sm + x.off + cluster_slots(big, x.w) * (TW + 1);
                if (fac) {
                    const uint32_t fi = f_index(it) + (big ? 0u : (uint32_t)lane);
                    if (!big || lane == 0) {
                        const bool in = big || (fi >= J.f_lo && fi < J.f_hi);
                        T *pq = reinterpret_cast<T *>(cst + cluster_meta_words(big));
                        reinterpret_cast<uint16_t *>(cst)[lane] =
                            in ? (uint16_t)(r.f.f_kind[fi] << 8 | (big ? 1 : r.f.f_deg[fi])) : (uint16_t)0;
                        pq[2 * lane] = in ? pqg[2 * (size_t)fi] : T(0);
                        pq[2 * lane + 1] = in ? pqg[2 * (size_t)fi + 1] : T(0);
                    }
                } else {
                    const uint32_t v = v_index(it) + (big ? 0u : (uint32_t)lane);
                    if (big ? lane == 0 : (v >= J.v_lo && v < J.v_hi))
                        for (uint32_t k = 0; k < PSZ; k++)
                            cst[PSZ * lane + k] = reinterpret_cast<const uint32_t *>(va.prior)[(size_t)PSZ * v + k];
                    if (DAMP) {
                        T *fd = reinterpret_cast<T *>(cst + cluster_prior_words(big, sizeof(T)));
                        for (uint32_t k = lane; k < n; k += 32) fd[k] = gfvd[x.base + k];
                    }
                }
            }
        }
        cluster_sync_all();  // maps and messages of all blocks
        if (!skip) {
            for (uint32_t j = wid; j < r.rows_f + r.rows_v; j += NW) {  // positions to receiving addresses
                const bool fac = j < r.rows_f;
                const uint32_t it = res_item_of(fac ? j : j - r.rows_f, b, nb);
                if (it >= (fac ? n_f : n_v)) continue;
                const ResRow x = rows[j];
                const bool big = it < (fac ? nfb : nvb);
                const uint32_t n = big ? x.w : 32u * x.w, np = cluster_slots(big, x.w);
                uint32_t *pos = sm + x.off + np * TW;
                const uint32_t i0 = (fac ? f_index(it) : v_index(it)) + (big ? 0u : (uint32_t)lane);
                const bool in = big || (fac ? i0 >= J.f_lo && i0 < J.f_hi : i0 >= J.v_lo && i0 < J.v_hi);
                for (uint32_t k = lane; k < n; k += 32) {
                    uint32_t e = in ? (fac ? r.f.f_pos[x.base + k] : va.v_ent[x.base + k]) : kSentinel;
                    if (fac && cut && e != kSentinel && ((cut[e >> 5] >> (e & 31u)) & 1u)) e = kSentinel;
                    if (e != kSentinel) {
                        const uint32_t rel = fac ? (e < vs_end ? e - vs0 : vsn + (e - vb0))
                                                 : (e < fs_end ? e - fs0 : fsn + (e - fb0));
                        e = __ldcg((fac ? vmap : fmap) + (rel >> 2)) + (rel & 3u) * (uint32_t)sizeof(T);
                    }
                    pos[k] = e;
                }
            }
            __syncwarp();
        }

        // ---- the run
        const long long run0 = r.groups ? (long long)r.v.gstate[2 * G + J.group] : run00;
        double node_frac_tol = ctl->node_frac_tol, frac = ctl->frac, maxdiff = ctl->maxdiff;
        unsigned long long nonconv = 0;
        int reason = FLBP_DIVERGED, stop = 0;  // stop: 1 finished, 2 time over
        uint32_t s = 0;
        for (; !skip && s < r.cap;) {
            if (tid == 0) s_pscale = (damping == 0.0) ? 1.0 : 1.0 - pow(damping, (double)(t0 + (r.groups ? run0 : 0) + (long long)s + 1));
            for (uint32_t j = wid; j < r.rows_f; j += NW) {
                const uint32_t it = res_item_of(j, b, nb);
                if (it >= n_f) break;
                const ResRow x = rows[j];
                const bool big = it < nfb;
                const uint32_t np = cluster_slots(big, x.w);
                const T *xs = reinterpret_cast<const T *>(sm + x.off);
                const uint32_t *pos = sm + x.off + np * TW, *cst = pos + np;
                const T *pq = reinterpret_cast<const T *>(cst + cluster_meta_words(big));
                const uint16_t *meta = reinterpret_cast<const uint16_t *>(cst);
                if (big) {
                    factor_tile_item<T>(xs, pos, x.w, (uint8_t)(meta[0] >> 8), pq[0], pq[1], lane, ClusterOut<T>{});
                } else {
                    const int deg = meta[lane] & 0xff;
                    const uint8_t kind = (uint8_t)(meta[lane] >> 8);
                    const T p = pq[2 * lane], q = pq[2 * lane + 1];
                    auto vb = [&](int k) { return xs[32 * k + lane]; };
                    auto ps = [&](int k) { return pos[32 * k + lane]; };
                    if (deg > 0) {
                        // columns past the group's width hold no slot: not read
                        auto vbn = [&](int k) { return (uint32_t)k < x.w ? vb(k) : T(0); };
                        if (x.w <= 4u) factor_reg<T, 4, true>(vbn, ps, deg, kind, p, q, ClusterOut<T>{});
                        else if (x.w <= 8u) factor_reg<T, 8, true>(vbn, ps, deg, kind, p, q, ClusterOut<T>{});
                        else factor_reg<T, kSellFactorDegree>(vb, ps, deg, kind, p, q, ClusterOut<T>{});
                    }
                }
            }
            cluster_sync_all();

            const bool last = s + 1 == r.cap;
            const int bm = mode == 3 ? 1 : mode != 0 ? mode : (last && r.final_beliefs) ? 3 : 0;
            const double pscale = s_pscale;
            double dmax = 0.0;
            unsigned long long cnt = 0;
            for (uint32_t j = wid; j < r.rows_v; j += NW) {
                const uint32_t it = res_item_of(j, b, nb);
                if (it >= n_v) break;
                const ResRow x = rows[r.rows_f + j];
                const bool big = it < nvb;
                const uint32_t np = cluster_slots(big, x.w);
                const T *xs = reinterpret_cast<const T *>(sm + x.off);
                const uint32_t *pos = sm + x.off + np * TW, *prior = pos + np;
                T *fd = reinterpret_cast<T *>(sm + x.off + np * (TW + 1) + cluster_prior_words(big, sizeof(T)));
                const uint32_t v = v_index(it) + (big ? 0u : (uint32_t)lane);
                const bool real = big ? lane == 0 : (v >= J.v_lo && v < J.v_hi);
                const double bold = (real && (bm == 1 || bm == 2)) ? va.belief[v] : 0.0;
                double Sv;
                int npos = 0, nneg = 0;
                if (big) {
                    typename WideAcc<T>::type S;
                    auto in = [&](uint32_t k) { return xs[k]; };
                    auto old = [&](uint32_t k) { return DAMP ? fd[k] : T(0); };
                    var_warp_sum<T, DAMP>(in, old, x.w, prior, 0u, r.d, pscale, lane, S, npos, nneg);
                    var_warp_send<T, DAMP, true>(in, old, [&](uint32_t k) { return pos[k]; }, fd, x.w, r.d, lane, S,
                                                 npos, nneg, ClusterOut<T>{});
                    Sv = AccOps<typename WideAcc<T>::type>::value(S);
                } else {
                    typedef typename NarrowAcc<T>::type A;
                    A S = AccOps<A>::zero();
                    if (real) decode_prior<T>(prior, lane, pscale, S, npos, nneg);
                    auto group = [&](auto width) {
                        constexpr int W = decltype(width)::value;
                        T xr[W], xo[DAMP ? W : 1];
#pragma unroll
                        for (int k = 0; k < W; k++) {
                            xr[k] = (uint32_t)k < x.w ? xs[32 * k + lane] : T(0);
                            if (DAMP) xo[k] = (uint32_t)k < x.w ? fd[32 * k + lane] : T(0);
                        }
                        var_lane_sum<T, W, DAMP>(x.w, xr, xo, r.d, S, npos, nneg);
                        if (DAMP) {
#pragma unroll
                            for (int k = 0; k < W; k++)
                                if ((uint32_t)k < x.w) fd[32 * k + lane] = xr[k];
                        }
                        var_lane_send<T, W>(x.w, xr, [&](int k) { return pos[32 * k + lane]; }, S, npos, nneg,
                                            ClusterOut<T>{});
                    };
                    if (real) {
                        if (x.w <= (uint32_t)kResNarrow) group(std::integral_constant<int, kResNarrow>());
                        else group(std::integral_constant<int, (int)kSellVarDegree>());
                    }
                    Sv = AccOps<A>::value(S);
                }
                if (bm && real) {
                    double dd = 0.0;
                    if (bm == 1) dd = var_finish<1>(va, v, Sv, npos, nneg, tol, bold, cnt);
                    else if (bm == 2) dd = var_finish<2>(va, v, Sv, npos, nneg, tol, bold, cnt);
                    else var_finish<3>(va, v, Sv, npos, nneg, tol, bold, cnt);
                    dmax = fmax(dmax, dd);
                }
            }
            s++;
            if (mode == 0) {
                cluster_sync_all();
                continue;
            }
            // ---- residual, to every block; stop rule
            dmax = warp_max(dmax);
            if (mode == 2) cnt = warp_sum(cnt);
            if (lane == 0) {
                s_max[wid] = dmax;
                s_cnt[wid] = cnt;
            }
            __syncthreads();
            if (wid == 0) {
                const double m = warp_max(lane < NW ? s_max[lane] : 0.0);
                const unsigned long long c = mode == 2 ? warp_sum(lane < NW ? s_cnt[lane] : 0ull) : 0ull;
                if ((uint32_t)lane < nb) {
                    cluster_st(cluster_addr(&s_cmax[b], lane), m);
                    if (mode == 2) cluster_st(cluster_addr(&s_ccnt[b], lane), c);
                    if (b == 0) {
                        unsigned long long now;
                        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
                        const double elapsed = (double)(now - t_start);
                        if (mode == 2 ? elapsed > maxtime_ns : elapsed >= maxtime_ns)
                            cluster_st(cluster_addr(&s_over, lane), 1u);
                    }
                }
            }
            cluster_sync_all();
            maxdiff = warp_max((uint32_t)lane < nb ? s_cmax[lane] : 0.0);
            const bool over = *(volatile uint32_t *)&s_over != 0;
            const long long n = run0 + (long long)s;
            if (mode == 2) {  // the rules of stop_rules
                nonconv = warp_sum((uint32_t)lane < nb ? s_ccnt[lane] : 0ull);
                frac = (double)nonconv / n_vars;
                if (n >= min_iters) node_frac_tol = (double)(n - min_iters) / (double)(max_iters - min_iters);
                if (maxdiff <= tol) {
                    stop = 1;
                    reason = FLBP_ALL_CONVERGED;
                } else if (n > min_iters && frac < node_frac_tol) {
                    stop = 1;
                    reason = FLBP_BIG_FRAC_CONVERGED;
                } else if (n > max_iters || over) {
                    stop = 1;
                }
            } else if (mode == 1) {
                if (!(iters0 + n < maxiter && maxdiff > tol && !over)) {
                    stop = 1;
                    reason = (maxdiff > tol) ? FLBP_DIVERGED : FLBP_ALL_CONVERGED;
                }
            } else {  // the rule of batch_stop_rules
                if (!(maxdiff > tol)) {
                    stop = 1;
                    reason = FLBP_ALL_CONVERGED;
                } else if (iters0 + n >= maxiter) {
                    stop = 1;
                } else if (over) {
                    stop = 2;
                }
            }
            if (stop) break;
        }

        // ---- the state back to global memory (the barrier above ended the last phase)
        if (!skip) {
            for (uint32_t j = wid; j < r.rows_f + r.rows_v; j += NW) {
                const bool fac = j < r.rows_f;
                const uint32_t it = res_item_of(fac ? j : j - r.rows_f, b, nb);
                if (it >= (fac ? n_f : n_v)) continue;
                const ResRow x = rows[j];
                const bool big = it < (fac ? nfb : nvb);
                const uint32_t n = big ? x.w : 32u * x.w, np = cluster_slots(big, x.w);
                const T *xs = reinterpret_cast<const T *>(sm + x.off);
                const uint32_t i0 = (fac ? f_index(it) : v_index(it)) + (big ? 0u : (uint32_t)lane);
                const bool in = big || (fac ? i0 >= J.f_lo && i0 < J.f_hi : i0 >= J.v_lo && i0 < J.v_hi);
                if (!in) continue;
                T *dst = fac ? const_cast<T *>(gvf) : const_cast<T *>(gfv);
                for (uint32_t k = lane; k < n; k += 32) dst[x.base + k] = xs[k];
                if (DAMP && !fac) {
                    const T *fd =
                        reinterpret_cast<const T *>(sm + x.off + np * (TW + 1) + cluster_prior_words(big, sizeof(T)));
                    for (uint32_t k = lane; k < n; k += 32) gfvd[x.base + k] = fd[k];
                }
            }
        }
        if (b == 0 && tid == 0 && !skip) {
            if (r.groups) {
                r.v.gstate[2 * G + J.group] = (int)(run0 + (long long)s);
                if (stop == 1) {
                    r.v.gstate[J.group] = 1;
                    r.v.gstate[3 * G + J.group] = reason;
                }
                r.gdiff[J.group] = maxdiff;
                if (stop == 2) *(volatile int *)&ctl->done = 1;  // the host stops relaunching
            } else {
                ctl->t = t0 + (long long)s;
                ctl->run_sweeps = run00 + (long long)s;
                ctl->t_start_ns = t_start;
                if (s) ctl->pscale = s_pscale;
                if (mode) {
                    ctl->maxdiff_bits = (unsigned long long)__double_as_longlong(maxdiff);
                    ctl->nonconv = nonconv;
                    ctl->maxdiff = maxdiff;
                    ctl->frac = frac;
                    ctl->node_frac_tol = node_frac_tol;
                    ctl->reason = reason;
                    if (stop) ctl->done = 1;
                }
            }
        }
        __syncthreads();  // the next job overwrites the shared memory just read
    }
}

}  // namespace flbp
