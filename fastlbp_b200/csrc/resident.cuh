// The resident run kernel: all sweeps of a run in one cooperative launch.
//
// What it is for: a sweep of a graph that fits on the chip takes a few
// microseconds of work, and two launches per sweep cost more than that. Here
// one wave of co-resident blocks stays on the GPU for the whole run. Every
// block owns a fixed set of items (sliced-ELL groups and large items, dealt
// in turn over the blocks, widest first) of both passes and keeps what never
// changes about them - scatter positions, degrees, kinds, (p, q), priors,
// graph ids - in shared memory; only the messages move, through L2. A sweep
// is factor phase, grid barrier, variable phase, grid barrier; the residual
// is reduced on the way into the second barrier, and every block evaluates
// the run's stop rule from the same numbers, so that all leave together.
//
// Items are evaluated by the functions of the pass kernels (factor_reg,
// factor_tile_item, factor_block_huge, excl_msg, var_finish), in the same
// order per item, so a run gives the bits of the staged and direct forms.
//
// Memory: messages written by other blocks are read with ld.global.cg after
// a barrier whose arrival releases and whose wait acquires at GPU scope.
// Beliefs, damped messages and the low-pass history of an item are only ever
// touched by the thread that owns it.
//
// What bounds it: latency. Per sweep and phase one L2 round trip for the
// messages, one item per warp, and a grid barrier of about 1.1 us (release
// fence, arrival, poll). Against the staged passes replayed from CUDA graphs
// (FP32 tolerance runs, one B200): 15.9 -> 9.1-9.7 us per sweep at 16 k
// device slots, 18.3 -> 11.1 at 158 k, 24.8 -> 14 at 396 k; and a new engine
// captures no graphs (its first run at 16 k slots: 1.57 -> 0.45 ms).
//
// All waits are bounded: a barrier that does not open within ~2 s records
// FLBP_ERR_TIMEOUT and the block returns (no asynchronous copies are ever in
// flight). The launch is cooperative, so all blocks are resident and the
// barrier cannot wait for a block that has not started.
#pragma once

#include "kernels.cuh"

namespace flbp {

constexpr int kResThreads = kConsumers;   // 16 warps: the huge-item paths synchronise all consumer threads
constexpr uint32_t kResMaxRows = 512;     // items of both passes together per block with cached constants

template <typename T>
struct ResArgs {
    FactorArgs f;
    VarArgs v;
    T *vf, *fv, *fvd;
    T d;
    Ctl *ctl;
    uint32_t cap;          // sweeps of this launch at most
    int final_beliefs;     // fixed runs: the last sweep also writes the beliefs
    uint32_t rows_f, rows_v;  // items per block of each pass (the last row may be short)
    // The first huge_blocks blocks take the factors too large for a tile and
    // no other factors (0: there are none): a block that had one beside its
    // full share of the others ended the phase late. 25.75 -> 22.75 us per
    // sweep at 842 k slots with fan-ins up to 4,096.
    uint32_t huge_blocks;
    // Runs that keep states (gradients): sweep s reads v0 (s = 0) or vseg +
    // s vstride, writes its f->v messages to fseg + s fstride and its v->f
    // messages to vseg + (s + 1) vstride, the last sweep to vlast, or, when
    // that is null, no v->f messages. Without states all sweeps use vf and fv.
    int states = 0;
    const T *v0 = nullptr;
    T *vseg = nullptr, *fseg = nullptr, *vlast = nullptr;
    uint64_t vstride = 0, fstride = 0;
};

// Shared-memory words of one cached item: positions of its W columns (a large
// item: its slots, rounded up), then one word per lane of degree and kind and
// the lanes' (p, q) (factors), or the lanes' priors (variables), then the
// lanes' graphs in a batched solve.
__host__ __device__ __forceinline__ uint32_t res_item_words(bool factor, bool big, uint32_t w, uint32_t tsize,
                                                            bool batch) {
    const uint32_t pos = big ? (w + 31u) & ~31u : 32u * w;
    const uint32_t cst = factor ? 32u + 2u * 32u * (tsize / 4) : 32u * (tsize == 4 ? 2u : 4u);
    return pos + cst + (batch ? 32u : 0u);
}

// Item of row j of block b: items are dealt over the blocks back and forth
// (row 0 forwards, row 1 backwards, ...), which evens out the decreasing widths.
__host__ __device__ __forceinline__ uint32_t res_item_of(uint32_t j, uint32_t b, uint32_t nb) {
    return j * nb + ((j & 1u) ? nb - 1u - b : b);
}

struct ResRow {
    uint32_t base, w, off;  // first slot (entry); width or degree; first shared-memory word
};

// Arrival and bounded wait of one thread; false on timeout.
__device__ __forceinline__ bool res_arrive_wait(unsigned int *arrive, unsigned int target) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrive) : "memory");
    auto opened = [&]() {
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrive) : "memory");
        return (int)(v - target) >= 0;
    };
    if (opened()) return true;
    const long long t0 = clock64();
    for (uint32_t i = 1;; i++) {
        if (opened()) return true;
        if ((i & 15u) == 0 && clock64() - t0 > kWaitCycles) return false;
    }
}

// The same at the end of a sweep, on the slot's end word, to which a block
// adds 1, kResMoved and kResTimeUp as they apply. What the stop rule needs of
// the other blocks is in the word that is polled, so that no further load
// follows the barrier; releases and acquire are 32-bit accesses of the one
// word, and order the residuals and messages of all blocks.
__device__ __forceinline__ bool res_end_wait(unsigned int *arrive, unsigned int nb, unsigned int add,
                                             unsigned int &word) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(arrive), "r"(add) : "memory");
    auto opened = [&]() {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(word) : "l"(arrive) : "memory");
        return (word & (kResMoved - 1u)) == nb;
    };
    if (opened()) return true;
    const long long t0 = clock64();
    for (uint32_t i = 1;; i++) {
        if (opened()) return true;
        if ((i & 15u) == 0 && clock64() - t0 > kWaitCycles) return false;
    }
}

// Widths share two instances of the group code, up to 8 and up to 16 columns:
// a run's code has to stay in the instruction caches, which one instance per
// width (fine where thousands of warps run the same width) does not. Columns
// beyond the group's width are not loaded, and no item has a slot there.
constexpr int kResNarrow = 8;

// One sliced-ELL factor group of at most W columns: all messages first.
template <typename T, int W, bool CACHE>
__device__ __forceinline__ void res_factor_group(uint32_t w, const T *vf, uint32_t base, const uint32_t *ps, int deg,
                                                 uint8_t kind, T p, T q, int lane, T *__restrict__ fv) {
    T x[W];
#pragma unroll
    for (int k = 0; k < W; k++) x[k] = (uint32_t)k < w ? __ldcg(vf + base + 32u * k + lane) : T(0);
    if (CACHE) {
        if (deg > 0)
            factor_reg<T, W>([&](int k) { return x[k]; }, [&](int k) { return ps[32 * k + lane]; }, deg, kind, p, q,
                             GlobalOut<T>{fv});
    } else {
        uint32_t pr[W];
#pragma unroll
        for (int k = 0; k < W; k++) pr[k] = (uint32_t)k < w ? __ldg(ps + 32 * k + lane) : kSentinel;
        if (deg > 0) factor_reg<T, W>([&](int k) { return x[k]; }, [&](int k) { return pr[k]; }, deg, kind, p, q,
                                     GlobalOut<T>{fv});
    }
}

template <typename T, bool CACHE>
__device__ __forceinline__ void res_factor_group_w(uint32_t w, const T *vf, uint32_t base, const uint32_t *ps, int deg,
                                                   uint8_t kind, T p, T q, int lane, T *__restrict__ fv) {
    if (w <= (uint32_t)kResNarrow) res_factor_group<T, kResNarrow, CACHE>(w, vf, base, ps, deg, kind, p, q, lane, fv);
    else res_factor_group<T, kSellFactorDegree, CACHE>(w, vf, base, ps, deg, kind, p, q, lane, fv);
}

// One sliced-ELL variable group of at most W columns (lane = variable): sum
// and counts in S, npos, nneg, messages sent.
template <typename T, int W, bool DAMP, bool CACHE, typename A>
__device__ __forceinline__ void res_var_group(uint32_t w, const T *fv, T *__restrict__ vf, T *fvd, T d, uint32_t base,
                                              bool live, const uint32_t *ent, int lane, A &S,
                                              int &npos, int &nneg) {
    T x[W];
    T xo[DAMP ? W : 1];
    uint32_t en[!CACHE ? W : 1];
#pragma unroll
    for (int k = 0; k < W; k++) x[k] = (uint32_t)k < w ? __ldcg(fv + base + 32u * k + lane) : T(0);
    if (DAMP) {
#pragma unroll
        for (int k = 0; k < W; k++) xo[k] = (uint32_t)k < w ? fvd[base + 32u * k + lane] : T(0);
    }
    if (!CACHE) {
#pragma unroll
        for (int k = 0; k < W; k++) en[k] = (uint32_t)k < w ? __ldg(ent + 32 * k + lane) : kSentinel;
    }
    if (!live) return;
    var_lane_sum<T, W, DAMP>(w, x, xo, d, S, npos, nneg);
    if (DAMP) {
#pragma unroll
        for (int k = 0; k < W; k++)
            if ((uint32_t)k < w) fvd[base + 32u * k + lane] = x[k];
    }
    var_lane_send<T, W>(w, x, [&](int k) { return CACHE ? ent[32 * k + lane] : en[k]; }, S, npos, nneg,
                        GlobalOut<T>{vf});
}

// The whole run. CACHE: the block's items' constants in shared memory (else
// read from L2 every sweep).
template <typename T, bool DAMP, bool CACHE>
__global__ void __launch_bounds__(kResThreads, sizeof(T) == 4 ? 2 : 1) resident_kernel(ResArgs<T> r) {
    extern __shared__ __align__(128) uint32_t sm[];
    __shared__ typename WideAcc<T>::type s_l[kConsumerWarps];
    __shared__ int s_a[kConsumerWarps], s_b[kConsumerWarps];
    __shared__ double s_max[kConsumerWarps];
    __shared__ unsigned long long s_cnt[kConsumerWarps];
    __shared__ double s_pscale;
    __shared__ int s_stop, s_open;  // s_stop: 1 finished, 2 a wait gave up
    __shared__ uint32_t s_done[kGroupWords], s_moved[kGroupWords];
    Ctl *ctl = r.ctl;
    ResSync *rs = &ctl->rs;
    if (*(volatile int *)&ctl->done) return;  // the same for every block: only earlier launches have written it
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t nb = gridDim.x, b = blockIdx.x;
    const bool batch = r.v.v_graph != nullptr;
    const uint32_t G = batch ? r.v.n_graphs : 0u, gwords = (G + 31) / 32;
    const VarArgs &va = r.v;
    const uint32_t nfb = r.f.nf_big - r.f.nf_huge, nvb = va.nv_big - va.nv_huge;
    const uint32_t n_f = nfb + r.f.n_fgroups, n_v = nvb + va.n_vgroups;
    const uint32_t psz = sizeof(T) == 4 ? 2 : 4;  // words of a prior
    ResRow *rows = reinterpret_cast<ResRow *>(sm);
    const T *pqg = reinterpret_cast<const T *>(r.f.f_pq);

    // ---- constants of the block's items
    auto f_row = [&](uint32_t it) -> ResRow {
        if (it < nfb) return ResRow{r.f.fb_off[r.f.nf_huge + it], r.f.fb_deg[r.f.nf_huge + it], 0u};
        const uint32_t g = r.f.n_fgroups - 1 - (it - nfb), b0 = r.f.fg_base[g];
        return ResRow{b0, (r.f.fg_base[g + 1] - b0) >> 5, 0u};
    };
    auto v_row = [&](uint32_t it) -> ResRow {
        if (it < nvb) return ResRow{va.vb_off[va.nv_huge + it], va.vb_deg[va.nv_huge + it], 0u};
        const uint32_t g = va.n_vgroups - 1 - (it - nvb), b0 = va.vg_base[g];
        return ResRow{b0, (va.vg_base[g + 1] - b0) >> 5, 0u};
    };
    const uint32_t hb = r.huge_blocks;
    auto f_item = [&](uint32_t j) { return b < hb ? ~0u : res_item_of(j, b - hb, nb - hb); };
    if (CACHE) {
        for (uint32_t j = tid; j < r.rows_f + r.rows_v; j += kResThreads) {
            const bool fac = j < r.rows_f;
            const uint32_t it = fac ? f_item(j) : res_item_of(j - r.rows_f, b, nb);
            ResRow x{0u, 0u, 0u};
            if (it < (fac ? n_f : n_v)) {
                x = fac ? f_row(it) : v_row(it);
                x.off = res_item_words(fac, it < (fac ? nfb : nvb), x.w, sizeof(T), batch);
            }
            rows[j] = x;
        }
        __syncthreads();
        if (tid == 0) {  // sizes to offsets, behind the table
            uint32_t at = (3u * (r.rows_f + r.rows_v) + 31u) & ~31u;
            for (uint32_t j = 0; j < r.rows_f + r.rows_v; j++) {
                const uint32_t n = rows[j].off;
                rows[j].off = at;
                at += n;
            }
        }
        __syncthreads();
        for (uint32_t j = wid; j < r.rows_f; j += kConsumerWarps) {
            const uint32_t it = f_item(j);
            if (it >= n_f) break;
            const ResRow x = rows[j];
            const bool big = it < nfb;
            const uint32_t np = big ? x.w : 32u * x.w, npad = big ? (x.w + 31u) & ~31u : 32u * x.w;
            for (uint32_t k = lane; k < np; k += 32) sm[x.off + k] = r.f.f_pos[x.base + k];
            uint32_t *meta = sm + x.off + npad;
            T *pq = reinterpret_cast<T *>(meta + 32);
            const uint32_t fi = big ? r.f.nf_sell + r.f.nf_huge + it : 32u * (r.f.n_fgroups - 1 - (it - nfb)) + lane;
            if (!big || lane == 0) {
                const bool in = big || fi < r.f.nf_sell;
                meta[lane] = in ? (uint32_t)r.f.f_kind[fi] << 8 | (big ? 0u : (uint32_t)r.f.f_deg[fi]) : 0u;
                pq[2 * lane] = in ? pqg[2 * (size_t)fi] : T(0);
                pq[2 * lane + 1] = in ? pqg[2 * (size_t)fi + 1] : T(0);
                if (batch) meta[32 + 64 * (sizeof(T) / 4) + lane] = in ? r.f.f_graph[fi] : 0u;
            }
        }
        for (uint32_t j = wid; j < r.rows_v; j += kConsumerWarps) {
            const uint32_t it = res_item_of(j, b, nb);
            if (it >= n_v) break;
            const ResRow x = rows[r.rows_f + j];
            const bool big = it < nvb;
            const uint32_t np = big ? x.w : 32u * x.w, npad = big ? (x.w + 31u) & ~31u : 32u * x.w;
            for (uint32_t k = lane; k < np; k += 32) sm[x.off + k] = va.v_ent[x.base + k];
            const uint32_t v = big ? va.nv_sell + va.nv_huge + it : 32u * (va.n_vgroups - 1 - (it - nvb)) + lane;
            const bool in = big ? lane == 0 : v < va.nv_sell;
            uint32_t *cst = sm + x.off + npad;
            if (in) {
                for (uint32_t k = 0; k < psz; k++)
                    cst[psz * lane + k] = reinterpret_cast<const uint32_t *>(va.prior)[(size_t)psz * v + k];
                if (batch) cst[32 * psz + lane] = va.v_graph[v];
            }
        }
        // every warp reads only what it wrote itself
        __syncwarp();
    }

    // ---- run state
    const int mode = ctl->mode;
    const double tol = ctl->tol, damping = ctl->damping;
    const long long t0 = ctl->t, run0 = ctl->run_sweeps, iters0 = ctl->iters0, maxiter = ctl->maxiter;
    const long long min_iters = ctl->min_iters, max_iters = ctl->max_iters;
    const double maxtime_ns = ctl->maxtime_ns, n_vars = (double)ctl->n_vars;
    double node_frac_tol = ctl->node_frac_tol, frac = ctl->frac, maxdiff = ctl->maxdiff;
    int reason = ctl->reason;
    unsigned long long t_start = ctl->t_start_ns, maxdiff_bits = 0, nonconv = 0;
    if (run0 == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_start));
    for (uint32_t w = tid; w < gwords; w += kResThreads) {
        uint32_t bits = 0;
        for (uint32_t k = 0; k < 32; k++) {
            const uint32_t g = 32 * w + k;
            if (g >= G || va.gstate[g] != 0) bits |= 1u << k;
        }
        s_done[w] = bits;
    }
    if (tid == 0) s_stop = 0;
    __syncthreads();
    auto stopped = [&](uint32_t g) { return ((s_done[g >> 5] >> (g & 31)) & 1u) != 0; };
    uint32_t s = 0;
    unsigned int target = 0;
    for (; s < r.cap; s++) {
        const uint32_t slot = s % 3u, nslot = (s + 1u) % 3u;
        // ---- factor phase
        if (tid == 0)
            s_pscale = (damping == 0.0) ? 1.0 : 1.0 - pow(damping, (double)(t0 + (long long)s + 1));
        if (b == 0) {  // the next sweep's slots
            if (tid == 0) {
                rs->end[nslot].maxdiff = 0ull;
                rs->end[nslot].arrive = 0u;
                rs->nonconv[nslot] = 0ull;
            }
            for (uint32_t w = tid; w < gwords; w += kResThreads) rs->moved[nslot][w] = 0u;
        }
        for (uint32_t w = tid; w < gwords; w += kResThreads) s_moved[w] = 0u;
        const T *vf = !r.states ? r.vf : s == 0 ? r.v0 : r.vseg + s * r.vstride;
        T *fv = !r.states ? r.fv : r.fseg + s * r.fstride;
        for (uint32_t h = b; b < hb && h < r.f.nf_huge; h += hb) {
            if (batch && stopped(r.f.f_graph[r.f.nf_sell + h])) continue;
            factor_block_huge<T>(r.f, h, tid, CgPtr<T>{vf}, fv, s_l, s_a);
        }
        for (uint32_t j = wid; j < r.rows_f; j += kConsumerWarps) {
            const uint32_t it = f_item(j);
            if (it >= n_f) break;
            const ResRow x = CACHE ? rows[j] : f_row(it);
            if (it < nfb) {
                const uint32_t fi = r.f.nf_sell + r.f.nf_huge + it, npad = (x.w + 31u) & ~31u;
                const uint32_t *meta = sm + x.off + npad;
                if (batch && stopped(CACHE ? meta[32 + 64 * (sizeof(T) / 4)] : r.f.f_graph[fi])) continue;
                const T *pq = CACHE ? reinterpret_cast<const T *>(meta + 32) : pqg + 2 * (size_t)fi;
                factor_tile_item<T>(CgPtr<T>{vf + x.base}, CACHE ? sm + x.off : r.f.f_pos + x.base, x.w,
                                    CACHE ? (uint8_t)(meta[0] >> 8) : r.f.f_kind[fi], pq[0], pq[1], lane,
                                    GlobalOut<T>{fv});
            } else {
                const uint32_t fi = 32u * (r.f.n_fgroups - 1 - (it - nfb)) + lane;
                int deg;
                uint8_t kind;
                T p, q;
                uint32_t g = 0;
                if (CACHE) {
                    const uint32_t *meta = sm + x.off + 32u * x.w;
                    const T *pq = reinterpret_cast<const T *>(meta + 32);
                    deg = (int)(meta[lane] & 0xffu);
                    kind = (uint8_t)(meta[lane] >> 8);
                    p = pq[2 * lane];
                    q = pq[2 * lane + 1];
                    if (batch) g = meta[32 + 64 * (sizeof(T) / 4) + lane];
                } else {  // per-item arrays are padded to whole groups
                    deg = r.f.f_deg[fi];
                    kind = r.f.f_kind[fi];
                    p = pqg[2 * (size_t)fi];
                    q = pqg[2 * (size_t)fi + 1];
                    if (batch) g = r.f.f_graph[fi];
                }
                if (batch) {
                    if (stopped(g)) deg = 0;
                    if (!__any_sync(0xffffffffu, deg > 0)) continue;
                }
                res_factor_group_w<T, CACHE>(x.w, vf, x.base, CACHE ? sm + x.off : r.f.f_pos + x.base, deg, kind, p, q,
                                             lane, fv);
            }
        }
        const bool last = s + 1 == r.cap;
        T *vout = !r.states ? r.vf : last ? r.vlast : r.vseg + (s + 1) * r.vstride;
        if (!vout) {  // the last sweep's f->v messages end the run
            s++;
            break;
        }
        target += nb;
        __syncthreads();
        if (tid == 0 && !res_arrive_wait(&rs->arrive, target)) s_stop = 2;
        __syncthreads();
        if (s_stop) break;

        // ---- variable phase
        const int bm = mode == 3 ? 1 : mode != 0 ? mode : (last && r.final_beliefs) ? 3 : 0;
        const double pscale = s_pscale;
        double dmax = 0.0;
        unsigned long long cnt = 0;
        for (uint32_t h = b; h < va.nv_huge; h += nb) {
            const uint32_t g = batch ? va.v_graph[va.nv_sell + h] : 0u;
            if (batch && stopped(g)) continue;
            double dd = 0.0;
#define FLBP_HUGE(M) \
    var_block_huge<T, M, true, DAMP, true>(va, h, tid, fv, vout, r.fvd, r.d, pscale, tol, cnt, s_l, s_a, s_b)
            if (bm == 0) dd = FLBP_HUGE(0);
            else if (bm == 1) dd = FLBP_HUGE(1);
            else if (bm == 2) dd = FLBP_HUGE(2);
            else dd = FLBP_HUGE(3);
#undef FLBP_HUGE
            dmax = fmax(dmax, dd);
            if (G && dd > tol) atomicOr(&s_moved[g >> 5], 1u << (g & 31));
        }
        for (uint32_t j = wid; j < r.rows_v; j += kConsumerWarps) {
            const uint32_t it = res_item_of(j, b, nb);
            if (it >= n_v) break;
            T *fvd = r.fvd;
            const ResRow x = CACHE ? rows[r.rows_f + j] : v_row(it);
            const uint32_t *ent = CACHE ? sm + x.off : va.v_ent + x.base;
            const bool big = it < nvb;
            const uint32_t grp = va.n_vgroups - 1 - (it - nvb);
            const uint32_t v = big ? va.nv_sell + va.nv_huge + it : 32u * grp + lane;
            const uint32_t *cst = sm + x.off + (big ? (x.w + 31u) & ~31u : 32u * x.w);  // cached priors, then graphs
            const void *prior = CACHE ? (const void *)cst : va.prior;
            const uint32_t pidx = CACHE ? (big ? 0u : (uint32_t)lane) : v;
            const bool real = big ? lane == 0 : v < va.nv_sell;
            uint32_t g = 0;
            bool live = true;
            if (batch) {
                g = CACHE ? cst[32 * psz + (big ? 0 : lane)] : (big || real) ? va.v_graph[v] : 0u;
                live = (big || real) && !stopped(g);
                if (!__any_sync(0xffffffffu, live)) continue;
            }
            const double bold = (real && (bm == 1 || bm == 2)) ? va.belief[v] : 0.0;
            double Sv;
            int npos = 0, nneg = 0;
            if (big) {
                typename WideAcc<T>::type S;
                const uint32_t k0 = x.base;
                auto in = [&](uint32_t k) { return __ldcg(fv + k0 + k); };  // the new message of entry k
                auto old = [&](uint32_t k) { return DAMP ? fvd[k0 + k] : T(0); };
                var_warp_sum<T, DAMP>(in, old, x.w, prior, pidx, r.d, pscale, lane, S, npos, nneg);
                var_warp_send<T, DAMP, true>(in, old, [&](uint32_t k) { return ent[k]; }, DAMP ? fvd + k0 : nullptr,
                                             x.w, r.d, lane, S, npos, nneg, GlobalOut<T>{vout});
                Sv = AccOps<typename WideAcc<T>::type>::value(S);
            } else {
                typedef typename NarrowAcc<T>::type A;
                A S = AccOps<A>::zero();
                if (real) decode_prior<T>(prior, pidx, pscale, S, npos, nneg);
                if (x.w <= (uint32_t)kResNarrow)
                    res_var_group<T, kResNarrow, DAMP, CACHE>(x.w, fv, vout, fvd, r.d, x.base, live, ent, lane, S,
                                                              npos, nneg);
                else
                    res_var_group<T, kSellVarDegree, DAMP, CACHE>(x.w, fv, vout, fvd, r.d, x.base, live, ent, lane,
                                                                  S, npos, nneg);
                Sv = AccOps<A>::value(S);
            }
            if (bm && real && live) {
                double dd = 0.0;
                if (bm == 1) dd = var_finish<1>(va, v, Sv, npos, nneg, tol, bold, cnt);
                else if (bm == 2) dd = var_finish<2>(va, v, Sv, npos, nneg, tol, bold, cnt);
                else var_finish<3>(va, v, Sv, npos, nneg, tol, bold, cnt);
                dmax = fmax(dmax, dd);
                if (G && dd > tol) {
                    const uint32_t bit = 1u << (g & 31);
                    if (!(*(volatile uint32_t *)&s_moved[g >> 5] & bit)) atomicOr(&s_moved[g >> 5], bit);
                }
            }
        }
        if (mode == 0 && last) {  // nothing follows
            s++;
            break;
        }

        // ---- residual, stop rule
        if (mode) {
            dmax = warp_max(dmax);
            cnt = mode == 2 ? warp_sum(cnt) : 0ull;
            if (lane == 0) {
                s_max[wid] = dmax;
                s_cnt[wid] = cnt;
            }
        }
        __syncthreads();
        for (uint32_t w = tid; w < gwords; w += kResThreads)
            if (s_moved[w]) atomicOr(&rs->moved[slot][w], s_moved[w]);
        if (gwords) __syncthreads();
        if (wid == 0) {
            unsigned int add = 1u;
            if (mode) {
                double m = warp_max(lane < kConsumerWarps ? s_max[lane] : 0.0);
                unsigned long long c = 0;
                if (mode == 2) c = warp_sum(lane < kConsumerWarps ? s_cnt[lane] : 0ull);
                if (lane == 0) {
                    if (m > 0.0) atomicMax(&rs->end[slot].maxdiff, (unsigned long long)__double_as_longlong(m));
                    if (c) atomicAdd(&rs->nonconv[slot], c);
                    if (m > tol) add += kResMoved;
                    if (b == 0) {
                        unsigned long long now;
                        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
                        const double elapsed = (double)(now - t_start);
                        if (mode == 2 ? elapsed > maxtime_ns : elapsed >= maxtime_ns) add += kResTimeUp;
                    }
                }
            }
            unsigned int word = 0;
            if (lane == 0 && !res_end_wait(&rs->end[slot].arrive, nb, add, word)) {
                s_stop = 2;
            } else if (lane == 0 && mode) {
                const bool over = (word & kResTimeUp) != 0, moved = (word & (kResTimeUp - kResMoved)) != 0;
                const long long n = run0 + (long long)s + 1;
                if (mode == 1) {  // the rules of stop_rules
                    if (!(iters0 + n < maxiter && moved && !over)) {
                        s_stop = 1;
                        reason = moved ? FLBP_DIVERGED : FLBP_ALL_CONVERGED;
                    }
                } else if (mode == 2) {
                    maxdiff = __longlong_as_double((long long)__ldcg(&rs->end[slot].maxdiff));
                    nonconv = __ldcg(&rs->nonconv[slot]);
                    frac = (double)nonconv / n_vars;
                    if (n >= min_iters) node_frac_tol = (double)(n - min_iters) / (double)(max_iters - min_iters);
                    if (maxdiff <= tol) {
                        s_stop = 1;
                        reason = FLBP_ALL_CONVERGED;
                    } else if (n > min_iters && frac < node_frac_tol) {
                        s_stop = 1;
                        reason = FLBP_BIG_FRAC_CONVERGED;
                    } else if (n > max_iters || over) {
                        s_stop = 1;
                        reason = FLBP_DIVERGED;
                    }
                } else {
                    s_open = 0;
                    if (over) {
                        s_stop = 1;
                        reason = FLBP_DIVERGED;
                    }
                }
            }
        }
        __syncthreads();
        if (s_stop == 2) break;
        if (mode == 3) {  // the rule of batch_stop_rules, the same in every block
            const long long n = run0 + (long long)s + 1;
            int open = 0;
            for (uint32_t w = tid; w < gwords; w += kResThreads) {
                const uint32_t live = ~s_done[w], moved = __ldcg(&rs->moved[slot][w]);
                const uint32_t conv = live & ~moved, stop = (iters0 + n >= maxiter) ? live : conv;
                if (b == 0) {
                    for (uint32_t bits = live; bits; bits &= bits - 1) {
                        const uint32_t g = 32 * w + __ffs(bits) - 1, bit = bits & (0u - bits);
                        va.gstate[2 * G + g] = (int)n;
                        if (stop & bit) {
                            va.gstate[g] = 1;
                            va.gstate[3 * G + g] = (conv & bit) ? FLBP_ALL_CONVERGED : FLBP_DIVERGED;
                        }
                    }
                }
                s_done[w] |= stop;
                open += __popc(live & ~stop);
            }
            if (open) atomicAdd(&s_open, open);
            __syncthreads();
            if (s_open == 0) {  // all groups have stopped
                if (tid == 0) {
                    s_stop = 1;
                    reason = FLBP_ALL_CONVERGED;
                }
            }
            __syncthreads();
        }
        if (s_stop) {
            s++;
            break;
        }
    }
    if (s_stop == 2) {
        if (tid == 0) {
            record_timeout(ctl);
            *(volatile int *)&ctl->done = 1;
        }
        return;
    }
    if (b == 0 && tid == 0) {
        if (mode) {  // the last sweep's residual: its slot is cleared two sweeps later at the earliest
            maxdiff_bits = __ldcg(&rs->end[(s - 1u) % 3u].maxdiff);
            maxdiff = __longlong_as_double((long long)maxdiff_bits);
        }
        ctl->t = t0 + (long long)s;
        ctl->run_sweeps = run0 + (long long)s;
        ctl->t_start_ns = t_start;
        if (s) ctl->pscale = s_pscale;
        ctl->maxdiff_bits = maxdiff_bits;
        ctl->nonconv = nonconv;
        ctl->maxdiff = maxdiff;
        ctl->frac = frac;
        ctl->node_frac_tol = node_frac_tol;
        ctl->reason = reason;
        if (s_stop) ctl->done = 1;
    }
}

}  // namespace flbp
