// Kernels of the sequential schedules (updates=SEQFIX / TOPO).
//
// A sweep runs the schedule's batches in order, each in two phases:
//   seq_factor_kernel  one warp per factor of the batch: the v->f message of
//                      every slot from the current variable totals (the
//                      reference's calcMessageVFKernel, causal_bp_seq.cu:
//                      113-147), then every output of the factor into the
//                      staging array (the f->v math of the PARALL pass);
//   seq_apply_kernel   one thread per target edge of the batch: its new f->v
//                      message replaces the old one in its variable's total
//                      and +-inf counts (update_message, :34-83).
// The factor kernel reads only state as it was before the batch, which is
// what the reference's two kernels per batch see, and the targets of a batch
// have distinct variables, so the apply kernel has no conflicts. A factor's
// outputs to slots that are not targets of the batch are staged but not
// applied. seq_begin_kernel opens a sweep; seq_belief_kernel closes it with
// the beliefs, residuals and stop rules of the run loops.
//
// seq_sweep_block_kernel runs all batches of a sweep in one launch on one
// block of 32 warps: the phases of a batch are separated by block barriers.
// A batch is bound by latency, and on one SM there is little of it: the
// block's own stores and loads meet in its L1, staged outputs stay in shared
// memory, a warp evaluates four factors of up to eight body slots at once
// (eight lanes each), and the records of the next batch are loaded while
// this one is evaluated. Per batch (one B200, FP32): SEQFIX on 4,000 tuples
// (88 slots a batch) 5.4 us with two launches, 3.7 us on a cluster of eight
// blocks that exchanged everything through L2, 2.35 us here; TOPO on 1,000
// tuples 4.8, 3.3 and 1.55 us.
#pragma once

#include "kernels.cuh"

namespace flbp {

struct SeqArgs {
    const uint4 *irec;      // per item: first device slot, degree, kind | staging offset in its batch << 8, factor
    const uint32_t *tvar;   // per target: its variable
    const uint32_t *tst;    // per target: staging offset of its message in its batch
    const uint2 *bo;        // per batch: (first item, first target), n_batches + 1
    const uint32_t *foff;   // per factor: first device slot (F + 1)
    const uint32_t *var;    // per device slot: internal variable
    const uint8_t *kind;    // per factor
    const void *cst;        // per factor: constant message, T
    const void *pq;         // per factor: p, q, T
    const uint32_t *items;  // factors of the batches
    const uint32_t *tgt;    // target device slots of the batches
    const uint32_t *iota;   // iota[s] = s: output positions of a factor's slots
    void *fv;               // per device slot: current f->v message, T
    void *vf;               // per device slot: v->f message of the current batch, T
    void *nw;               // per device slot: staged f->v message, T
    double *S;              // per internal variable: sum of its finite f->v messages
    int2 *cnt;              // per internal variable: (+inf count, -inf count)
};

// Programmatic dependent launch: a kernel lets the next one in the stream
// launch at once and waits (in hardware) for the previous one to finish and
// its memory to be visible before it reads any state. Both are no-ops for a
// kernel launched without the attribute.
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

constexpr int kSeqWarps = 8;           // warps per block of the factor kernel
template <typename T>
constexpr int kSeqBlockWarps = sizeof(T) == 4 ? 32 : 16;  // warps of the one-block sweep kernel (registers of the item code)
constexpr int kSegLanes = 8;           // lanes per factor of a packed item group
constexpr size_t kSeqStageMax = 96 * 1024;  // staged messages of a batch in shared memory at most (the rest is L1)

static __global__ void seq_begin_kernel(Ctl *ctl) {
    pdl_enter();
    if (*(volatile int *)&ctl->done) return;
    unsigned long long now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if (ctl->run_sweeps == 0) ctl->t_start_ns = now;
    ctl->t += 1;
    ctl->run_sweeps += 1;
    ctl->maxdiff_bits = 0ull;
    ctl->nonconv = 0ull;
    ctl->arrive = 0u;
}

// A factor with more than kBigFactorBody body slots, one warp: a log-sigmoid
// sum of the body in FP64 with a count of -inf terms, then every slot removes
// its own term (the warp form of factor_block_huge). vb[0] is the head's
// v->f message, vb[1 + k] body slot k's; outputs go to out[0] (head) and
// out[1 + k].
template <typename T>
__device__ void seq_factor_huge(const T *vb, uint32_t nbody, uint8_t kind, T p, T q, int lane, T *out) {
    const T s = (kind & KIND_OR) ? T(-1) : T(1);
    const T inf = Num<T>::inf();
    double L = 0.0;
    int nz = 0;
    for (uint32_t k = 1 + lane; k <= nbody; k += 32) {
        const T ls = log_sigmoid<T>(s * vb[k]);
        if (ls == -inf) nz++;
        else L += (double)ls;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        L += __shfl_xor_sync(0xffffffffu, L, o);
        nz += __shfl_xor_sync(0xffffffffu, nz, o);
    }
    if ((kind & HEAD_MASK) == HEAD_FREE && lane == 0) out[0] = s * head_out<T>(nz ? -inf : (T)L, p, q, Num<T>::log(p));
    const BodyDen<T> D = body_den<T>(s * head_effective<T>(kind, vb[0]), p, q);
    for (uint32_t k = 1 + lane; k <= nbody; k += 32) {
        const T ls = log_sigmoid<T>(s * vb[k]);
        const bool z = (ls == -inf);
        const T lo = (nz - (int)z) ? -inf : (T)(z ? L : L - (double)ls);
        out[k] = s * body_out<T>(lo, p, q, D);
    }
}

// Item `it` of the batches' item list, one whole warp: every v->f message of
// the factor from the current totals, then all its outputs into the staging
// array.
template <typename T>
__device__ __forceinline__ void seq_factor_item(const SeqArgs &a, uint32_t it, int lane) {
    const uint4 r = a.irec[it];  // first slot, degree, kind, factor
    const uint32_t s0 = r.x, deg = r.y, f = r.w;
    const uint8_t kind = (uint8_t)r.z;  // the staging offset above it is the one-block kernel's
    T *nw = reinterpret_cast<T *>(a.nw);
    const T c = reinterpret_cast<const T *>(a.cst)[f];
    if (kind & kSeqConst) {  // singleton, or an AND/OR factor reduced to its head
        if (lane == 0) nw[s0] = c;
        return;
    }
    const T *fv = reinterpret_cast<const T *>(a.fv);
    T *vf = reinterpret_cast<T *>(a.vf);
    for (uint32_t k = lane; k < deg; k += 32) {
        const uint32_t s = s0 + k, v = a.var[s];
        const T x = __ldcg(fv + s);
        const int2 n = __ldcg(a.cnt + v);
        vf[s] = excl_msg<T>(__ldcg(a.S + v), n.x, n.y, x);
    }
    __syncwarp();  // orders the v->f stores before the other lanes' loads
    const T *pq = reinterpret_cast<const T *>(a.pq);
    const T p = pq[2 * f], q = pq[2 * f + 1];
    if (deg - 1 <= kBigFactorBody) factor_tile_item<T>(vf + s0, a.iota + s0, deg, kind, p, q, lane,
                                                              GlobalOut<T>{nw});
    else seq_factor_huge<T>(vf + s0, deg - 1, kind, p, q, lane, nw + s0);
    if ((kind & HEAD_MASK) != HEAD_FREE && lane == 0) nw[s0] = c;  // a clamped head's constant
}

// Target k of the batches' target list: its staged message replaces the old
// one in its variable's total and counts.
template <typename T, bool DAMP>
__device__ __forceinline__ void seq_apply_one(const SeqArgs &a, uint32_t k, T d) {
    const uint32_t s = a.tgt[k], v = a.tvar[k];
    T *fv = reinterpret_cast<T *>(a.fv);
    const T old = __ldcg(fv + s);
    T x = __ldcg(reinterpret_cast<const T *>(a.nw) + s);
    double S = __ldcg(a.S + v);
    int2 n = __ldcg(a.cnt + v);
    if (DAMP) x = damp_mix<T>(x, old, d);
    const T inf = Num<T>::inf();
    if (old == inf) n.x--;
    else if (old == -inf) n.y--;
    else S -= (double)old;
    if (x == inf) n.x++;
    else if (x == -inf) n.y++;
    else S += (double)x;
    a.S[v] = S;
    a.cnt[v] = n;
    fv[s] = x;
}

// Items [i0, i1) of the batches' item list: one warp per factor.
template <typename T>
__global__ void __launch_bounds__(32 * kSeqWarps) seq_factor_kernel(SeqArgs a, uint32_t i0, uint32_t i1, Ctl *ctl) {
    pdl_enter();
    if (*(volatile int *)&ctl->done) return;
    const uint32_t it = i0 + blockIdx.x * kSeqWarps + (threadIdx.x >> 5);
    if (it >= i1) return;  // whole warps leave together
    seq_factor_item<T>(a, it, threadIdx.x & 31);
}

// Targets [t0, t1) of the batches' target list.
template <typename T, bool DAMP>
__global__ void seq_apply_kernel(SeqArgs a, uint32_t t0, uint32_t t1, T d, Ctl *ctl) {
    pdl_enter();
    if (*(volatile int *)&ctl->done) return;
    const uint32_t k = t0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= t1) return;
    seq_apply_one<T, DAMP>(a, k, d);
}

// One factor of at most WIDTH body slots on WIDTH lanes (sl: lane within
// them): x is the v->f message of body slot sl (in: there is one), vh the
// head's. The scans and the products around them are those of
// factor_tile_big<T, 1>, whose lanes past the body only ever combine with the
// identity pair, so the outputs are the same bits. All 32 lanes call it.
// out_b: the message to the lane's body slot; out_h: the head's.
template <typename T, int WIDTH>
__device__ __forceinline__ void factor_seg(T x, bool in, T vh, uint8_t kind, T p, T q, int sl, T &out_b, T &out_h) {
    const unsigned full = 0xffffffffu;
    const T sgn = (kind & KIND_OR) ? T(-1) : T(1);
    T sg = T(1), ta = T(0);
    if (in) sig_pair<T>(sgn * x, sg, ta);
    T fP = sg, fR = ta, bP = sg, bR = ta;
#pragma unroll
    for (int off = 1; off < WIDTH; off <<= 1) {
        const T oP = __shfl_up_sync(full, fP, off, WIDTH), oR = __shfl_up_sync(full, fR, off, WIDTH);
        if (sl >= off) {
            fR = fma(oP, fR, oR);
            fP = oP * fP;
        }
        const T dP = __shfl_down_sync(full, bP, off, WIDTH), dR = __shfl_down_sync(full, bR, off, WIDTH);
        if (sl + off < WIDTH) {
            bR = fma(bP, dR, bR);
            bP = bP * dP;
        }
    }
    const T P = __shfl_sync(full, fP, WIDTH - 1, WIDTH), R = __shfl_sync(full, fR, WIDTH - 1, WIDTH);
    T eP = __shfl_up_sync(full, fP, 1, WIDTH), eR = __shfl_up_sync(full, fR, 1, WIDTH);        // lanes before
    T xP = __shfl_down_sync(full, bP, 1, WIDTH), xR = __shfl_down_sync(full, bR, 1, WIDTH);    // lanes after
    if (sl == 0) eP = T(1), eR = T(0);
    if (sl == WIDTH - 1) xP = T(1), xR = T(0);
    T lP = T(0);
    if (__any_sync(full, q == T(0) && P < Num<T>::tiny())) {  // rare: log P as the sum of the body's log-sigmoids
        typedef AccOps<typename WideAcc<T>::type> O;
        typename WideAcc<T>::type l = O::zero();
        int nz = 0;
        if (in) {
            const T ls = log_sigmoid<T>(sgn * x);
            if (ls == -Num<T>::inf()) nz = 1;
            else O::add(l, ls);
        }
#pragma unroll
        for (int o = WIDTH / 2; o > 0; o >>= 1) {
            O::combine(l, O::shfl_xor(l, o));
            nz += __shfl_xor_sync(full, nz, o);
        }
        lP = nz ? -Num<T>::inf() : (T)O::value(l);
    }
    out_h = sgn * head_from_pair<T>(P, R, p, q, [&]() { return lP; });
    const BodyDen<T> D = body_den<T>(sgn * head_effective<T>(kind, vh), p, q);
    out_b = sgn * body_out_pr<T>(eP * xP, fma(eP, xR, eR), p, q, D);
}

// Schedule data, read once a sweep in order: not kept in L1, whose room the
// totals and messages need.
__device__ __forceinline__ uint32_t ld_pass(const uint32_t *p) {
    uint32_t x;
    asm("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(x) : "l"(p));
    return x;
}
__device__ __forceinline__ uint4 ld_pass(const uint4 *p) {
    uint4 x;
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
        : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w)
        : "l"(p));
    return x;
}
__device__ __forceinline__ float ld_pass(const float *p) {
    float x;
    asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(x) : "l"(p));
    return x;
}
__device__ __forceinline__ double ld_pass(const double *p) {
    double x;
    asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(x) : "l"(p));
    return x;
}

// What one lane needs of its item besides the totals: loaded a batch ahead.
template <typename T>
struct SeqRec {
    uint4 r;         // the item's record
    uint32_t v, vh;  // variables of the lane's body slot and of the head
    T p, q, c;
};

// One whole sweep (its opening included) on one block. Totals, counts and
// messages are only touched by this block, through its L1; stage: where the
// batch's outputs wait (shared memory, or global memory for batches of more
// slots than it holds).
template <typename T, bool DAMP>
__global__ void __launch_bounds__(32 * kSeqBlockWarps<T>, 1)
    seq_sweep_block_kernel(SeqArgs a, uint32_t n_batches, int stage_shared, T d, Ctl *ctl) {
    extern __shared__ __align__(16) unsigned char seq_sm[];
    if (*(volatile int *)&ctl->done) return;
    constexpr uint32_t NW = kSeqBlockWarps<T>, NT = 32 * NW;
    if (threadIdx.x == 0) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (ctl->run_sweeps == 0) ctl->t_start_ns = now;
        ctl->t += 1;
        ctl->run_sweeps += 1;
        ctl->maxdiff_bits = 0ull;
        ctl->nonconv = 0ull;
        ctl->arrive = 0u;
    }
    T *stage = stage_shared ? reinterpret_cast<T *>(seq_sm) : reinterpret_cast<T *>(a.nw);
    T *fv = reinterpret_cast<T *>(a.fv);
    const T *pqa = reinterpret_cast<const T *>(a.pq), *cst = reinterpret_cast<const T *>(a.cst);
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t sub = lane / kSegLanes, sl = lane % kSegLanes;
    constexpr uint32_t per = 32 / kSegLanes;  // items of a group
    auto load_item = [&](uint32_t it, uint32_t end) {
        SeqRec<T> x;
        x.r = it < end ? ld_pass(a.irec + it) : make_uint4(0u, 0u, kSeqConst, 0u);
        return x;
    };
    auto load_rest = [&](SeqRec<T> &x, bool valid) {  // what hangs on the record
        x.v = x.vh = 0u;
        x.p = x.q = x.c = T(0);
        if (!valid) return;
        x.vh = ld_pass(a.var + x.r.x);
        if (sl + 1 < x.r.y) x.v = ld_pass(a.var + x.r.x + 1 + sl);
        x.p = ld_pass(pqa + 2 * (size_t)x.r.w);
        x.q = ld_pass(pqa + 2 * (size_t)x.r.w + 1);
        x.c = ld_pass(cst + x.r.w);
    };
    uint2 lo = a.bo[0], hi = n_batches ? a.bo[1] : lo;
    SeqRec<T> nx = load_item(lo.x + per * wid + sub, hi.x);
    load_rest(nx, lo.x + per * wid + sub < hi.x);
    for (uint32_t b = 0; b < n_batches; b++) {
        const uint2 hi2 = b + 2 <= n_batches ? a.bo[b + 2] : hi;
        const uint32_t kt = lo.y + tid;  // the thread's first target
        uint32_t ts = 0, tv = 0, tst = 0;
        if (kt < hi.y) {
            ts = ld_pass(a.tgt + kt);
            tv = ld_pass(a.tvar + kt);
            tst = ld_pass(a.tst + kt);
        }
        SeqRec<T> cur = nx;
        const uint32_t nit = hi.x + per * wid + sub;
        nx = load_item(nit, hi2.x);
        for (uint32_t g = lo.x + per * wid; g < hi.x; g += per * NW) {
            const uint32_t it = g + sub;
            const bool valid = it < hi.x;
            if (g != lo.x + per * wid) {
                cur = load_item(it, hi.x);
                load_rest(cur, valid);
            }
            const uint32_t s0 = cur.r.x, deg = cur.r.y, st = cur.r.z >> 8;
            const uint8_t kind = (uint8_t)cur.r.z;
            const bool cons = (kind & kSeqConst) != 0;
            const bool narrow = deg <= kSegLanes + 1;
            {
                const bool act = valid && !cons && narrow, in = act && sl + 1 < deg;
                T m = T(0), mh = T(0);
                if (act) {
                    const T xh = fv[s0], x = in ? fv[s0 + 1 + sl] : T(0);
                    const double Sh = a.S[cur.vh], S = in ? a.S[cur.v] : 0.0;
                    const int2 nh = a.cnt[cur.vh], n = in ? a.cnt[cur.v] : make_int2(0, 0);
                    mh = excl_msg<T>(Sh, nh.x, nh.y, xh);
                    m = excl_msg<T>(S, n.x, n.y, x);
                }
                T ob, oh;
                factor_seg<T, kSegLanes>(m, in, mh, act ? kind : (uint8_t)0, cur.p, cur.q, (int)sl, ob, oh);
                if (in) stage[st + 1 + sl] = ob;
                if (valid && (cons || narrow) && sl == 0)  // a constant, a clamped head's constant, or the head's message
                    stage[st] = (cons || (kind & HEAD_MASK) != HEAD_FREE) ? cur.c : oh;
            }
            // wider factors of the group, a warp each
            for (uint32_t wide = __ballot_sync(0xffffffffu, valid && !cons && !narrow && sl == 0); wide;
                 wide &= wide - 1) {
                const int src = __ffs(wide) - 1;
                const uint32_t s = __shfl_sync(0xffffffffu, s0, src), dg = __shfl_sync(0xffffffffu, deg, src);
                const uint32_t so = __shfl_sync(0xffffffffu, st, src);
                const uint8_t kd = (uint8_t)__shfl_sync(0xffffffffu, (uint32_t)kind, src);
                const T p = __shfl_sync(0xffffffffu, cur.p, src), q = __shfl_sync(0xffffffffu, cur.q, src);
                const T c = __shfl_sync(0xffffffffu, cur.c, src);
                auto vf_of = [&](uint32_t k) {  // the v->f message of slot s + k
                    const uint32_t v = ld_pass(a.var + s + k);
                    const int2 n = a.cnt[v];
                    return excl_msg<T>(a.S[v], n.x, n.y, fv[s + k]);
                };
                if (dg <= 33) {
                    const bool in = lane + 1 < dg;
                    const T m = in ? vf_of(1 + lane) : T(0), mh = vf_of(0);
                    T ob, oh;
                    factor_seg<T, 32>(m, in, mh, kd, p, q, (int)lane, ob, oh);
                    if (in) stage[so + 1 + lane] = ob;
                    if (lane == 0) stage[so] = (kd & HEAD_MASK) != HEAD_FREE ? c : oh;
                } else {
                    T *vf = reinterpret_cast<T *>(a.vf);
                    for (uint32_t k = lane; k < dg; k += 32) vf[s + k] = vf_of(k);
                    __syncwarp();  // orders the v->f stores before the other lanes' loads
                    auto put = [&](uint32_t e, T o) { stage[so + (e - s)] = o; };
                    if (dg - 1 <= kBigFactorBody) factor_tile_item<T>(vf + s, a.iota + s, dg, kd, p, q, (int)lane, put);
                    else seq_factor_huge<T>(vf + s, dg - 1, kd, p, q, (int)lane, stage + so);
                    if ((kd & HEAD_MASK) != HEAD_FREE && lane == 0) stage[so] = c;
                    __syncwarp();
                }
            }
        }
        load_rest(nx, nit < hi2.x);
        __syncthreads();
        const T inf = Num<T>::inf();
        for (uint32_t k = kt; k < hi.y; k += NT) {  // seq_apply_one
            if (k != kt) {
                ts = ld_pass(a.tgt + k);
                tv = ld_pass(a.tvar + k);
                tst = ld_pass(a.tst + k);
            }
            const T old = fv[ts];
            T x = stage[tst];
            double S = a.S[tv];
            int2 n = a.cnt[tv];
            if (DAMP) x = damp_mix<T>(x, old, d);
            if (old == inf) n.x--;
            else if (old == -inf) n.y--;
            else S -= (double)old;
            if (x == inf) n.x++;
            else if (x == -inf) n.y++;
            else S += (double)x;
            a.S[tv] = S;
            a.cnt[tv] = n;
            fv[ts] = x;
        }
        __syncthreads();
        lo = hi;
        hi = hi2;
    }
}

// Beliefs of every internal variable from its total and counts, with the
// residual, history and stop rules of the run loop's mode (BMODE of
// var_finish: 1 tolerance loop, 2 low-pass loop, 3 beliefs only).
template <int BMODE>
__global__ void __launch_bounds__(256) seq_belief_kernel(VarArgs va, const double *S, const int2 *cnt, uint32_t V,
                                                         Ctl *ctl) {
    constexpr bool RESID = (BMODE == 1 || BMODE == 2);
    pdl_enter();
    if (BMODE != 3 && *(volatile int *)&ctl->done) return;
    const double tol = ctl->tol;
    double dmax = 0.0;
    unsigned long long c = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        const int2 n = cnt[v];
        const double dd = var_finish<BMODE>(va, v, S[v], n.x, n.y, tol, RESID ? va.belief[v] : 0.0, c);
        dmax = fmax(dmax, dd);
    }
    if (!RESID) return;
    __shared__ double s_max[8];
    __shared__ unsigned long long s_cnt[8];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    dmax = warp_max(dmax);
    c = warp_sum(c);
    if (lane == 0) {
        s_max[wid] = dmax;
        s_cnt[wid] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = 0.0;
        unsigned long long t = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) {
            m = fmax(m, s_max[i]);
            t += s_cnt[i];
        }
        atomicMax(&ctl->maxdiff_bits, (unsigned long long)__double_as_longlong(m));
        if (BMODE == 2) atomicAdd(&ctl->nonconv, t);
        __threadfence();
        s_last = (atomicAdd(&ctl->arrive, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (s_last && threadIdx.x == 0) {
        __threadfence();
        stop_rules(ctl);
    }
}

}  // namespace flbp
