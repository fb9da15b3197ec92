// Persistent mixed-precision M2L over a work queue: the batched evaluate's M2L.
//
// A batch of plans (batch.cu) runs every plan's upward pass, then ONE launch of this
// kernel for the M2L of every plan, level and kernel family, then every plan's
// downward pass. Each work item is one target tile x one 128-row block of one
// (plan, level, family) M2L -- the unit one CTA of k_m2l_split computes -- and the
// items are queued by decreasing cost, so large levels start first and the small
// problems' few coarse tiles fill the tail. One CTA per SM stays resident and takes
// the next item with an atomic counter until the queue is empty: tensor memory is
// allocated, mbarriers initialised and registers split once per CTA, and the stage
// and accumulation-unit counters run on across items, so consecutive items keep the
// pipeline's barrier phases. The per-item arithmetic is k_m2l_split's (three FP16 plane
// products, FP32 units of 24 MMAs folded into FP64 sums held in registers), the call
// parameters (MixedCall) and the TMA tensor maps of every (plan, level, family) come
// from global memory. Every wait is bounded as in k_m2l_split; a timeout stops the
// CTA after the item, drains what it issued and frees tensor memory.
#include "hfmm_internal.cuh"
#include "m2l_common.cuh"
#include "mixed.cuh"

#include <algorithm>

namespace hfmm {

using namespace mxk;

namespace {

struct __align__(8) QueueCtl {
    uint64_t full[STAGES];
    uint64_t tfull[STAGES];
    uint64_t empty[STAGES];
    uint64_t acc_full[NACC];
    uint64_t acc_empty[NACC];
    uint64_t done;
    uint32_t tmem;
    int abort_flag;
    int item;                 // the item this CTA works on (-1: queue empty)
    int n_act;
    int tgt[BN];
    short act[M2L_ENTRIES + 1];
    short zidx[M2L_ENTRIES + 1];
    unsigned char used[M2L_ENTRIES + 1];
    short ztab[M2L_ENTRIES + 1];
    MixedCall c;              // the item's call parameters
};

// Start of an item, called by every thread of the CTA in the same order (four block
// barriers): the first fold warp takes the next item and copies its call parameters,
// the fold warps (which hold the most registers) load the tile's targets and find its
// active entries. Returns false, for every thread at once, when the queue is empty or
// the CTA has timed out. FOLDER: compiled for the fold warps, which do the work.
template <int R, bool FOLDER>
__device__ __forceinline__ bool next_item(QueueCtl& ctl, const MixedCall* __restrict__ calls,
                                          const M2LItem* __restrict__ items, int n_items, int* next,
                                          int warp, int lane, int tid) {
    constexpr int TT = BN / R;
    if (FOLDER && warp == FOLD_WARP0 && lane == 0) {
        const int it = ctl.abort_flag ? n_items : atomicAdd(next, 1);
        ctl.item = it < n_items ? it : -1;
        if (it < n_items) ctl.c = calls[items[it].call];
    }
    __syncthreads();
    if (ctl.item < 0) return false;
    const int ft = tid - FOLD_WARP0 * 32;   // 0..511 in the fold warps
    if (FOLDER) {
        const MixedCall& c = ctl.c;
        const int tile = items[ctl.item].tile;
        if (ft < TT) {
            int t = c.tile_tgt[(int64_t)tile * TT + ft];
            const int64_t lo = c.src_hi > 0 ? c.src_lo : 0, hi = c.src_hi > 0 ? c.src_hi : c.nb;
            if (t >= 0 && (t < lo || t >= hi)) {
                atomicOr(c.err, ERRF_BOUNDS);
                t = -1;
            }
            ctl.tgt[ft] = t;
        }
        for (int e = ft; e < M2L_ENTRIES; e += 32 * N_FOLD_WARPS) {
            ctl.used[e] = 0;
            ctl.ztab[e] = (short)(e < N_DISP ? c.disp_compact[e] : -1);
        }
    }
    __syncthreads();
    if (FOLDER) {
        const MixedCall& c = ctl.c;
        constexpr int BATCH = 4;
        constexpr int PAIRS = TT * M2L_ENTRIES;
        constexpr int NT = 32 * N_FOLD_WARPS;
        for (int i0 = ft; i0 < PAIRS; i0 += NT * BATCH) {
            int src[BATCH];
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const int i = i0 + u * NT;
                src[u] = -1;
                if (i < PAIRS) {
                    const int t = ctl.tgt[i / M2L_ENTRIES];
                    if (t >= 0) src[u] = __ldg(c.src_tab + (int64_t)t * M2L_ENTRIES + i % M2L_ENTRIES);
                }
            }
#pragma unroll
            for (int u = 0; u < BATCH; ++u)
                if (src[u] >= 0) ctl.used[(i0 + u * NT) % M2L_ENTRIES] = 1;
        }
    }
    __syncthreads();
    if (FOLDER && warp == FOLD_WARP0) {
        int base = 0;
        for (int e0 = 0; e0 < M2L_ENTRIES; e0 += 32) {
            int e = e0 + lane;
            const bool act = e < M2L_ENTRIES && ctl.used[e] && ctl.ztab[e] >= 0;
            unsigned bal = __ballot_sync(0xffffffffu, act);
            if (act) {
                const int slot = base + __popc(bal & ((1u << lane) - 1));
                ctl.act[slot] = (short)e;
                ctl.zidx[slot] = ctl.ztab[e];
            }
            base += __popc(bal);
        }
        if (lane == 0) ctl.n_act = base;
    }
    __syncthreads();
    return true;
}

template <int R>
__global__ void __launch_bounds__(THREADS, 1)
    k_m2l_queue(const MixedCall* __restrict__ calls, const MixedMaps* __restrict__ maps,
                const M2LItem* __restrict__ items, int n_items, int* next, uint64_t wait_ns_in,
                int starve) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* sm = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    QueueCtl& ctl = *reinterpret_cast<QueueCtl*>(sm + STAGES * STAGE_BYTES);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    volatile int* abort_flag = &ctl.abort_flag;
    const uint64_t wait_ns = wait_ns_in ? wait_ns_in : WAIT_NS;

    if (tid == 0) {
        ctl.abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&ctl.full[s]), 128);
            mbar_init(smem_u32(&ctl.tfull[s]), 1);
            mbar_init(smem_u32(&ctl.empty[s]), 1);
        }
        for (int b = 0; b < NACC; ++b) {
            mbar_init(smem_u32(&ctl.acc_full[b]), 1);
            mbar_init(smem_u32(&ctl.acc_empty[b]), N_FOLD_WARPS);
        }
        mbar_init(smem_u32(&ctl.done), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&ctl.tmem)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = ctl.tmem;
    if (warp < 4)
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REG_GATHER));
    else if (warp < FOLD_WARP0)
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REG_CTRL));
    else
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REG_FOLD));

    // Every role runs its own loop over the items; the loops meet at the same block
    // barriers (four in next_item, one at each item's end). q_total and u_total are the
    // stages and accumulation units this CTA has issued before the current item.
    int q_total = 0, u_total = 0;
    if (warp < 4) {
        // ---------------- B gathers (k_m2l_split's, for items that are not in grid mode). The
        // next entry's sources are looked up while the current one's chunks are copied.
        constexpr int RSTEP = 128 / CPR;
        const int ch = tid % CPR;
        const uint32_t soff0 = (uint32_t)((tid / CPR >> 3) * 8 * ROW_BYTES + (tid / CPR & 7) * ROW_BYTES +
                                          ((ch ^ (tid / CPR & 7)) << 4));   // rows RSTEP apart: the same swizzle
        static_assert(RSTEP % 8 == 0, "gather rows");
        int st = 0;
        uint32_t phase = 1;
        while (next_item<R, false>(ctl, calls, items, n_items, next, warp, lane, tid)) {
            const MixedCall& c = ctl.c;
            const int kch = (c.valid + BK - 1) / BK, n_act = ctl.n_act, nq = n_act * kch;
            if (!c.grid) {
                const int src_lo = c.src_hi > 0 ? (int)c.src_lo : 0, src_hi = (int)(c.src_hi > 0 ? c.src_hi : c.nb);
                const int ldk = c.ldk;
                const int32_t* src_tab = c.src_tab;
                const uint16_t* B = c.B + ch * 8;
                const int64_t b_plane = c.b_plane;
                int nsrc[CPR];
                auto look_up = [&](int ai) {
                    const int e = ctl.act[ai];
#pragma unroll
                    for (int i = 0; i < CPR; ++i) {
                        const int t = ctl.tgt[(tid / CPR + RSTEP * i) / R];
                        nsrc[i] = t >= 0 ? __ldg(src_tab + (int64_t)t * M2L_ENTRIES + e) : -1;
                    }
                };
                if (n_act > 0) look_up(0);
                bool ok = true;
                int qg = q_total;
                for (int ai = 0; ai < n_act && ok; ++ai) {
                    int goff[CPR];   // element offsets: the host keeps nb x R x ldk below 2^31
#pragma unroll
                    for (int i = 0; i < CPR; ++i) {
                        int s_ = nsrc[i];
                        if (s_ >= 0 && (s_ < src_lo || s_ >= src_hi)) {
                            atomicOr(c.err, ERRF_BOUNDS);
                            s_ = -1;
                        }
                        goff[i] = s_ >= 0 ? (s_ * R + (tid / CPR + RSTEP * i) % R) * ldk : -1;
                    }
                    if (ai + 1 < n_act) look_up(ai + 1);
                    for (int kc = 0; kc < kch; ++kc, ++qg) {
                        const int k0 = kc * BK;
                        if (!mbar_wait(smem_u32(&ctl.empty[st]), phase, abort_flag, wait_ns)) {
                            ok = false;
                            break;
                        }
                        const uint32_t sb = smem_u32(sm) + st * STAGE_BYTES + PLANES * TILE_BYTES + soff0;
                        const bool in = k0 + ch * 8 < ldk;
#pragma unroll
                        for (int i = 0; i < CPR; ++i) {
                            const bool okk = goff[i] >= 0 && in;
                            const uint16_t* g = okk ? B + goff[i] + k0 : c.B;
#pragma unroll
                            for (int pl = 0; pl < PLANES; ++pl)
                                cp_async16(sb + pl * TILE_BYTES + i * (RSTEP * ROW_BYTES), g + (okk ? pl * b_plane : 0), okk);
                        }
                        if (!(starve && qg == 0))   // (test: the CTA's first stage never fills)
                            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(
                                             smem_u32(&ctl.full[st]))
                                         : "memory");
                        if (++st == STAGES) {
                            st = 0;
                            phase ^= 1;
                        }
                    }
                }
                asm volatile("cp.async.wait_all;\n" ::: "memory");
            } else {   // the stages of a grid item pass by
                const int at = st + nq;
                phase ^= (uint32_t)(at / STAGES) & 1u;
                st = at % STAGES;
            }
            q_total += nq;
            __syncthreads();
        }
    } else if (warp >= FOLD_WARP0) {
        // ---------------- fold into FP64 sums in registers; store at each item's end
        const int quad = warp & 3;
        const int c_lo = ((warp - FOLD_WARP0) >> 2) * COLS_PER_FOLD_WARP;
        const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
        while (next_item<R, true>(ctl, calls, items, n_items, next, warp, lane, tid)) {
            const MixedCall& c = ctl.c;
            const int m0 = items[ctl.item].mblock * BM;
            const bool half = c.valid - m0 <= 64;
            const int kch = (c.valid + BK - 1) / BK, nq = ctl.n_act * kch;
            const int n_units = (nq + (1 << c.fold2) - 1) >> c.fold2;
            const int m = half ? m0 + quad * 16 + lane : m0 + quad * 32 + lane;
            const bool row_ok = half ? (lane < 16 && m < c.ldm) : (m0 + quad * 32 < c.ldm);
            double sum[COLS_PER_FOLD_WARP];
#pragma unroll
            for (int j = 0; j < COLS_PER_FOLD_WARP; ++j) sum[j] = 0.0;
            bool ok = true;
            for (int u = 0; u < n_units; ++u) {
                const int ug = u_total + u, b = ug & (NACC - 1);
                const bool got = mbar_wait(smem_u32(&ctl.acc_full[b]), (ug / NACC) & 1, abort_flag, wait_ns);
                if (!__all_sync(0xffffffffu, got)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t v[16];
                    tmem_ld16(lane_base + b * BN + c_lo + 16 * h, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 16; ++j) sum[16 * h + j] += (double)__uint_as_float(v[j]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&ctl.acc_empty[b]));
            }
            const bool aborted = !__all_sync(0xffffffffu, ok && !*abort_flag);
            if (aborted) {
                if (lane == 0) atomicOr(c.err, ERRF_TIMEOUT);
            } else if (row_ok) {
                double unscale[R];
#pragma unroll
                for (int r = 0; r < R; ++r) unscale[r] = 1.0 / (c.a_scale[0] * plane_scale(c.b_max[0][r]));
#pragma unroll
                for (int j = 0; j < COLS_PER_FOLD_WARP; ++j) {
                    const int n = c_lo + j;
                    const int t = ctl.tgt[n / R];
                    if (t >= 0) c.out[((int64_t)t * R + (n % R)) * c.ldm + m] = sum[j] * unscale[j % R];
                }
            }
            u_total += n_units;
            __syncthreads();
        }
    } else if (warp == 4) {
        // ---------------- A (and, in grid mode, B) tiles by TMA. One thread issues every stage's
        // copies, so what it computes a stage is on the pipeline's path: coordinates change
        // with the entry only, stage and phase are carried along.
        int last_q[STAGES];   // the last stage index loaded into each stage
#pragma unroll
        for (int st = 0; st < STAGES; ++st) last_q[st] = -1;
        int* err = nullptr;
        int st = 0;
        uint32_t phase = 1;   // of empty[st]: the first round finds every stage free
        while (next_item<R, false>(ctl, calls, items, n_items, next, warp, lane, tid)) {
            const MixedCall& c = ctl.c;
            const int kch = (c.valid + BK - 1) / BK, n_act = ctl.n_act, nq = n_act * kch;
            if (lane == 0) {
                err = c.err;
                const int tile = items[ctl.item].tile, m0 = items[ctl.item].mblock * BM;
                const MixedMaps* mp = maps + items[ctl.item].call;
                // the maps were written through the generic proxy (a host copy): make them
                // visible to the tensor-map proxy before their use in this item
#pragma unroll
                for (int pl = 0; pl < PLANES; ++pl)
                    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(&mp->a[0][pl])
                                 : "memory");
                const bool grid = c.grid;
                int ox = 0, oy = 0, oz = 0;
                if (grid) {
#pragma unroll
                    for (int pl = 0; pl < PLANES; ++pl)
                        asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(&mp->b[0][pl])
                                     : "memory");
                    ox = c.tile_org[3 * (int64_t)tile] + 3;
                    oy = c.tile_org[3 * (int64_t)tile + 1] + 3;
                    oz = c.tile_org[3 * (int64_t)tile + 2] + 3;
                }
                const uint32_t bytes = (grid ? 2 : 1) * PLANES * TILE_BYTES;
                int qg = q_total;
                bool ok = true;
                for (int ai = 0; ai < n_act && ok; ++ai) {
                    const int e = ctl.act[ai], z = ctl.zidx[ai];
                    const int sx = ox - e / 49, sy = oy - (e / 7) % 7, sz = oz - e % 7;   // sources at target - d
                    for (int k0 = 0; k0 < kch * BK; k0 += BK, ++qg) {
                        const uint32_t fb = smem_u32(&ctl.tfull[st]);
                        const uint32_t sa = smem_u32(sm) + st * STAGE_BYTES;
                        if (!mbar_wait(smem_u32(&ctl.empty[st]), phase, abort_flag, wait_ns)) {
                            ok = false;
                            break;
                        }
                        if (!(grid && starve && qg == 0)) {   // (test: stage 0 never fills)
                            mbar_arrive_tx(fb, bytes);
#pragma unroll
                            for (int pl = 0; pl < PLANES; ++pl)
                                tma_load_3d(sa + pl * TILE_BYTES, &mp->a[0][pl], k0, m0, z, fb);
                            if (grid) {
#pragma unroll
                                for (int pl = 0; pl < PLANES; ++pl)
                                    tma_load_5d(sa + (PLANES + pl) * TILE_BYTES, &mp->b[0][pl], k0, 0, sz, sy, sx, fb);
                            }
#pragma unroll
                            for (int j = 0; j < STAGES; ++j)
                                if (j == st) last_q[j] = qg;
                        }
                        if (++st == STAGES) {
                            st = 0;
                            phase ^= 1;
                        }
                    }
                }
            }
            q_total += nq;
            __syncthreads();
        }
        if (lane == 0) {   // drain: every stage's last load has landed
            bool drained = true;
#pragma unroll
            for (int j = 0; j < STAGES; ++j)
                if (last_q[j] >= 0) drained &= mbar_drain(smem_u32(&ctl.tfull[j]), (last_q[j] / STAGES) & 1, wait_ns);
            if (!drained && err) atomicOr(err, ERRF_TIMEOUT);
        }
    } else if (warp == 5) {
        // ---------------- MMA issue (one thread; stage, phase and buffer are carried along)
        bool issued = false;
        int* err = nullptr;
        // The gather warps complete a stage's full barrier only for items that are not in
        // grid mode, so its phase is not the stage counter's: bit st holds the parity of
        // full[st]'s next phase.
        uint32_t full_par = 0, phase = 0;
        int st = 0;
        const uint64_t desc0 = sw_desc(smem_u32(sm));
        while (next_item<R, false>(ctl, calls, items, n_items, next, warp, lane, tid)) {
            const MixedCall& c = ctl.c;
            const int kch = (c.valid + BK - 1) / BK, nq = ctl.n_act * kch;
            const int n_units = (nq + (1 << c.fold2) - 1) >> c.fold2;
            if (lane == 0) {
                err = c.err;
                const int m0 = items[ctl.item].mblock * BM;
                const uint32_t idesc = c.valid - m0 <= 64 ? IDESC64 : IDESC;
                const int last = (1 << c.fold2) - 1;
                // k-steps of an entry's last chunk
                const int tail = (c.valid - (kch - 1) * BK + KSTEP - 1) / KSTEP;
                const bool grid = c.grid;
                int ug = u_total, uq = 0, kc = 0;
                for (int q = 0; q < nq; ++q) {
                    const int b = ug & (NACC - 1);
                    if (uq == 0 && ug >= NACC) {
                        if (!mbar_wait(smem_u32(&ctl.acc_empty[b]), ((ug / NACC) & 1) ^ 1, abort_flag, wait_ns))
                            break;
                        asm volatile("tcgen05.fence::after_thread_sync;");
                    }
                    if (!grid) {
                        if (!mbar_wait(smem_u32(&ctl.full[st]), (full_par >> st) & 1u, abort_flag, wait_ns))
                            break;
                        full_par ^= 1u << st;
                    }
                    if (!mbar_wait(smem_u32(&ctl.tfull[st]), phase, abort_flag, wait_ns)) break;
                    if (!grid) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    const uint64_t d = desc0 + (uint64_t)(st * (STAGE_BYTES >> 4));
                    ++kc;
                    stage_mmas(tmem + b * BN, d, kc < kch ? BK / KSTEP : tail, idesc, uq == 0);
                    if (kc == kch) kc = 0;
                    issued = true;
                    umma_commit(smem_u32(&ctl.empty[st]));
                    if (uq == last || q == nq - 1) umma_commit(smem_u32(&ctl.acc_full[b]));
                    if (uq == last) {
                        uq = 0;
                        ++ug;
                    } else {
                        ++uq;
                    }
                    if (++st == STAGES) {
                        st = 0;
                        phase ^= 1;
                    }
                }
            }
            q_total += nq;
            u_total += n_units;
            __syncthreads();
        }
        if (lane == 0 && issued) {   // drain: the commit tracks every MMA issued
            umma_commit(smem_u32(&ctl.done));
            if (!mbar_drain(smem_u32(&ctl.done), 0, wait_ns) && err) atomicOr(err, ERRF_TIMEOUT);
        }
    } else {
        // warps 6 and 7: no role; they keep the item barriers' count
        while (next_item<R, false>(ctl, calls, items, n_items, next, warp, lane, tid)) __syncthreads();
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 5) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

void check_queue_split() {
    static int verdict = 0;
    if (verdict == 0) {
        int fits = 1;
        for (int r = 0; r < 2; ++r) {
            cudaFuncAttributes a{};
            HFMM_CUDA(cudaFuncGetAttributes(&a, r ? (const void*)k_m2l_queue<2> : (const void*)k_m2l_queue<1>));
            const long need = 128L * REG_GATHER + 128L * REG_CTRL + 32L * N_FOLD_WARPS * REG_FOLD;
            if ((long)a.numRegs * THREADS < need || a.maxThreadsPerBlock < THREADS) fits = 0;
        }
        verdict = fits ? 1 : -1;
    }
    if (verdict < 0)
        throw Error{HFMM_ERR_STATE, "m2l_queue: the warp roles' register split exceeds the launch's registers"};
}

}  // namespace

size_t m2l_queue_smem() { return (size_t)STAGES * STAGE_BYTES + sizeof(QueueCtl) + 1024; }

void m2l_queue(const MixedCall* calls, const MixedMaps* maps, const M2LItem* items, int n_items,
               int* next, int R, int n_ctas, cudaStream_t s, int starve) {
    if (n_items <= 0) return;
    check_queue_split();
    const size_t smem = m2l_queue_smem();
    const int grid = std::max(1, std::min(n_ctas, n_items));
    HFMM_CUDA(cudaMemsetAsync(next, 0, sizeof(int), s));
    if (R == 1) {
        HFMM_CUDA(cudaFuncSetAttribute(k_m2l_queue<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        HFMM_LAUNCH(k_m2l_queue<1>, grid, THREADS, smem, s, calls, maps, items, n_items, next, g_m2l_wait_ns.load(),
                    starve);
    } else {
        HFMM_CUDA(cudaFuncSetAttribute(k_m2l_queue<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        HFMM_LAUNCH(k_m2l_queue<2>, grid, THREADS, smem, s, calls, maps, items, n_items, next, g_m2l_wait_ns.load(),
                    starve);
    }
}

}  // namespace hfmm
