// FP64 output-stationary gather-GEMM for the plain (float64) path.
//
// For a tile of target boxes t_1..t_T (same level; for M2L also the same octant)
// and one M-tile of the n_s surface rows it computes
//     out[t_j][r][m] (+)= scale[m] * sum_e sum_k A_e[m][k] * B_e[src(t_j, e)][r][k]
// with the accumulator kept on chip across every entry e, so no partial sum
// ever goes back to memory and the result is deterministic. One kernel serves
// the four dense contractions of the KIFMM evaluate:
//   M2M  (phases.py:163-171): e = child octant, A_e = M2M_K_lv[parent][e]
//   M2L  (phases.py:211-236): e = displacement (343 slots), A_e = M2L_K_lv[level][e];
//        plus L2L (phases.py:273-278): e = 343 + octant, A_e = L2L_K_lv[level-1][octant],
//        src = parent -- the L2L check potential is summed with the M2L one and
//        decoded once (the decode is linear)
//   decode (phases.py:21-34): A = U^T with scale d, then A = Vt^T.
// A is stored transposed (k-major, leading dimension ld, zero padded) so both
// operand tiles stream into shared memory with 16-byte cp.async copies.
//
// Tensor path: mma.sync.m16n8k4 f64 (DMMA). tcgen05 has no f64 kind, so this
// is the FP64 tensor path on sm_100a. CTA tile 64 (m) x 64 (n = targets x R), or 32 x 32 on
// small grids, k-chunk 16, 4 warps of 32 x 32 (16 x 16), three-stage cp.async pipeline with one barrier a chunk.
// An SM sub-partition takes 32 cycles per DMMA, so a chunk's 32 a warp are 1,024 cycles; what
// kept it from them were the instructions around (640 a chunk and warp: copy addresses and
// source lookups worked out anew every chunk, eight 8-byte fragment loads a step). Now the
// copy addresses are pointers that advance, looked up once an entry, and fragments are
// 16-byte loads: lane t of four takes k = 2t and 2t + 1 of eight as two steps' B values, and
// accumulator rows g and g + 8 are matrix rows 2g and 2g + 1 (the order of k and m within a
// tile is free), which the epilogue then stores as 16-byte pairs straight from registers.
// Small grids (coarse levels: a few dozen output tiles, each walking all its entries)
// are latency-bound, so there the entries are split into contiguous ranges, one CTA
// per range and output tile; each writes its partial tile to a scratch array and
// k_gemm_reduce adds the partials in range order before the usual epilogue, so the
// result does not depend on scheduling.
#include "hfmm_internal.cuh"

#include <algorithm>

namespace hfmm {

namespace {

constexpr int TM = 64, TN = 64, KC = 16, STAGES = 3;   // the tile of large grids
constexpr int TS = 32;                                  // and of small ones: 32 x 32
constexpr int BP = KC + 8;   // Bs[n][BP]: one column apart is 64 bytes mod 128
constexpr int MAX_ENTRIES = 352;
constexpr int SRC_ENTRIES = 8;   // entry counts whose tile sources are kept in shared memory

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    int sz = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b0) {
    asm volatile(
        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
        "{%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a0), "d"(a1), "d"(b0));
}

template <int T>
struct __align__(16) Smem {
    static constexpr int AP = T + 2;   // A[k][AP]: two k rows apart is 32 bytes mod 128
    double A[STAGES][KC][AP];
    double B[STAGES][T][BP];
    int src[T][SRC_ENTRIES + 1];
    int tgt[T];
    short act[MAX_ENTRIES];
    unsigned char used[MAX_ENTRIES];   // entry has a source for some target of the tile
    int n_act;
};

// scale, accumulation and store of one column's rows m, m + 1
__device__ __forceinline__ void store_pair(const GemmCall& c, double* out, const double* sc, int64_t row, int m,
                                           double v0, double v1) {
    if (sc) {
        v0 *= sc[m];
        v1 *= sc[m + 1];
    }
    double2* o = reinterpret_cast<double2*>(out + row * c.ldm + m);
    if (c.accumulate) {
        const double2 old = *o;
        v0 += old.x;
        v1 += old.y;
    }
    *o = make_double2(v0, v1);
}

// T: the square tile, 64 or 32 (four warps of T / 2 squared). A tile list has 64 columns a
// tile; with T = 32 two CTAs share one.
template <int R, int T>
__global__ void __launch_bounds__(128, 3) k_gemm_f64(GemmCall c, int* err) {
    constexpr int TT = T / R, AP = Smem<T>::AP, MI = T / 32, NI = T / 16;
    constexpr int ACH = T / 2, CPT = KC * ACH / 128;   // 16-byte copies: of an A row; of each operand a thread
    extern __shared__ __align__(16) char smem_raw[];
    Smem<T>& sm = *reinterpret_cast<Smem<T>*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int S = c.n_split > 1 ? c.n_split : 1;
    const int tile = blockIdx.x, m0 = blockIdx.y * T, fam = blockIdx.z / S, split = blockIdx.z % S;
    const int e_lo = (int)((int64_t)split * c.n_entries / S);
    const int e_hi = (int)((int64_t)(split + 1) * c.n_entries / S);
    const double* const* A = c.A + (int64_t)fam * c.a_fam_stride;
    const double* B0 = c.B0 + (int64_t)fam * c.fam_stride;
    const double* B1 = c.B1 ? c.B1 + (int64_t)fam * c.fam_stride : nullptr;
    double* out = c.out + (int64_t)fam * c.fam_stride;
    const bool keep = c.src_tab && c.n_entries <= SRC_ENTRIES;

    if (tid < TT) {
        int t = c.tile_tgt[(int64_t)tile * TT + tid];
        if (t >= c.nb) {
            atomicOr(err, ERRF_BOUNDS);
            t = -1;
        }
        sm.tgt[tid] = t;
    }
    if (tid == 0) sm.n_act = 0;
    for (int e = tid; e < c.n_entries; e += 128) sm.used[e] = c.src_tab ? 0 : 1;
    __syncthreads();
    // active entries: A present and at least one target of the tile has a source. Every
    // thread tests (target, entry) pairs, the loads of a batch independent of each other
    if (c.src_tab) {
        constexpr int BATCH = 8;
        const int pairs = TT * c.n_entries;
        for (int i0 = tid; i0 < pairs; i0 += 128 * BATCH) {
            int src[BATCH];
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const int i = i0 + u * 128;
                src[u] = -1;
                if (i < pairs) {
                    const int t = sm.tgt[i / c.n_entries];
                    if (t >= 0) src[u] = __ldg(c.src_tab + (int64_t)t * c.src_ld + i % c.n_entries);
                }
            }
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const int i = i0 + u * 128;
                if (i >= pairs) break;
                if (src[u] >= c.nb) {
                    atomicOr(err, ERRF_BOUNDS);
                    src[u] = -1;
                }
                if (src[u] >= 0) sm.used[i % c.n_entries] = 1;
                if (keep) sm.src[i / c.n_entries][i % c.n_entries] = src[u];
            }
        }
        __syncthreads();
    }
    if (warp == 0) {
        int base = 0;
        for (int e0 = 0; e0 < c.n_entries; e0 += 32) {
            int e = e0 + lane;
            const bool act = e >= e_lo && e < e_hi && A[e] != nullptr && sm.used[e];
            unsigned bal = __ballot_sync(0xffffffffu, act);
            if (act) sm.act[base + __popc(bal & ((1u << lane) - 1))] = (short)e;
            base += __popc(bal);
        }
        if (lane == 0) sm.n_act = base;
    }
    __syncthreads();
    const int k_len = c.k_valid > 0 ? c.k_valid : c.ldk;   // rows of A^T that can be nonzero
    const int kch = (k_len + KC - 1) / KC;
    const int nq = sm.n_act * kch;

    // the next chunk to copy: its entry, its k, and this thread's source addresses there
    int l_e = 0, l_k = 0;
    const double* ap = nullptr;
    const double* bp[CPT];
    unsigned bok = 0;
    const int a_row = tid / ACH, a_col = tid % ACH * 2;   // rows 128 / ACH apart
    const bool aok = m0 + a_col < c.ldm;
    auto load = [&](int buf) {
        if (l_k == 0) {   // a new entry
            const int e = sm.act[l_e++];
            ap = A[e] + (int64_t)a_row * c.ldm + (aok ? m0 + a_col : 0);
            const double* Bsel = (e >= c.b_split && B1) ? B1 : B0;
            bok = 0;
#pragma unroll
            for (int i = 0; i < CPT; ++i) {   // B: T columns x 16 doubles, 8 threads a column
                const int col = (tid >> 3) + 16 * i, j = col / R, r = col % R;
                const int t = sm.tgt[j];
                int s = -1;
                if (keep) s = sm.src[j][e];
                else if (t >= 0) s = c.src_tab ? c.src_tab[(int64_t)t * c.src_ld + e] : t;
                const bool ok = s >= 0 && s < c.nb;
                if (ok) bok |= 1u << i;
                bp[i] = ok ? Bsel + ((int64_t)s * R + r) * c.ldk + (tid & 7) * 2 : B0;
            }
        }
#pragma unroll
        for (int i = 0; i < CPT; ++i)   // A: 16 rows x T doubles
            cp_async16(&sm.A[buf][a_row + 128 / ACH * i][a_col], ap + (int64_t)(128 / ACH * i) * c.ldm, aok);
#pragma unroll
        for (int i = 0; i < CPT; ++i)
            cp_async16(&sm.B[buf][(tid >> 3) + 16 * i][(tid & 7) * 2], bp[i], bok >> i & 1);
        ap += (int64_t)KC * c.ldm;
#pragma unroll
        for (int i = 0; i < CPT; ++i)
            if (bok >> i & 1) bp[i] += KC;
        l_k = l_k + 1 == kch ? 0 : l_k + 1;
    };

    double acc[MI][NI][4];
#pragma unroll
    for (int a = 0; a < MI; ++a)
#pragma unroll
        for (int b = 0; b < NI; ++b)
#pragma unroll
            for (int d = 0; d < 4; ++d) acc[a][b][d] = 0.0;

    const int wm = (warp & 1) * (T / 2), wn = (warp >> 1) * (T / 2);
    const int g = lane >> 2, t4 = lane & 3;
    // 16-row halves of the warp's tile with rows that can be nonzero
    const int m_rows = min(MI, max(0, ((c.ldm == c.ld ? c.n_s : c.ldm) - (m0 + wm) + 15) / 16));
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) {
        if (i < nq) load(i);
        cp_async_commit();
    }
    int buf = 0, kq = 0;
    for (int q = 0; q < nq; ++q) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();   // chunk q is there, and every warp is done with chunk q - 1
        if (q + STAGES - 1 < nq) load(buf == 0 ? STAGES - 1 : buf - 1);
        cp_async_commit();
        const int k8n = min(KC, k_len - kq * KC);   // the entry's last chunk may be partial
        kq = kq + 1 == kch ? 0 : kq + 1;
        if (m_rows > 0) {
            const double* As = &sm.A[buf][2 * t4][wm + 2 * g];
            const double* Bs = &sm.B[buf][wn + g][2 * t4];
#pragma unroll
            for (int kk = 0; kk < KC; kk += 8) {
                if (kk >= k8n) break;
                double2 b[NI];
#pragma unroll
                for (int ni = 0; ni < NI; ++ni) b[ni] = *reinterpret_cast<const double2*>(Bs + ni * 8 * BP + kk);
#pragma unroll
                for (int mi = 0; mi < MI; ++mi) {
                    if (mi >= m_rows) break;
                    const double2 a0 = *reinterpret_cast<const double2*>(As + kk * AP + mi * 16);
                    const double2 a1 = *reinterpret_cast<const double2*>(As + (kk + 1) * AP + mi * 16);
#pragma unroll
                    for (int ni = 0; ni < NI; ++ni) dmma(acc[mi][ni], a0.x, a0.y, b[ni].x);
#pragma unroll
                    for (int ni = 0; ni < NI; ++ni) dmma(acc[mi][ni], a1.x, a1.y, b[ni].y);
                }
            }
        }
        buf = buf + 1 == STAGES ? 0 : buf + 1;
    }
    cp_async_wait<0>();
    // epilogue from registers: rows m, m + 1 of columns n and n + 1, 128 bytes a column
    double* part = S > 1 ? c.part + ((int64_t)(blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * TN * TM
                         : nullptr;
    const double* sc = (fam == 1 && c.scale_f1) ? c.scale_f1 : c.scale;
    if (c.most) {   // (one-entry calls without scale or split: what is stored is acc)
#pragma unroll
        for (int r = 0; r < R; ++r) {   // acc's odd values are odd columns'
            double top = 0.0;
            bool odd = false;   // infinities and NaN: the largest bits there are
#pragma unroll
            for (int i = r; i < MI * NI * 4; i += R) {
                const double v = fabs((&acc[0][0][0])[i]);
                odd = odd || !(v <= 1.7976931348623157e308);
                top = fmax(top, v);
            }
            unsigned long long bits = odd ? 0x7ff0000000000000ull : (unsigned long long)__double_as_longlong(top);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long v = __shfl_xor_sync(0xffffffffu, bits, o);
                bits = v > bits ? v : bits;
            }
            if (lane == 0 && bits) atomicMax(c.most + r, bits);
        }
    }
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < NI; ++ni)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int ml = wm + mi * 16 + 2 * g, col = wn + ni * 8 + 2 * t4 + h, m = m0 + ml;
                const double v0 = acc[mi][ni][h], v1 = acc[mi][ni][2 + h];
                if (S > 1) {   // a split: the partial tile goes to the scratch, k_gemm_reduce finishes it
                    *reinterpret_cast<double2*>(part + col * TM + ml) = make_double2(v0, v1);
                    continue;
                }
                const int t = sm.tgt[col / R];
                if (t < 0 || m >= c.ldm) continue;
                store_pair(c, out, sc, (int64_t)t * R + col % R, m, v0, v1);
            }
}

// The split GEMM's epilogue: per output tile, the n_split partial tiles added in
// entry-range order, then the scale, accumulation and store of k_gemm_f64. RED_COLS columns
// of a tile per CTA: a coarse level has 10 to 50 tiles, and a CTA a tile took 15 to 24 us.
constexpr int RED_COLS = 8;
template <int R>
__global__ void __launch_bounds__(128) k_gemm_reduce(GemmCall c, int* err) {
    constexpr int TT = TN / R, PARTS = TN / RED_COLS;
    const int tid = threadIdx.x;
    const int tile = blockIdx.x, m0 = blockIdx.y * TM, fam = blockIdx.z / PARTS, S = c.n_split;
    double* out = c.out + (int64_t)fam * c.fam_stride;
    const double* sc = (fam == 1 && c.scale_f1) ? c.scale_f1 : c.scale;
    const int64_t tile_of = (int64_t)gridDim.y * gridDim.x * TN * TM;   // doubles between ranges
    const double* part = c.part + (int64_t)fam * S * tile_of + ((int64_t)blockIdx.y * gridDim.x + tile) * TN * TM;
#pragma unroll
    for (int q = 0; q < RED_COLS * (TM / 2) / 128; ++q) {
        const int idx = tid + q * 128;
        const int col = blockIdx.z % PARTS * RED_COLS + idx / (TM / 2), mm = (idx % (TM / 2)) * 2;
        const int t = c.tile_tgt[(int64_t)tile * TT + col / R], m = m0 + mm;
        if (t >= c.nb) {
            atomicOr(err, ERRF_BOUNDS);
            continue;
        }
        if (t < 0 || m >= c.ldm) continue;
        double v0 = 0.0, v1 = 0.0;
        const double* src = part + col * TM + mm;
#pragma unroll 4
        for (int sp = 0; sp < S; ++sp) {
            const double2 v = *reinterpret_cast<const double2*>(src + sp * tile_of);
            v0 += v.x;
            v1 += v.y;
        }
        store_pair(c, out, sc, (int64_t)t * R + col % R, m, v0, v1);
    }
}

}  // namespace

int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0, v = 0;
        HFMM_CUDA(cudaGetDevice(&dev));
        HFMM_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
        n = v > 0 ? v : 148;
    }
    return n;
}

void gemm_f64(const GemmCall& call, int* d_err, cudaStream_t s) {
    if (call.ntiles == 0) return;
    GemmCall c = call;
    if (!c.ldk) c.ldk = c.ld;
    if (!c.ldm) c.ldm = c.ld;
    if (c.ldk % KC != 0 || c.ldm % KC != 0)
        throw Error{HFMM_ERR_STATE, "gemm_f64: ld must be a multiple of 16"};
    if (c.k_valid > c.ldk) throw Error{HFMM_ERR_STATE, "gemm_f64: k_valid beyond ldk"};
    if (c.n_entries > MAX_ENTRIES) throw Error{HFMM_ERR_STATE, "gemm_f64: too many entries"};
    if (c.R != 1 && c.R != 2) throw Error{HFMM_ERR_ARG, "gemm_f64: R must be 1 or 2"};
    dim3 grid(c.ntiles, (c.ldm + TM - 1) / TM, c.n_fam);
    const int64_t ctas = (int64_t)grid.x * grid.y * grid.z;
    const int sms = sm_count();
    if (c.most && (c.scale || c.accumulate || c.n_entries != 1))
        throw Error{HFMM_ERR_STATE, "gemm_f64: largest magnitude of a plain one-entry call only"};
    // Under six CTAs an SM, calls of one entry a tile take 32 x 32 tiles: four times the CTAs,
    // each with a quarter of the serial chain, five an SM instead of three. All GEMMs of
    // 20,000 points p = 8 / p = 12: 351 / 848 us with 64 x 64 tiles only, 274 / 775 with the
    // line at one CTA an SM, 259 / 767 at two, 253 / 711 at four and above (real 1e5 p = 6:
    // 453, 381, 382, 352). On every size, operands read twice as often cost: 1e6 points
    // 6.83 to 7.38 ms. Calls of several entries keep 64 x 64 and the split below (p = 12:
    // 853 with small tiles there too against 767).
    if ((c.n_entries == 1 || c.one_entry) && ctas < 6 * sms) {
        c.n_split = 1;
        grid.x *= 2;
        grid.y = (c.ldm + TS - 1) / TS;
        auto kern = c.R == 1 ? k_gemm_f64<1, TS> : k_gemm_f64<2, TS>;
        HFMM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem<TS>)));
        HFMM_LAUNCH(kern, grid, 128, sizeof(Smem<TS>), s, c, d_err);
        return;
    }
    // entry splits when the grid gives the SMs fewer than four CTAs each (a CTA of 128
    // threads hides little latency on its own): up to about four per SM
    int S = 1;
    if (c.part && c.n_entries > 1 && !c.one_entry && ctas < 4 * sms) {
        S = (int)std::min<int64_t>({(int64_t)c.n_entries, 16, (4 * sms + ctas - 1) / ctas});
        while (S > 1 && ctas * S * TN * TM > c.part_cap) --S;
    }
    c.n_split = S;
    grid.z *= S;
    auto kern = c.R == 1 ? k_gemm_f64<1, TM> : k_gemm_f64<2, TM>;
    HFMM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem<TM>)));
    HFMM_LAUNCH(kern, grid, 128, sizeof(Smem<TM>), s, c, d_err);
    if (S > 1) {
        grid.z = grid.z / S * (TN / RED_COLS);
        if (c.R == 1) HFMM_LAUNCH(k_gemm_reduce<1>, grid, 128, 0, s, c, d_err);
        else HFMM_LAUNCH(k_gemm_reduce<2>, grid, 128, 0, s, c, d_err);
    }
}

}  // namespace hfmm
