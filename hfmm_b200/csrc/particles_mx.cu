// Mixed-precision near field (P2P; the role of the near field of near.py:48-312 on
// the mixed path): FP32 pair arithmetic, FP64 only where accuracy needs it.
//   * Separations come from FP32 hi/lo position pairs, (hi - hi') + (lo - lo'), so
//     they carry a relative error of eps32 however close the points are (box-local
//     FP32 coordinates gave 3.7e-6 on clustered clouds).
//   * The phase k r is an FP32 product: r itself carries eps32, and forming k r in
//     FP64 with an FP64 reduction before sincosf measured the same error.
//   * Sums run in FP32 over one source leaf and are combined in FP64, as is the
//     final per-target sum.
// P2M, P2L, L2P and M2P stay FP64 on the mixed path: their outputs feed or read
// the damped decodes, and FP32 there reached 2.7e-2 on the sin component.
// Same outputs and layouts as particles_f64.cu.
#include "hfmm_internal.cuh"
#include "particles.cuh"

namespace hfmm {

namespace {

constexpr int WARPS = 4;       // one target leaf per CTA, its source leaves dealt to the warps
constexpr int CHAIN = 128;     // sources per FP32 partial-sum chain

// Two FP32 values in one 64-bit register pair: each operation rounds both halves as the
// scalar one does, in one issue slot.
struct f2 {
    unsigned long long v;
};
__device__ __forceinline__ f2 pack2(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
    return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ f2 both(float a) { return pack2(a, a); }
__device__ __forceinline__ f2 neg2(f2 a) { return f2{a.v ^ 0x8000000080000000ull}; }

// sin and cos of two phases |x| <= 1.5 by their Taylor series about 0 (Horner
// form in x^2): the first omitted terms, x^13 / 13! and x^14 / 14!, stay below 3.2e-8
// and 3.3e-9 there, under the FP32 rounding of the pair arithmetic. Larger phases
// (big leaves at coarse levels, large k) take sincosf.
constexpr float SMALL_PHASE = 1.5f;
__device__ __forceinline__ void sincos_phase2(f2 x, f2* s, f2* c) {
    const float2 xx = unpack2(x);
    if (fabsf(xx.x) <= SMALL_PHASE && fabsf(xx.y) <= SMALL_PHASE) {
        const f2 x2 = mul2(x, x);
        f2 ps = both(-1.f / 39916800.f);
        f2 pc = both(1.f / 479001600.f);
        ps = fma2(ps, x2, both(1.f / 362880.f));
        pc = fma2(pc, x2, both(-1.f / 3628800.f));
        ps = fma2(ps, x2, both(-1.f / 5040.f));
        pc = fma2(pc, x2, both(1.f / 40320.f));
        ps = fma2(ps, x2, both(1.f / 120.f));
        pc = fma2(pc, x2, both(-1.f / 720.f));
        ps = fma2(ps, x2, both(-1.f / 6.f));
        pc = fma2(pc, x2, both(1.f / 24.f));
        ps = fma2(ps, x2, both(1.f));
        pc = fma2(pc, x2, both(-0.5f));
        *s = mul2(x, ps);
        *c = fma2(pc, x2, both(1.f));
    } else {
        float2 sn, cs;
        sincosf(xx.x, &sn.x, &cs.x);
        sincosf(xx.y, &sn.y, &cs.y);
        *s = pack2(sn.x, sn.y);
        *c = pack2(cs.x, cs.y);
    }
}

// The mixed near field. One CTA per target leaf, its four warps taking every fourth source
// leaf; 32 sources at a time in the warp's slice of shared memory, as pairs (positions
// negated, hi and lo halves, charges), read back as broadcasts. 32 / G targets a pass with G
// lanes each on the source pairs, G chosen per leaf (p2p_lanes); only __syncwarp orders the
// slices. A lane works on two sources at once in packed FP32 arithmetic: the kernel was
// bound by issue slots (58 % issue active at 51 % of the FP32 pipe), and a packed operation
// takes one slot for two. FP32 sums of one source leaf (at most CHAIN sources) go into the
// lane's FP64 sums; the lanes' and the warps' FP64 sums are added in a fixed order.
template <int NF, int R, bool FIELD>
__global__ void __launch_bounds__(WARPS * 32) k_p2p_mx(EvalView v, const int32_t* __restrict__ leaves,
                                                      const int32_t* __restrict__ off,
                                                      const int32_t* __restrict__ srcs, double* pot,
                                                      double* fld) {
    constexpr int NC = PairSums<NF, R, FIELD>::NC, NA = PairSums<NF, R, FIELD>::N;
    // per source pair: -xh, -yh | -zh, -xl | -yl, -zl | q columns, two floats each; rows of
    // 80 bytes spread the lanes' stores over the banks
    __shared__ __align__(16) float2 stage[WARPS][16][10];
    __shared__ double part[WARPS - 1][NA][32];
    const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = leaves[row];
    const int s0t = v.leaf_start[t], cnt_t = v.counts[t];
    const double C16 = 1.2621774483536189e-29;   // (16 * 2^-52)^2: the FP64 pair floor
    const double rt = v.rmax[t];
    const f2 kf = both((float)v.k);
    const int64_t n = v.n;
    const int e0 = off[row], e1 = off[row + 1];
    const int G = p2p_lanes(cnt_t), TG = 32 / G;
    const int tg = lane & (TG - 1), sub = lane / TG;
    float2(&sw)[16][10] = stage[warp];
    for (int i0 = 0; i0 < cnt_t; i0 += TG) {
        const int i = i0 + tg;
        const bool act = i < cnt_t;
        const int64_t gt = s0t + (act ? i : 0);
        const f2 xh = both(v.pos_f[gt]), yh = both(v.pos_f[n + gt]), zh = both(v.pos_f[2 * n + gt]);
        const f2 xl = both(v.pos_f[3 * n + gt]), yl = both(v.pos_f[4 * n + gt]), zl = both(v.pos_f[5 * n + gt]);
        double acc[NA];
#pragma unroll
        for (int q = 0; q < NA; ++q) acc[q] = 0.0;
        for (int e = e0 + warp; e < e1; e += WARPS) {
            const int sb = srcs[e];
            const int s0 = v.leaf_start[sb], cnt = v.counts[sb];
            const double rs = rt + v.rmax[sb];
            const float thr = (float)(C16 * rs * rs);
            for (int c0 = 0; c0 < cnt; c0 += CHAIN) {
                const int cend = min(cnt, c0 + CHAIN);
                f2 a32[NA];
#pragma unroll
                for (int q = 0; q < NA; ++q) a32[q] = both(0.f);
                for (int b0 = c0; b0 < cend; b0 += 32) {
                    const int nbat = min(32, cend - b0);
                    __syncwarp();   // the previous batch has been read
                    if (lane < ((nbat + 1) & ~1)) {
                        // an odd batch ends with its last source again, at zero charge
                        const int64_t gs = s0 + b0 + min(lane, nbat - 1);
                        float* o = reinterpret_cast<float*>(sw[lane >> 1]) + (lane & 1);
                        o[0] = -v.pos_f[gs];
                        o[2] = -v.pos_f[n + gs];
                        o[4] = -v.pos_f[2 * n + gs];
                        o[6] = -v.pos_f[3 * n + gs];
                        o[8] = -v.pos_f[4 * n + gs];
                        o[10] = -v.pos_f[5 * n + gs];
                        o[12] = lane < nbat ? (float)v.q_s[gs] : 0.f;
                        o[14] = R > 1 && lane < nbat ? (float)v.q_s[n + gs] : 0.f;
                    }
                    __syncwarp();
                    const int npair = (nbat + 1) >> 1;
                    for (int j = sub; j < npair; j += G) {
                        const ulonglong2* w4 = reinterpret_cast<const ulonglong2*>(sw[j]);
                        const ulonglong2 p0 = w4[0], p1 = w4[1], p2 = w4[2], p3 = w4[3];
                        const f2 dx = add2(add2(xh, f2{p0.x}), add2(xl, f2{p1.y}));
                        const f2 dy = add2(add2(yh, f2{p0.y}), add2(yl, f2{p2.x}));
                        const f2 dz = add2(add2(zh, f2{p1.x}), add2(zl, f2{p2.y}));
                        const f2 d2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
                        const float2 d2s = unpack2(d2);
                        // pairs under the floor (the target itself) contribute nothing
                        const f2 ir = pack2(d2s.x > thr ? rsqrtf(d2s.x) : 0.f, d2s.y > thr ? rsqrtf(d2s.y) : 0.f);
                        const f2 kr = mul2(kf, mul2(d2, ir));
                        f2 sn, cs;
                        if (v.yukawa) {   // the kernel seam (particles.cuh): one family
                            const float2 k2 = unpack2(kr);
                            sn = cs = pack2(__expf(-k2.x) * 0.0795774715f, __expf(-k2.y) * 0.0795774715f);
                        } else {
                            sincos_phase2(kr, &sn, &cs);
                        }
                        const f2 w0 = mul2(cs, ir), w1 = mul2(sn, ir);
                        const f2 q0{p3.x}, q1{p3.y};
                        // real and imaginary part (PairSums): E_cos(q0) - E_sin(q1), E_sin(q0) + E_cos(q1)
                        a32[0] = fma2(q0, w0, a32[0]);
                        if (NF == 2 && R == 2) a32[0] = fma2(neg2(q1), w1, a32[0]);
                        if (NF == 2) a32[NC - 1] = fma2(q0, w1, a32[NC - 1]);
                        if (R == 2) a32[NC - 1] = fma2(q1, w0, a32[NC - 1]);
                        if (FIELD) {
                            const f2 ir3 = mul2(mul2(ir, ir), ir);
                            const f2 f0 = mul2(fma2(kr, sn, cs), ir3), f1 = mul2(fma2(neg2(kr), cs, sn), ir3);
                            f2 g[2];
                            g[0] = mul2(q0, f0);
                            if (NF == 2 && R == 2) g[0] = fma2(neg2(q1), f1, g[0]);
                            if (NF == 2) g[1] = mul2(q0, f1);
                            if (R == 2) g[1] = NF == 2 ? fma2(q1, f0, g[1]) : mul2(q1, f0);
#pragma unroll
                            for (int c = 0; c < NC; ++c) {
                                a32[NC + 3 * c + 0] = fma2(g[c], dx, a32[NC + 3 * c + 0]);
                                a32[NC + 3 * c + 1] = fma2(g[c], dy, a32[NC + 3 * c + 1]);
                                a32[NC + 3 * c + 2] = fma2(g[c], dz, a32[NC + 3 * c + 2]);
                            }
                        }
                    }
                }
#pragma unroll
                for (int q = 0; q < NA; ++q) {
                    const float2 u = unpack2(a32[q]);
                    acc[q] += (double)u.x + (double)u.y;
                }
            }
        }
        for (int o = TG; o < 32; o <<= 1)
#pragma unroll
            for (int q = 0; q < NA; ++q) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
        __syncthreads();   // the previous pass's parts have been read
        if (warp > 0)
#pragma unroll
            for (int q = 0; q < NA; ++q) part[warp - 1][q][lane] = acc[q];
        __syncthreads();
        if (warp == 0 && act && sub == 0) {
#pragma unroll
            for (int w = 0; w < WARPS - 1; ++w)
#pragma unroll
                for (int q = 0; q < NA; ++q) acc[q] += part[w][q][lane];
#pragma unroll
            for (int q = 0; q < NC; ++q) pot[q * n + gt] = acc[q];
            if (FIELD)
#pragma unroll
                for (int q = 0; q < NC * 3; ++q) fld[q * n + gt] = acc[NC + q];
        }
    }
}

template <int NF, int R, bool FIELD>
void impl(const ParticlePass& p, cudaStream_t s) {
    if (p.op != ParticleOp::P2P)
        throw Error{HFMM_ERR_STATE, "particles_mixed: only the near field runs in FP32"};
    HFMM_LAUNCH((k_p2p_mx<NF, R, FIELD>), (unsigned)p.nrows, WARPS * 32, 0, s, p.v, p.rows, p.off, p.srcs,
                p.pot, p.fld);
}

}  // namespace

void particles_mixed(const ParticlePass& p, cudaStream_t s) {
    if (p.nrows == 0) return;
    const int key = (p.nf - 1) * 4 + (p.R - 1) * 2 + (p.field ? 1 : 0);
    switch (key) {
        case 0: impl<1, 1, false>(p, s); break;
        case 1: impl<1, 1, true>(p, s); break;
        case 2: impl<1, 2, false>(p, s); break;
        case 3: impl<1, 2, true>(p, s); break;
        case 4: impl<2, 1, false>(p, s); break;
        case 5: impl<2, 1, true>(p, s); break;
        case 6: impl<2, 2, false>(p, s); break;
        case 7: impl<2, 2, true>(p, s); break;
        default: throw Error{HFMM_ERR_ARG, "particles_mixed: bad configuration"};
    }
}

}  // namespace hfmm
