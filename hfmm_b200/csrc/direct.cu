// Direct-sum referee: phi_t = sum_{s: r > 0} q_s e^{ikr} / r at sampled targets
// (test.py:11-18), and the field -grad phi = sum q_s e^{ikr} (1 - ikr) / r^3 (x_t - x_s).
// With the screened-Coulomb kernel (yukawa != 0, k = kappa): phi_t = sum q_s G(r),
// G = exp(-kappa r) / (4 pi r), field sum q_s (1 + kappa r) exp(-kappa r) / (4 pi r^3) d.
//
// Sources are split into n_split contiguous chunks; each (target block, chunk)
// CTA writes its partial sums to scratch, and a second kernel adds the chunks
// in a fixed order, so the result does not depend on scheduling.
#include "hfmm_internal.cuh"
#include "particles.cuh"

#include <algorithm>
#include <cstring>
#include <type_traits>

namespace hfmm {

namespace {

constexpr int DT = 128;        // targets per CTA
constexpr int DSTAGE = 256;    // sources staged per pass
constexpr int NV = 8;          // phi re/im + field 3 x re/im

// One FP64 pair costs 51 operations with complex charges and the field, which bound the
// kernel; two sources a step keep the FP64 pipe fed (their chains are independent).
// FAST: the Helmholtz kernel in pair64's branch-free form.
template <int NF, int R, bool FIELD, bool FAST>
__global__ void __launch_bounds__(DT, 5) k_direct_partial(const double* __restrict__ pos,
                                                       const double* __restrict__ q_re,
                                                       const double* __restrict__ q_im, int64_t n,
                                                       const int32_t* __restrict__ tg, int64_t n_t,
                                                       double k, unsigned lo_hi, unsigned range, int n_split,
                                                       double* scratch, int* err) {
    constexpr int NC = PairSums<NF, R, FIELD>::NC, NA = PairSums<NF, R, FIELD>::N;
    __shared__ double sx[DSTAGE], sy[DSTAGE], sz[DSTAGE], sq[R][DSTAGE];
    const int64_t ti = blockIdx.x * (int64_t)DT + threadIdx.x;
    const int split = blockIdx.y;
    const int64_t chunk = (n + n_split - 1) / n_split;
    const int64_t lo = split * chunk, hi = (lo + chunk < n) ? lo + chunk : n;
    bool act = ti < n_t;
    double x = 0, y = 0, z = 0;
    if (act) {
        int64_t t = tg[ti];
        if (t < 0 || t >= n) {
            atomicOr(err, ERRF_BOUNDS);
            act = false;
        } else {
            x = pos[3 * t];
            y = pos[3 * t + 1];
            z = pos[3 * t + 2];
        }
    }
    double acc[NA];
#pragma unroll
    for (int v = 0; v < NA; ++v) acc[v] = 0.0;
    for (int64_t p0 = lo; p0 < hi; p0 += DSTAGE) {
        __syncthreads();
        for (int i = threadIdx.x; i < DSTAGE; i += DT) {
            int64_t s = p0 + i;
            if (s < hi) {
                sx[i] = pos[3 * s];
                sy[i] = pos[3 * s + 1];
                sz[i] = pos[3 * s + 2];
                sq[0][i] = q_re[s];
                if (R == 2) sq[R - 1][i] = q_im[s];
            }
        }
        __syncthreads();
        if (!act) continue;
        const int np = (int)((hi - p0 < DSTAGE) ? hi - p0 : DSTAGE);
        // The staged sources into sums of their own, so that a stage with a separation outside
        // [1e-290, 1e290] (a NaN among them) or a phase over 1e5 (judged by r2's high word) is
        // done over in the general form; a coincident source counts as one at zero charge there,
        // and a separation that is no number is left out.
        double part[NA];
        bool odd = false;
        auto sources = [&](auto fast) {
#pragma unroll
            for (int v = 0; v < NA; ++v) part[v] = 0.0;
#pragma unroll 2
            for (int i = 0; i < np; ++i) {
                const double dx = x - sx[i], dy = y - sy[i], dz = z - sz[i];
                const double r2 = dx * dx + dy * dy + dz * dz;
                if (!decltype(fast)::value && !(r2 >= 0.0)) continue;
                const bool far = r2 != 0.0;
                double q[NF][R];
#pragma unroll
                for (int f = 0; f < NF; ++f)
#pragma unroll
                    for (int r = 0; r < R; ++r) q[f][r] = far ? sq[r][i] : 0.0;
                const double r2s = far ? r2 : 1.0;
                if (decltype(fast)::value) odd = odd || (unsigned)__double2hiint(r2s) - lo_hi >= range;
                pair64<NF, R, FIELD, decltype(fast)::value>(NF == 1, k, dx, dy, dz, r2s, q, part);
            }
        };
        if (FAST) sources(std::true_type());
        if (!FAST || odd) sources(std::false_type());
#pragma unroll
        for (int v = 0; v < NA; ++v) acc[v] += part[v];
    }
    if (act) {   // re, im of the potential, then of the field's components
        double* o = scratch + ((int64_t)split * n_t + ti) * NV;
        o[0] = acc[0];
        o[1] = NC == 2 ? acc[NC - 1] : 0.0;
        if (FIELD)
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                o[2 + 2 * a] = acc[NC + a];
                o[3 + 2 * a] = NC == 2 ? acc[NC + 3 * (NC - 1) + a] : 0.0;
            }
    }
}

// The chunks' partial sums of one (target, value) pair added by one warp: lane j takes
// chunks j, j + 32, ... in order, then a fixed shuffle tree adds the lanes, so the
// result does not depend on scheduling. (One thread per target had walked all chunks
// serially: 0.26 ms for the 256-target check at 1e6 sources.)
__global__ void k_direct_reduce(const double* __restrict__ scratch, int64_t n_t, int n_split,
                                int field, double* phi, double* fld) {
    const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= n_t * NV) return;
    const int64_t ti = w / NV;
    const int v = (int)(w % NV);
    if (!field && v >= 2) return;
    double acc = 0.0;
    for (int s = lane; s < n_split; s += 32) acc += scratch[((int64_t)s * n_t + ti) * NV + v];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane != 0) return;
    if (v < 2) phi[2 * ti + v] = acc;
    else if (fld) fld[(ti * 3 + (v - 2) / 2) * 2 + (v - 2) % 2] = acc;
}

}  // namespace

int direct_splits(int64_t n, int64_t n_t) {
    int64_t tblocks = ceil_div(std::max<int64_t>(n_t, 1), DT);
    // five CTAs per SM are resident: at most so many in all, one wave
    int64_t want = std::max<int64_t>(1, 5 * 148 / tblocks);
    int64_t by_work = ceil_div(std::max<int64_t>(n, 1), 2048);  // at least 2048 sources a split
    return (int)std::max<int64_t>(1, std::min<int64_t>(want, by_work));
}

void direct_sum(const double* pos, const double* q_re, const double* q_im, int64_t n,
                const int32_t* targets, int64_t n_t, double k, double* phi, double* fld,
                double* scratch, int n_split, cudaStream_t s, int* err, int yukawa) {
    if (n_t == 0) return;
    dim3 grid((unsigned)ceil_div(n_t, DT), (unsigned)n_split);
    // r2 in [1e-290, min(1e290, (1e5 / k)^2)), by high words (rounded inwards)
    auto high = [](double v) {
        uint64_t u;
        std::memcpy(&u, &v, sizeof(u));
        return (unsigned)(u >> 32);
    };
    const double far = k == 0.0 ? 1e290 : std::min(1e290, 1e10 / (k * k));
    const unsigned lo_hi = high(1e-290) + 1, hi_hi = far > 1e-289 ? high(far) : lo_hi;
    auto launch = [&](auto kern) {
        HFMM_LAUNCH(kern, grid, DT, 0, s, pos, q_re, q_im, n, targets, n_t, k, lo_hi, hi_hi - lo_hi, n_split,
                    scratch, err);
    };
    if (yukawa) {   // one real kernel
        if (q_im) fld ? launch(k_direct_partial<1, 2, true, false>) : launch(k_direct_partial<1, 2, false, false>);
        else fld ? launch(k_direct_partial<1, 1, true, false>) : launch(k_direct_partial<1, 1, false, false>);
    } else {
        if (q_im) fld ? launch(k_direct_partial<2, 2, true, true>) : launch(k_direct_partial<2, 2, false, true>);
        else fld ? launch(k_direct_partial<2, 1, true, true>) : launch(k_direct_partial<2, 1, false, true>);
    }
    HFMM_LAUNCH(k_direct_reduce, (unsigned)ceil_div(n_t * NV * 32, 256), 256, 0, s, scratch, n_t, n_split,
                fld ? 1 : 0, phi, fld);
}

}  // namespace hfmm
