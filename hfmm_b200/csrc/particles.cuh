// Shared view of a plan for the particle kernels (plain and mixed precision).
#pragma once
#include "hfmm_internal.cuh"

namespace hfmm {

struct EvalView {
    int64_t n, nb;
    int n_s, ld;
    double k;                  // Helmholtz wavenumber, or the screening constant kappa
    int yukawa;                // 0: Helmholtz (two families); 1: exp(-kappa r) / (4 pi r)
    int fast;                  // Helmholtz with two families, every phase k r under 1e5, |k| under
                               // 1e15 (a coincident point stands in at r = 1 with no charge: its
                               // phase need not be right, but finite) and the domain's size in
                               // [1e-100, 1e100]: pair64's FAST form
    int root;                  // phases so large that the near field takes pair64's ROOT form
    const double* pos_s;       // 3 x n, leaf-major sorted
    const float* pos_f;        // 6 x n: FP32 hi parts x|y|z, then lo parts (pos = hi + lo)
    const double* q_s;         // R x n, leaf-major sorted
    const int32_t* leaf_start;
    const int32_t* counts;
    const int32_t* lvls;
    const double* centre;      // 3 x nb
    const double* hbox;
    const double* rmax;
};

enum class ParticleOp { P2M, P2L, L2P, M2P, P2P, COMBINE };

struct ParticlePass {
    ParticleOp op;
    EvalView v;
    int nf = 1, R = 1;
    bool field = false;
    const int32_t* rows = nullptr;   // target boxes (P2M/P2L/L2P/M2P/P2P) or sort_idx (COMBINE)
    int64_t nrows = 0;
    const int32_t* off = nullptr;    // CSR offsets into srcs (P2L/M2P/P2P)
    const int32_t* srcs = nullptr;
    const double* surf = nullptr;    // unit surface (3 x n_s)
    const double* dens = nullptr;    // equivalent densities [fam][box][R][ld]
    double* out = nullptr;           // check potentials [fam][box][R][ld]
    int64_t fam_stride = 0;
    int level = -1;                  // P2L: one level's targets, or all (-1)
    int maxleaf = 1;                 // the widest leaf (L2P/M2P)
    double* pot = nullptr;           // [re, im][n] (re alone: one family, real charges)
    double* fld = nullptr;           // [re, im][x, y, z][n]
    double* phi = nullptr;           // COMBINE outputs (complex interleaved)
    double* E = nullptr;
};

// Coefficients in constant memory: an FP64 operation takes one operand from there, where a
// literal costs two moves into registers at every use (117 instructions a P2M pair, 38 of
// them FP64, with literals).
static __constant__ double c_trig[] = {
    0.6366197723675814, 6755399441055744.0,            // 2 / pi, 1.5 * 2^52
    1.5707963267948966, 6.123233995736766e-17,         // pi / 2 in two parts
    -1.591810123027412e-10, 2.5051131455427946e-08, -2.755731610068303e-06,   // P, degree 5 down
    0.0001984126983675497, -0.008333333333330946, 0.16666666666666666,
    1.1367978191553177e-11, -2.0875886390883725e-09, 2.755731556415141e-07,   // Q, degree 6 down
    -2.480158729368715e-05, 0.0013888888888880767, -0.04166666666666664, 0.5};

// sin and cos of a phase. Cody-Waite reduction against pi/2 in two parts, its FP64 value and
// the remainder of pi: x - n hi is exact for |x| < 1e5 (n < 2^16), and n comes from adding
// 1.5 * 2^52, whose low word holds the quadrant. On |r| <= pi/4, sin r = r - r^3 P(r^2) and
// cos r = 1 - r^2 Q(r^2) with P and Q interpolated at the Chebyshev nodes of [0, (pi/4)^2]
// (degrees 5 and 6, computed in 60 digits): 2.0e-17 and 6.1e-19 relative, under the rounding.
// 19 FP64 operations for any phase met; larger ones (and NaN) take sincos. The Taylor series
// through x^22 used before took 25 up to 1.5 and left larger phases to sincos.
__device__ __forceinline__ void sincos_reduced64(double x, double* s, double* c) {   // |x| < 1e5
    const double t = fma(x, c_trig[0], c_trig[1]);
    const double n = t - c_trig[1];
    const int quad = __double2loint(t);
    double r = fma(-n, c_trig[2], x);
    r = fma(-n, c_trig[3], r);
    const double z = r * r;
    double P = fma(z, c_trig[4], c_trig[5]);
    double Q = fma(z, c_trig[10], c_trig[11]);
    P = fma(P, z, c_trig[6]);
    Q = fma(Q, z, c_trig[12]);
    P = fma(P, z, c_trig[7]);
    Q = fma(Q, z, c_trig[13]);
    P = fma(P, z, c_trig[8]);
    Q = fma(Q, z, c_trig[14]);
    P = fma(P, z, c_trig[9]);
    Q = fma(Q, z, c_trig[15]);
    Q = fma(Q, z, c_trig[16]);
    const double sr = fma(-(r * z), P, r);
    const double cr = fma(-z, Q, 1.0);
    const double a = quad & 1 ? cr : sr, b = quad & 1 ? sr : cr;
    *s = __hiloint2double(__double2hiint(a) ^ (int)((unsigned)(quad & 2) << 30), __double2loint(a));
    *c = __hiloint2double(__double2hiint(b) ^ (int)((unsigned)((quad + 1) & 2) << 30), __double2loint(b));
}

__device__ __forceinline__ void sincos_phase64(double x, double* s, double* c) {
    if ((__double2hiint(x) & 0x7fffffff) >= 0x40f86a00) sincos(x, s, c);   // 1e5
    else sincos_reduced64(x, s, c);
}

// 1 / sqrt(x) for x in [1e-290, 1e290]: the hardware's approximation, then one step of
// Householder's third-order iteration, y (1 + e/2 + 3 e^2/8) with e = 1 - x y^2 (an error
// d of the seed leaves 2.5 d^3). Five FP64 operations and no branch, so that a loop can run
// two pairs' chains side by side.
__device__ __forceinline__ double rsqrt_normal(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
}

// The kernel seam of the particle kernels. Helmholtz: (sn, cs) = sin, cos of the phase
// kr, so family 0 is cs / r, family 1 sn / r and their field weights (cs + kr sn) / r^3
// and (sn - kr cs) / r^3 (HFMM.py:25-40). The screened-Coulomb kernel (one family,
// jaxfmm/kernels/yukawa/kernel.py:36-75; kappa = 0 is Laplace,
// kernels/laplace/kernel.py:40-104) puts exp(-kr) / (4 pi) in both slots, so family 0's
// value cs / r and field weight (cs + kr sn) / r^3 = (1 + kr) exp(-kr) / (4 pi r^3) come
// out of the same expressions.
constexpr double INV_4PI = 0.07957747154594767;
__device__ __forceinline__ void kernel_pair64(int yukawa, double kr, double* sn, double* cs) {
    if (yukawa) {
        const double e = exp(-kr) * INV_4PI;
        *sn = e;
        *cs = e;
    } else {
        sincos_phase64(kr, sn, cs);
    }
}

// Sums at a particle. The result of complex charges is phi = E_cos(q_re) - E_sin(q_im) +
// i (E_sin(q_re) + E_cos(q_im)), so a particle needs its real and imaginary part only (the
// real one alone with one family and real charges), not one sum per family and column:
// 10 operations a pair for the field instead of 16, and half the sums to store.
template <int NF, int R, bool FIELD>
struct PairSums {
    static constexpr int NC = NF == 1 && R == 1 ? 1 : 2;
    static constexpr int N = NC * (FIELD ? 4 : 1);   // potential, then the field's x, y, z
};

// a[0] + i a[1] += the families' weights w on the columns of family f, column r: d[f][r]
template <int NF, int R, typename T>
__device__ __forceinline__ void pair_columns(const T (&w)[2], const T (&d)[NF][R], T (&g)[2]) {
    g[0] = d[0][0] * w[0];
    if (NF == 2 && R == 2) g[0] -= d[NF - 1][R - 1] * w[1];
    g[1] = T(0);
    if (NF == 2) g[1] = d[NF - 1][0] * w[1];
    if (R == 2) g[1] += d[0][R - 1] * w[0];
}

// Lanes per target of a near-field warp on a leaf of cnt particles (a power of two): the
// count that costs the fewest source steps, ceil(cnt / (32 / G)) passes of 32 / G steps per
// 32 sources and one step's worth of staging each. 30 particles: 1 lane (one pass, 94 % of
// the lanes busy); 33: 4 lanes (five passes of eight targets, 82 %, where two passes of 32
// would leave half the lanes idle); 4: 8 lanes.
__device__ __forceinline__ int p2p_lanes(int cnt) {
    int best = 1, cost = 1 << 30;
#pragma unroll
    for (int G = 1; G <= 32; G *= 2) {
        const int TG = 32 / G, c = ((cnt + TG - 1) / TG) * (TG + 1);
        if (c < cost) {
            cost = c;
            best = G;
        }
    }
    return best;
}

// One FP64 pair at separation (dx, dy, dz), r2 > 0, into the sums. FAST: a Helmholtz phase
// under 1e5 and r2 in [1e-290, 1e290], without a branch; else any kernel and any values.
// ROOT: r to the last bit, one Newton step on from r2 / sqrt(r2), for large phases k r.
template <int NF, int R, bool FIELD, bool FAST, bool ROOT = false>
__device__ __forceinline__ void pair64(int yukawa, double k, double dx, double dy, double dz, double r2,
                                       const double (&d)[NF][R],
                                       double (&acc)[PairSums<NF, R, FIELD>::N]) {
    constexpr int NC = PairSums<NF, R, FIELD>::NC;
    double ir, r;
    if (ROOT && !FAST && !(r2 > 1e-290 && r2 < 1e290)) {
        r = sqrt(r2);
        ir = 1.0 / r;
    } else {
        ir = FAST ? rsqrt_normal(r2) : rsqrt(r2);
        r = r2 * ir;
        if (ROOT) r = fma(fma(-r, r, r2), 0.5 * ir, r);
    }
    const double kr = k * r;
    double sn, cs;
    if (FAST) sincos_reduced64(kr, &sn, &cs);
    else kernel_pair64(yukawa, kr, &sn, &cs);
    const double w[2] = {cs * ir, sn * ir};
    if (NF == 2 && R == 2) {
        acc[0] = fma(d[0][0], w[0], fma(-d[NF - 1][R - 1], w[1], acc[0]));
        acc[NC - 1] = fma(d[NF - 1][0], w[1], fma(d[0][R - 1], w[0], acc[NC - 1]));
    } else {
        acc[0] = fma(d[0][0], w[0], acc[0]);
        if (NF == 2) acc[NC - 1] = fma(d[NF - 1][0], w[1], acc[NC - 1]);
        if (R == 2) acc[NC - 1] = fma(d[0][R - 1], w[0], acc[NC - 1]);
    }
    if (FIELD) {
        const double ir2 = ir * ir;
        const double wf[2] = {fma(kr, w[1], w[0]) * ir2, fma(-kr, w[0], w[1]) * ir2};
        double g[2];
        pair_columns<NF, R, double>(wf, d, g);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            acc[NC + 3 * c + 0] = fma(g[c], dx, acc[NC + 3 * c + 0]);
            acc[NC + 3 * c + 1] = fma(g[c], dy, acc[NC + 3 * c + 1]);
            acc[NC + 3 * c + 2] = fma(g[c], dz, acc[NC + 3 * c + 2]);
        }
    }
}

void particles_f64(const ParticlePass& p, cudaStream_t s);
void particles_mixed(const ParticlePass& p, cudaStream_t s);
void gather_charges(int64_t n, const int32_t* sidx, const double* q_re, const double* q_im,
                    double* q_s, unsigned long long* q_max, cudaStream_t s);

}  // namespace hfmm
