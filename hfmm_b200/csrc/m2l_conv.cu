// FP64 M2L as a convolution. Both M2L surfaces are the same regular grid (surface points
// of a p x p x p lattice, kifmm/surfaces.py:40-85 at radius 1.05), so the matrix of one
// displacement d, G(x_m + 2 d - y_k), depends on the lattice lag m - k alone: a translation
// (phases.py:211-236) is a 3-D convolution of p^3 values with (2p-1)^3 lags. A cyclic
// transform of n = 2p - 1 points per axis makes it exact, and every displacement a
// multiplication by a number per frequency, summed over the V list before one inverse
// transform per target:
//     X = F(x) of every box;   Y_t = sum_d K_d .* X_{s(t, d)};   check_t = F^-1(Y_t).
// With two families complex charges travel as one complex sequence (the kernel is real), real
// charges as the half spectrum; with one family the result's real and imaginary parts are
// those of the charges, and each column is a real sequence of its own. Against the dense tables (2 n_s^2 a pair and column) that is 8 n^3 a pair
// and column pair: 27 against 350 kFLOP at p = 8, 97 against 2,120 at p = 12. One
// evaluate, complex charges, field (B200): 1e6 points, p = 8, depth 5: 210.2 ms with the
// tables, 31.7 now (products 13.2, transforms 3.3 and 4.0 of it); 20,000 points, depth 3:
// p = 8 6.69 and 0.84 ms, p = 12 32.7 and 2.23 ms.
//
// Work is laid out by PARENT: the children of one parent ("slot") sit side by side, absent
// ones as zeros, X as [frequency][slot][child]. The products of one frequency and one of
// the 26 parent offsets D are then an 8 x 8 complex block (target child x source child), the
// same for every slot: a small matrix times the columns of all slots, which the FP64 tensor
// instruction m16n8k4 takes as it is (16 rows = re and im of 8 target children). 1,512 of
// its 1,664 products are V pairs; the adjacent ones multiply a stored zero.
#include "hfmm_internal.cuh"
#include "m2l_conv.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

namespace hfmm {

namespace {

// K of one frequency in shared memory, [dx + 3][dy + 3][dz + 3] with strides 66, 9, 1: a
// phase of eight lanes reads (two target children) x (four source children), offsets
// {-66, 0, 66} - {0, 9}, which are distinct 16-byte banks mod 8.
constexpr int KSX = 66, KSY = 9, KTAB = 6 * KSX + 6 * KSY + 7;

__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b0) {
    asm volatile(
        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
        "{%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a0), "d"(a1), "d"(b0));
}

// ---------------------------------------------------------------- tables
// G at lag (ax, ay, az) of displacement slot d, layout [cell][343] (d fastest, as in every
// pass below); fam as in tables.cu: 0 cos(kr)/r, 1 sin(kr)/r, 2 exp(-kr)/(4 pi r).
__global__ void k_conv_gen(int p, int n, double spacing, double s, double kw, int fam, double* out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= (int64_t)n * n * n * N_DISP) return;
    const int d = (int)(i % N_DISP);
    const int cell = (int)(i / N_DISP);
    const int dx = d / 49 - 3, dy = (d / 7) % 7 - 3, dz = d % 7 - 3;
    const int near = max(abs(dx), max(abs(dy), abs(dz)));
    double v = 0.0;
    if (near > 1) {
        const int a[3] = {cell % n, (cell / n) % n, cell / (n * n)};
        const int dd[3] = {dx, dy, dz};
        double x[3];
        for (int c = 0; c < 3; ++c) x[c] = (2.0 * dd[c] + spacing * (a[c] < p ? a[c] : a[c] - n)) * s;
        const double r = sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
        if (fam == 2) {
            v = exp(-kw * r) / (4.0 * M_PI * r);
        } else {
            double sn, cs;
            sincos(kw * r, &sn, &cs);
            v = (fam == 1 ? sn : cs) / r;
        }
    }
    out[i] = v;
}

// One axis of the tables' transform: out[hi][k][lo][d] = scale sum_a in[hi][a][lo][d] w^(a k)
// for k < nk, w = e^{-2 pi i / n}; `lo` cells vary faster than the axis. REAL: in is real.
template <bool REAL>
__global__ void k_conv_axis(const double* __restrict__ in, int n, int nk, int64_t n_lo, int64_t total,
                            const double2* __restrict__ tw, double scale, double2* out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int64_t lo = i % n_lo;
    const int k = (int)((i / n_lo) % nk);
    const int64_t hi = i / (n_lo * nk);
    double re = 0.0, im = 0.0;
    int m = 0;
    for (int a = 0; a < n; ++a) {
        const double2 w = tw[m];
        const int64_t src = (hi * n + a) * n_lo + lo;
        if (REAL) {
            const double x = in[src];
            re = fma(x, w.x, re);
            im = fma(-x, w.y, im);
        } else {
            const double2 x = reinterpret_cast<const double2*>(in)[src];
            re = fma(x.x, w.x, fma(x.y, w.y, re));
            im = fma(x.y, w.x, fma(-x.x, w.y, im));
        }
        m += k;
        if (m >= n) m -= n;
    }
    out[i] = make_double2(re * scale, im * scale);
}

// ---------------------------------------------------------------- schedule
// nbr[slot][D]: the slot of the parent at offset D when it holds a V source of this slot's
// children (read off the M2L source table), else the zero slot.
__global__ void k_conv_nbr(const int32_t* __restrict__ child, const int32_t* __restrict__ m2l_src,
                           const int32_t* __restrict__ p_id, const int32_t* __restrict__ slot_of,
                           int n_slots, int32_t* nbr) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_slots * 26) return;
    const int slot = i / 26, D = i % 26;
    int ox, oy, oz;
    neigh_offset(D, ox, oy, oz);
    int found = n_slots;
    for (int t = 0; t < 8 && found == n_slots; ++t) {
        const int b = child[slot * 8 + t];
        if (b < 0) continue;
        for (int s = 0; s < 8; ++s) {
            const int dx = -2 * ox + (t & 1) - (s & 1);
            const int dy = -2 * oy + ((t >> 1) & 1) - ((s >> 1) & 1);
            const int dz = -2 * oz + ((t >> 2) & 1) - ((s >> 2) & 1);
            if (max(abs(dx), max(abs(dy), abs(dz))) <= 1) continue;
            const int src = m2l_src[(int64_t)b * M2L_ENTRIES + (dx + 3) * 49 + (dy + 3) * 7 + dz + 3];
            if (src >= 0) {
                found = slot_of[p_id[src]];
                break;
            }
        }
    }
    nbr[i] = found;
}

// ---------------------------------------------------------------- transforms
// A transform leaves a rounding of the larger column in the smaller one of a complex sequence.
// The column of smaller charges is therefore brought to the scale of the other, by a power of two
// (exact; up, so that nothing underflows), on the way in and back on the way out: each column's error is then that of its own
// magnitude, as where the columns travel apart (k = 1e-6, imaginary charges 1e-8 of the real
// ones: imaginary part off by 4e-10 without, 4e-15 with it). A column of zeros stays zeros.
struct Balance {
    double up[2] = {1.0, 1.0}, down[2] = {1.0, 1.0};
    bool any[2] = {true, true};   // the column holds a charge
};
__device__ __forceinline__ Balance balance(const unsigned long long* q_max) {
    Balance b;
    b.any[0] = q_max[0] != 0;
    b.any[1] = q_max[1] != 0;
    const int er = (int)(q_max[0] >> 52), ei = (int)(q_max[1] >> 52), d = abs(er - ei);
    if (er > 0 && ei > 0 && er < 2047 && ei < 2047 && d < 1000) {
        const double up = __longlong_as_double((long long)(1023 + d) << 52);
        const double down = __longlong_as_double((long long)(1023 - d) << 52);
        b.up[0] = er < ei ? up : 1.0;
        b.down[0] = er < ei ? down : 1.0;
        b.up[1] = er < ei ? 1.0 : up;
        b.down[1] = er < ei ? 1.0 : down;
    }
    return b;
}

// One axis is a small real matrix times many columns, and runs on the FP64 tensor
// instruction too. The pairs (k, n - k) share their sums: with v_j complex,
//   forward, j < p values in:   C_k = sum_j v_j cos(2 pi j k / n), S_k = sum_j v_j sin(..),
//                               X_k = C_k - i S_k, X_(n-k) = C_k + i S_k;
//   inverse, j < p values out:  P_k = Y_k + Y_(n-k), M_k = Y_k - Y_(n-k),
//                               u_j = Y_0 + sum_k P_k cos(2 pi j k / n) + i M_k sin(..).
// k and j both run over p = (n + 1) / 2 values, so one table serves: T[u][s][lane] = cos and
// sin of 2 pi (4 s + lane % 4) (8 u + lane / 4) / n, zero where the first factor is >= p.
// (One thread per column with scalar sums before spent its issue slots on twiddle indexes:
// FP64 pipe 17 and 12 % busy; forward 4.0 and inverse 6.0 ms at 1e6 points, p = 8.)
struct AxisShape {
    int p, n, CH, lch, SR, KS, MT;   // lch = log2 CH; SR: row length in smem (CH + 2: no bank
                                     // conflicts); KS, MT: steps of 4 and tiles of 8 over p
};

__device__ __forceinline__ AxisShape axis_shape(const ConvCall& c) {
    AxisShape a;
    a.p = c.p;
    a.n = c.n;
    a.CH = c.CH;
    a.lch = 31 - __clz(c.CH);
    a.SR = c.CH + 2;
    a.KS = (c.p + 3) / 4;
    a.MT = (c.p + 7) / 8;
    return a;
}

__device__ __forceinline__ void axis_table(const AxisShape& a, const double2* tw, double2* T) {
    for (int i = threadIdx.x; i < a.MT * a.KS * 32; i += blockDim.x) {
        const int lane = i & 31, s = (i >> 5) % a.KS, u = (i >> 5) / a.KS;
        const int f = 4 * s + (lane & 3);
        T[i] = f < a.p ? tw[f * (8 * u + (lane >> 2)) % a.n] : make_double2(0.0, 0.0);
    }
}

// Forward axis over n_grp groups of p rows of CH columns (rows[(grp * p + j) * SR + ch]):
// a 16 x 8 tile is (C and S of eight k) x (re and im of four columns), so a lane ends with
// C_k and S_k of one column. store(grp, ch, k, X_k, X_(n-k)) for k < p. KS > 0: the steps
// over p at compile time, their table values in registers for all tiles (0: any count).
template <int KS, class Store>
__device__ __forceinline__ void axis_forward(const AxisShape& a, const double2* rows, int n_grp, const double2* T,
                                             Store store) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int g = lane >> 2, t4 = lane & 3, ks = KS ? KS : a.KS;
    const int ncol = n_grp * a.CH, step = 8 * a.SR;   // doubles between rows j and j + 4
    for (int u = 0; u < a.MT; ++u) {
        const double2* Tu = T + u * ks * 32 + lane;
        double2 w[KS ? KS : 1];
#pragma unroll
        for (int s = 0; s < KS; ++s) w[s] = Tu[s * 32];
        const int k = 8 * u + g;
        for (int tile = warp; tile * 4 < ncol; tile += nw) {
            const int col = tile * 4 + (g >> 1), oc = tile * 4 + t4;
            const bool ok = col < ncol;
            const double* b = reinterpret_cast<const double*>(rows + ((ok ? col >> a.lch : 0) * a.p + t4) * a.SR +
                                                              (col & (a.CH - 1))) + (g & 1);
            double acc[4] = {0.0, 0.0, 0.0, 0.0};
            if (KS) {
                double v[KS ? KS : 1];
#pragma unroll
                for (int s = 0; s < KS; ++s) v[s] = ok && 4 * s + t4 < a.p ? b[s * step] : 0.0;
#pragma unroll
                for (int s = 0; s < KS; ++s) dmma(acc, w[s].x, w[s].y, v[s]);
            } else {
                for (int s = 0; s < ks; ++s) {
                    const double2 ws = Tu[s * 32];
                    dmma(acc, ws.x, ws.y, ok && 4 * s + t4 < a.p ? b[s * step] : 0.0);
                }
            }
            if (oc < ncol && k < a.p)
                store(oc >> a.lch, oc & (a.CH - 1), k, make_double2(acc[0] + acc[3], acc[1] - acc[2]),
                      make_double2(acc[0] - acc[3], acc[1] + acc[2]));
        }
    }
}

// Inverse axis over n_grp groups: load(grp, ch, k, P, M) gives P_k and M_k; a 16 x 8 tile is
// (re and im of eight columns) x (eight j). store(grp, ch, j, u_j) for j < p. (Steps at
// compile time, all loads ahead, took twice the registers and 35 % more time.)
template <class Load, class Store>
__device__ __forceinline__ void axis_inverse(const AxisShape& a, int n_grp, const double2* T, Load load,
                                             Store store) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const int ncol = n_grp * a.CH;
    for (int u = 0; u < a.MT; ++u)
        for (int tile = warp; tile * 8 < ncol; tile += nw) {
            const int col = tile * 8 + g, grp = col >> a.lch, ch = col & (a.CH - 1);
            const bool ok = col < ncol;
            double acc[4] = {0.0, 0.0, 0.0, 0.0};
            for (int s = 0; s < a.KS; ++s) {
                const int k = 4 * s + t4;
                double2 P = make_double2(0.0, 0.0), M = P;
                if (ok && k < a.p) load(grp, ch, k, P, M);
                const double2 w = T[(u * a.KS + s) * 32 + lane];
                dmma(acc, P.x, P.y, w.x);
                dmma(acc, -M.y, M.x, w.y);
            }
            const int j = 8 * u + 2 * t4;
            if (ok) {
                if (j < a.p) store(grp, ch, j, make_double2(acc[0], acc[2]));
                if (j + 1 < a.p) store(grp, ch, j + 1, make_double2(acc[1], acc[3]));
            }
        }
}

// Forward transform of a slot's children (c.CH of them per CTA): the frequencies of rows
// kz in [kz0, kz1) x ky in [ky0, ky1), all kx. Per kz: z sums of the surface lines (interior
// lines hold two points), then the y and x axes; the x axis stores 16 bytes x 4 children a
// frequency. 16 n^3 bytes a box leave the CTA: bound by those stores at large sizes.
template <int R, int KS>
__global__ void __launch_bounds__(256) k_conv_fwd(ConvCall c) {
    extern __shared__ double2 sh[];
    const AxisShape a = axis_shape(c);
    const int p = c.p, n = c.n, nh = p, CH = c.CH, nky = c.ky1 - c.ky0;
    const int slot = blockIdx.x, c0 = blockIdx.y * CH, seq = blockIdx.z / c.n_seg, seg = blockIdx.z % c.n_seg;
    const int nz = c.kz1 - c.kz0, kz0 = c.kz0 + seg * nz / c.n_seg, kz1 = c.kz0 + (seg + 1) * nz / c.n_seg;
    double2* tw = sh;                          // n
    double2* tz = tw + n;                      // p: e^{2 pi i k kz / n}
    double2* T = tz + p;
    double2* A1 = T + a.MT * a.KS * 32;        // [i][j][SR]
    double2* A2 = A1 + p * p * a.SR;           // [ky][i][SR]
    double* xs = reinterpret_cast<double*>(A2 + p * nky * a.SR);   // [point][CH][R]
    const int nkx = R == 2 ? n : nh;
    const int64_t fstride = (int64_t)(c.n_slots + 1) * 8;   // values of one frequency
    double2* X = c.X + (int64_t)seq * c.rows * nkx * fstride + (int64_t)slot * 8 + c0;
    const int tid = threadIdx.x, nt = blockDim.x;
    if (slot == c.n_slots) {   // the zero slot
        for (int64_t i = tid; seg == 0 && i < (int64_t)c.rows * nkx * CH; i += nt)
            X[(i / CH) * fstride + i % CH] = make_double2(0.0, 0.0);
        return;
    }
    for (int i = tid; i < n; i += nt) tw[i] = c.tw[i];
    const Balance bal = R == 2 ? balance(c.q_max) : Balance();
    for (int ch = 0; ch < CH; ++ch) {
        const int b = c.child[slot * 8 + c0 + ch];
        const double* src = c.dens + seq * c.seq_stride + b * c.box_stride;
        for (int r = 0; r < R; ++r)
            for (int s = tid; s < c.n_s; s += nt)
                xs[(c.pos[s] * CH + ch) * R + r] = b >= 0 ? src[r * c.ld + s] * (R == 2 ? bal.up[r] : 1.0) : 0.0;
    }
    __syncthreads();
    axis_table(a, tw, T);
    // the z items of this thread, (line, child): first value, count and spacing of its points
    // and its place in A1, worked out once for the first ZI of them
    constexpr int ZI = 3;
    int z_x[ZI], z_n[ZI], z_o[ZI];
    auto item = [&](int it, int& x, int& cnt, int& o) {
        const int ch = it & (CH - 1), line = it >> a.lch, i = line / p, j = line - i * p;
        cnt = i == 0 || j == 0 || i == p - 1 || j == p - 1 ? p : 2;
        x = (c.line_off[line] * CH + ch) * R;
        o = line * a.SR + ch;
    };
#pragma unroll
    for (int q = 0; q < ZI; ++q) {
        z_n[q] = 0;
        if (tid + q * nt < p * p * CH) item(tid + q * nt, z_x[q], z_n[q], z_o[q]);
    }
    auto line_sum = [&](int x0, int cnt, int o) {
        const double* x = xs + x0;
        const double2* w = tz;
        const int step = cnt == p ? 1 : p - 1;
        double re = 0.0, im = 0.0;
        for (int q = 0; q < cnt; ++q, x += CH * R, w += step) {
            if (R == 2) {
                const double2 v = *reinterpret_cast<const double2*>(x);
                re = fma(v.x, w->x, fma(v.y, w->y, re));
                im = fma(v.y, w->x, fma(-v.x, w->y, im));
            } else {
                re = fma(x[0], w->x, re);
                im = fma(-x[0], w->y, im);
            }
        }
        A1[o] = make_double2(re, im);
    };
    const bool full = R == 2 || nky == n;   // complex sequences come in whole planes
    for (int kz = kz0; kz < kz1; ++kz) {
        if (tid < p) tz[tid] = tw[tid * kz % n];
        __syncthreads();
#pragma unroll
        for (int q = 0; q < ZI; ++q)
            if (z_n[q]) line_sum(z_x[q], z_n[q], z_o[q]);
        for (int it = tid + ZI * nt; it < p * p * CH; it += nt) {
            int x, cnt, o;
            item(it, x, cnt, o);
            line_sum(x, cnt, o);
        }
        __syncthreads();
        axis_forward<KS>(a, A1, p, T, [&](int i, int ch, int k, double2 Xk, double2 Xn) {   // y
            const int m = n - k;
            if (full) {
                A2[(k * p + i) * a.SR + ch] = Xk;
                if (k > 0) A2[(m * p + i) * a.SR + ch] = Xn;
            } else {
                if (k >= c.ky0 && k < c.ky1) A2[((k - c.ky0) * p + i) * a.SR + ch] = Xk;
                if (k > 0 && m >= c.ky0 && m < c.ky1) A2[((m - c.ky0) * p + i) * a.SR + ch] = Xn;
            }
        });
        __syncthreads();
        double2* o = X + (int64_t)(kz - c.kz0) * nky * nkx * fstride;
        axis_forward<KS>(a, A2, nky, T, [&](int ky, int ch, int k, double2 Xk, double2 Xn) {   // x, to memory
            double2* q = o + (int64_t)ky * nkx * fstride + ch;
            q[k * fstride] = Xk;
            if (R == 2 && k > 0) q[(n - k) * fstride] = Xn;
        });
    }
}

// The products of one frequency and CONV_GROUP slots: per offset D and four source children,
// A = the 16 x 4 block of K (rows: re and im of the eight target children) against re and
// im of the sources, 8 slots per instruction; NT slot tiles per warp share each A. FP64
// tensor work is the bound (the CTA's X rows, 128 bytes a slot, hit L1 after the first
// offsets); K and the neighbour lists come from shared memory.
constexpr int NT = 2, CONV_WARPS = 4, CONV_GROUP = 8 * NT * CONV_WARPS;

// HALF: warps left with one tile's slots (the eight at the coarsest level, a level's remainder)
// skip the other tile. Where every warp is full that form takes 3 % more time, so it runs where
// such warps are one in 16 or more: 20,000 points, p = 8 260 to 247 us, p = 12 906 to 845; 1e6
// points 13.2 ms without, 13.7 with it. (One tile a warp everywhere: 247, 868 us and 14.8 ms.)
// Eight CTAs an SM: with six (75 registers, the second tile under a branch in the loop) 14.2 ms.
template <bool HALF>
__global__ void __launch_bounds__(32 * CONV_WARPS, 8) k_conv_mul(ConvCall c, int nkx) {
    __shared__ double2 Kt[KTAB];
    __shared__ int nb[CONV_GROUP][27];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int grp = blockIdx.x % c.n_groups;
    const int64_t f = blockIdx.x / c.n_groups;      // frequency within the chunk
    const int seq = blockIdx.y;
    const int4 G = c.groups[grp];                   // level, first slot, slots
    const int nky = c.ky1 - c.ky0;
    {
        const int row = (int)(f / nkx), n = c.n, nh = (n + 1) / 2;
        int kx = (int)(f % nkx), ky = c.ky0 + row % nky, kz = c.kz0 + row / nky;
        const bool mirror = kx >= nh;   // K is real: the other half is the conjugate
        if (mirror) {
            kx = n - kx;
            ky = ky ? n - ky : 0;
            kz = kz ? n - kz : 0;
        }
        const double2* K = c.K + (((int64_t)(G.x - 2) * c.n_fam + seq * c.seq_fam) * n * n * nh +
                                  ((int64_t)kz * n + ky) * nh + kx) * N_DISP;
        for (int d = tid; d < N_DISP; d += 32 * CONV_WARPS) {
            double2 v = K[d];
            if (mirror) v.y = -v.y;
            Kt[(d / 49) * KSX + ((d / 7) % 7) * KSY + d % 7] = v;
        }
        for (int i = tid; i < CONV_GROUP * 26; i += 32 * CONV_WARPS) {
            const int s = i / 26, D = i - s * 26;
            nb[s][D] = s < G.z ? c.nbr[(int64_t)(G.y + s) * 26 + D] : c.n_slots;
        }
    }
    __syncthreads();
    const int t0 = warp * NT * 8;   // the warp's first slot in the group
    if (t0 >= G.z) return;
    const int g = lane >> 2, t4 = lane & 3;
    const int64_t fstride = (int64_t)(c.n_slots + 1) * 8;
    const int64_t fo = ((int64_t)seq * c.rows * nkx + f) * fstride;
    const double2* X = c.X + fo + t4;
    const int off_t = (g & 1) * KSX + ((g >> 1) & 1) * KSY + (g >> 2);
    const int off_s = (t4 & 1) * KSX + (t4 >> 1) * KSY;
    const double2* Kl = Kt + 3 * (KSX + KSY + 1) + off_t - off_s;   // source children 4.. are one z further
    auto tiles = [&](auto n_tiles) {
        constexpr int N = n_tiles;
        double acc[N][4];
#pragma unroll
        for (int a = 0; a < N; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
        double2 x[2][N][2];
        auto load = [&](int D, double2 (&v)[N][2]) {
#pragma unroll
            for (int a = 0; a < N; ++a) {
                const double2* q = X + (int64_t)nb[t0 + a * 8 + g][D] * 8;
                v[a][0] = __ldg(q);
                v[a][1] = __ldg(q + 4);
            }
        };
        auto mul = [&](int D, const double2 (&v)[N][2]) {
            int ox, oy, oz;
            neigh_offset(D, ox, oy, oz);
            const double2* Kd = Kl - 2 * (ox * KSX + oy * KSY + oz);
            const double2 k0 = Kd[0], k1 = Kd[-1];
#pragma unroll
            for (int a = 0; a < N; ++a) dmma(acc[a], k0.x, k0.y, v[a][0].x);
#pragma unroll
            for (int a = 0; a < N; ++a) dmma(acc[a], -k0.y, k0.x, v[a][0].y);
#pragma unroll
            for (int a = 0; a < N; ++a) dmma(acc[a], k1.x, k1.y, v[a][1].x);
#pragma unroll
            for (int a = 0; a < N; ++a) dmma(acc[a], -k1.y, k1.x, v[a][1].y);
        };
        load(0, x[0]);
#pragma unroll 1
        for (int D = 0; D < 26; D += 2) {
            load(D + 1, x[1]);
            mul(D, x[0]);
            if (D + 2 < 26) load(D + 2, x[0]);
            mul(D + 1, x[1]);
        }
        double2* Y = c.Y + fo + g;
#pragma unroll
        for (int a = 0; a < N; ++a) {
            const int s = t0 + a * 8 + 2 * t4;
            if (s < G.z) Y[(int64_t)(G.y + s) * 8] = make_double2(acc[a][0], acc[a][2]);
            if (s + 1 < G.z) Y[(int64_t)(G.y + s + 1) * 8] = make_double2(acc[a][1], acc[a][3]);
        }
    };
    if (HALF && G.z - t0 <= 8) tiles(std::integral_constant<int, 1>());
    else tiles(std::integral_constant<int, NT>());
}

// Inverse transform of a slot's children onto the surface points: per kz the x axis straight
// from memory, the y axis, then every surface point's z term, added into the points' sums in
// kz order. The sums start from 0 on the first chunk and from the check potentials after, so
// whole-plane chunks of any number give the same bits. Bound by the reads of Y at large
// sizes. R = 1: the half spectrum, terms kx > 0 doubled, real part kept.
template <int R>
__global__ void __launch_bounds__(256) k_conv_inv(ConvCall c) {
    extern __shared__ double2 sh[];
    const AxisShape a = axis_shape(c);
    const int p = c.p, n = c.n, nh = p, CH = c.CH, nky = c.ky1 - c.ky0;
    const int slot = blockIdx.x, c0 = blockIdx.y * CH, seq = blockIdx.z;
    double2* tw = sh;                          // n
    double2* tz = tw + n;                      // p
    double2* T = tz + p;
    double2* U1 = T + a.MT * a.KS * 32;        // [i][j][SR]
    double2* U2 = U1 + p * p * a.SR;           // [i][ky][SR]
    double* acc = reinterpret_cast<double*>(U2 + p * nky * a.SR);   // [point][CH][R]
    int* pts = reinterpret_cast<int*>(acc + c.n_s * CH * R);        // [point] U1 row and k
    const int nkx = R == 2 ? n : nh;
    const int64_t fstride = (int64_t)(c.n_slots + 1) * 8;
    const double2* Y = c.Y + (int64_t)seq * c.rows * nkx * fstride + (int64_t)slot * 8 + c0;
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int i = tid; i < n; i += nt) tw[i] = c.tw[i];
    for (int i = tid; i < c.n_s; i += nt) pts[i] = c.line_k[i];
    const Balance bal = R == 2 ? balance(c.q_max) : Balance();
    for (int ch = 0; ch < CH; ++ch) {
        const int b = c.child[slot * 8 + c0 + ch];
        const double* src = c.check + seq * c.seq_stride + b * c.box_stride;
        for (int r = 0; r < R; ++r)
            for (int s = tid; s < c.n_s; s += nt)
                acc[(c.pos[s] * CH + ch) * R + r] = c.first || b < 0 ? 0.0 : src[r * c.ld + s] * (R == 2 ? bal.up[r] : 1.0);
    }
    __syncthreads();
    axis_table(a, tw, T);
    for (int kz = c.kz0; kz < c.kz1; ++kz) {
        __syncthreads();   // T is there; the previous plane's points have read tz and U1
        if (tid < p) tz[tid] = tw[tid * kz % n];
        const double2* y = Y + (int64_t)(kz - c.kz0) * nky * nkx * fstride;
        axis_inverse(a, nky, T, [&](int ky, int ch, int k, double2& P, double2& M) {   // x, from memory
            const double2* q = y + (int64_t)ky * nkx * fstride + ch;
            const double2 v = __ldg(q + k * fstride);
            if (k == 0) {
                P = v;
            } else if (R == 2) {
                const double2 m = __ldg(q + (n - k) * fstride);
                P = make_double2(v.x + m.x, v.y + m.y);
                M = make_double2(v.x - m.x, v.y - m.y);
            } else {
                P = M = make_double2(2.0 * v.x, 2.0 * v.y);
            }
        }, [&](int ky, int ch, int i, double2 u) { U2[(i * nky + ky) * a.SR + ch] = u; });
        __syncthreads();
        if (R == 2 || nky == n) {   // y (complex sequences come in whole planes)
            axis_inverse(a, p, T, [&](int i, int ch, int k, double2& P, double2& M) {
                const double2* q = U2 + i * n * a.SR + ch;
                const double2 v = q[k * a.SR];
                if (k == 0) {
                    P = v;
                } else {
                    const double2 m = q[(n - k) * a.SR];
                    P = make_double2(v.x + m.x, v.y + m.y);
                    M = make_double2(v.x - m.x, v.y - m.y);
                }
            }, [&](int i, int ch, int j, double2 u) { U1[(i * p + j) * a.SR + ch] = u; });
        } else {   // some rows of a plane (a workspace under one plane): their sums unfolded
            for (int it = tid; it < p * p * CH; it += nt) {
                const int ch = it & (CH - 1), line = it >> a.lch, i = line / p, j = line - i * p;
                double re = 0.0, im = 0.0;
                for (int ky = 0; ky < nky; ++ky) {
                    const double2 v = U2[(i * nky + ky) * a.SR + ch], w = tw[(c.ky0 + ky) * j % n];
                    re = fma(v.x, w.x, fma(-v.y, w.y, re));
                    im = fma(v.y, w.x, fma(v.x, w.y, im));
                }
                U1[line * a.SR + ch] = make_double2(re, im);
            }
        }
        __syncthreads();
        for (int it = tid; it < c.n_s * CH; it += nt) {   // z: each surface point's own term
            const int ch = it & (CH - 1), lk = pts[it >> a.lch];
            const double2 v = U1[(lk >> 8) * a.SR + ch], w = tz[lk & 255];
            if (R == 2) {
                double2* q = reinterpret_cast<double2*>(acc) + it;
                double2 t = *q;
                t.x = fma(v.x, w.x, fma(-v.y, w.y, t.x));
                t.y = fma(v.y, w.x, fma(v.x, w.y, t.y));
                *q = t;
            } else {
                acc[it] = fma(v.x, w.x, fma(-v.y, w.y, acc[it]));
            }
        }
    }
    __syncthreads();
    for (int ch = 0; ch < CH; ++ch) {
        const int b = c.child[slot * 8 + c0 + ch];
        if (b < 0) continue;
        double* dst = c.check + seq * c.seq_stride + b * c.box_stride;
        for (int r = 0; r < R; ++r)
            for (int s = tid; s < c.n_s; s += nt)
                dst[r * c.ld + s] = R == 1 || bal.any[r] ? acc[(c.pos[s] * CH + ch) * R + r] * (R == 2 ? bal.down[r] : 1.0)
                                                         : 0.0;
    }
}

// shared memory of the transform kernels for CH children and nky rows of a plane
size_t transform_smem(int p, int n_s, int R, int CH, int nky) {
    const size_t table = (size_t)((p + 7) / 8) * ((p + 3) / 4) * 32;
    return ((size_t)(3 * p - 1) + table + (size_t)(CH + 2) * (p * p + p * nky)) * sizeof(double2) +
           (size_t)n_s * CH * R * sizeof(double) + (size_t)n_s * sizeof(int);
}

// The transforms' working set when the plan owns it: chunks of whole planes up to this
// size (1e6 points, p = 8: 8 GiB of spectra in all, four chunks; larger chunks measured
// the same, smaller ones add launches)
constexpr size_t CONV_WS = (size_t)2 << 30;

int64_t chunk_values(const hfmm_plan* P, int nkx, int nf) {   // values of one (ky, kz) row
    return (int64_t)nkx * (P->conv.n_slots + 1) * 8 * nf;
}

}  // namespace

// The surface as lattice points: false when the points given are not the p x p x p
// lattice's surface (then the dense tables serve).
bool conv_surface(hfmm_plan* P, const double* equiv) {
    ConvPlan& C = P->conv;
    C.ok = false;
    const int p = P->p, n_s = P->n_s;
    if (p < 2 || p > 255) return false;
    double r0 = 0.0;
    for (int i = 0; i < 3 * n_s; ++i) r0 = std::max(r0, std::fabs(equiv[i]));
    if (!(r0 > 0.0) || !std::isfinite(r0)) return false;
    C.spacing = 2.0 * r0 / (p - 1);
    std::vector<int32_t> at((size_t)p * p * p, -1);
    for (int s = 0; s < n_s; ++s) {
        int g[3];
        bool face = false;
        for (int a = 0; a < 3; ++a) {
            const double t = (equiv[3 * s + a] + r0) / C.spacing;
            g[a] = (int)std::lround(t);
            if (!(std::fabs(t - g[a]) < 1e-11) || g[a] < 0 || g[a] >= p) return false;
            face = face || g[a] == 0 || g[a] == p - 1;
        }
        int32_t& cell = at[((size_t)g[0] * p + g[1]) * p + g[2]];
        if (!face || cell >= 0) return false;
        cell = s;
    }
    // points in line order (x, y lattice column, then z): every surface cell must be there
    std::vector<int32_t> pos(n_s), off((size_t)p * p), lk(n_s);
    int e = 0;
    for (int i = 0; i < p; ++i)
        for (int j = 0; j < p; ++j) {
            off[(size_t)i * p + j] = e;
            const bool edge = i == 0 || j == 0 || i == p - 1 || j == p - 1;
            for (int k = 0; k < p; k += (edge || p == 2) ? 1 : p - 1) {
                const int s = at[((size_t)i * p + j) * p + k];
                if (s < 0 || e >= n_s) return false;
                pos[s] = e;
                lk[e++] = ((i * p + j) << 8) | k;
            }
        }
    if (e != n_s) return false;
    // at least one child per CTA must fit
    if (transform_smem(p, n_s, 2, 1, 2 * p - 1) > SMEM_MAX) return false;
    C.n = 2 * p - 1;
    std::vector<double> tw(2 * C.n);
    for (int i = 0; i < C.n; ++i) {
        const long double a = 2.0L * 3.141592653589793238462643383279502884L * i / C.n;
        tw[2 * i] = (double)std::cos(a);
        tw[2 * i + 1] = (double)std::sin(a);
    }
    auto up = [](auto& buf, const auto& h) {
        buf.alloc(h.size());
        HFMM_CUDA(cudaMemcpy(buf.p, h.data(), h.size() * sizeof(h[0]), cudaMemcpyHostToDevice));
    };
    up(C.pos, pos);
    up(C.line_off, off);
    up(C.line_k, lk);
    up(C.tw, tw);
    C.tables = false;
    C.ok = true;
    return true;
}

// Spectra of every level's and family's 316 displacements, half of the frequencies (kx <=
// n / 2; K is real), [level - 2][family][kz][ky][kx][343].
void conv_tables(hfmm_plan* P) {
    ConvPlan& C = P->conv;
    const int n = C.n, nh = (n + 1) / 2, nl = P->md - 1;
    const int64_t per = (int64_t)n * n * nh * N_DISP;
    C.K.alloc((size_t)std::max(nl, 1) * P->n_fam * per * 2);
    DevBuf<double> a, b;
    a.alloc((size_t)n * n * n * N_DISP);
    b.alloc((size_t)per * 2);
    DevBuf<double> t;
    t.alloc((size_t)per * 2);
    const double2* tw = reinterpret_cast<const double2*>(C.tw.p);
    auto blocks = [](int64_t m) { return (unsigned)ceil_div(m, 256); };
    for (int l = 2; l <= P->md; ++l)
        for (int f = 0; f < P->n_fam; ++f) {
            const double s = P->extent * std::ldexp(1.0, -(l + 1));
            const int64_t cells = (int64_t)n * n * n * N_DISP;
            HFMM_LAUNCH(k_conv_gen, blocks(cells), 256, 0, 0, P->p, n, C.spacing, s, P->k,
                        P->yukawa ? 2 : f, a.p);
            double2* tp = reinterpret_cast<double2*>(t.p);
            double2* bp = reinterpret_cast<double2*>(b.p);
            double2* K = reinterpret_cast<double2*>(C.K.p) + ((int64_t)(l - 2) * P->n_fam + f) * per;
            HFMM_LAUNCH(k_conv_axis<true>, blocks(per), 256, 0, 0, a.p, n, nh, (int64_t)N_DISP, per, tw, 1.0, tp);
            HFMM_LAUNCH(k_conv_axis<false>, blocks(per), 256, 0, 0, t.p, n, n, (int64_t)nh * N_DISP, per, tw,
                        1.0, bp);
            HFMM_LAUNCH(k_conv_axis<false>, blocks(per), 256, 0, 0, b.p, n, n, (int64_t)n * nh * N_DISP, per,
                        tw, 1.0 / ((double)n * n * n), K);
        }
    HFMM_CUDA(cudaDeviceSynchronize());
    C.tables = true;
}

// Slots, neighbour lists and groups of the current tree.
void conv_schedule(hfmm_plan* P) {
    ConvPlan& C = P->conv;
    std::vector<int32_t> slot_of(P->nb, -1), child;
    std::vector<int4> groups;
    int n_slots = 0;
    for (int l = 2; l <= P->md; ++l) {
        const int first = n_slots;
        for (int b = P->level_lo[l]; b < P->level_hi[l]; ++b) {
            int32_t& s = slot_of[P->h_p_id[b]];
            if (s < 0) {
                s = n_slots++;
                child.insert(child.end(), 8, -1);
            }
            child[(size_t)s * 8 + (P->h_m_id[b] & 7ull)] = b;
        }
        for (int s = first; s < n_slots; s += CONV_GROUP)
            groups.push_back(make_int4(l, s, std::min(CONV_GROUP, n_slots - s), 0));
    }
    C.n_slots = n_slots;
    C.n_groups = (int)groups.size();
    int64_t warps = 0, halves = 0;
    for (const int4& g : groups) {
        warps += ceil_div(g.z, 8 * NT);
        halves += (g.z - 1) % (8 * NT) < 8;
    }
    C.half = halves * 16 >= warps;
    if (!n_slots) return;
    auto up = [](auto& buf, const auto& h) {
        buf.alloc(h.size());
        HFMM_CUDA(cudaMemcpy(buf.p, h.data(), h.size() * sizeof(h[0]), cudaMemcpyHostToDevice));
    };
    DevBuf<int32_t> so;
    up(so, slot_of);
    up(C.child, child);
    up(C.groups, groups);
    C.nbr.alloc((size_t)n_slots * 26);
    HFMM_LAUNCH(k_conv_nbr, (unsigned)ceil_div((int64_t)n_slots * 26, 256), 256, 0, 0, C.child.p,
                P->m2l_src.p, P->p_id.p, so.p, n_slots, C.nbr.p);
    HFMM_CUDA(cudaDeviceSynchronize());
}

// The plan's own workspace (a streamed plan's is P->ws): X and Y of as many whole planes as the
// limit holds; where not one fits, the limit (one family or some rows of a plane at a time).
// Taken after every other buffer of the plan, and smaller where the device is nearly full, one
// row of one family at least: chunks cost time (1e6 points, p = 4: 7.5 ms with 2 GiB, 9.4 with
// 64 MiB), but a plan that otherwise fits is not refused for them.
void conv_workspace(hfmm_plan* P) {
    ConvPlan& C = P->conv;
    if (!C.on || !C.n_slots || P->streamed) {
        C.ws.release();
        return;
    }
    const size_t row = 2 * (size_t)chunk_values(P, C.n, 1) * sizeof(double2);
    // two complex sequences, or one family's two real ones of (n + 1) / 2 values a row
    const size_t plane = (P->n_fam > 1 ? 2 * row : row / C.n * (C.n + 1)) * C.n;
    const size_t planes = std::min<size_t>(C.n, CONV_WS / plane);
    const size_t want = (planes ? plane * planes : std::max(row, CONV_WS)) / sizeof(double);
    if (C.ws.n < want) C.ws.alloc_between(row / sizeof(double), want);
}

bool conv_fits(const hfmm_plan* P) {   // a streamed plan's workspace must hold one row
    if (!P->streamed) return true;
    return 2 * (size_t)chunk_values(P, P->conv.n, 1) * sizeof(double2) <= stream_ws_bytes(P);
}

void conv_m2l(hfmm_plan* P, int R, int64_t fam_stride, cudaStream_t s) {
    const ConvPlan& C = P->conv;
    if (!C.n_slots) return;
    ConvCall c{};
    c.p = P->p;
    c.n = C.n;
    c.n_s = P->n_s;
    c.ld = P->ld;
    c.n_slots = C.n_slots;
    c.n_groups = C.n_groups;
    c.child = C.child.p;
    c.nbr = C.nbr.p;
    c.pos = C.pos.p;
    c.line_off = C.line_off.p;
    c.line_k = C.line_k.p;
    c.groups = C.groups.p;
    c.tw = reinterpret_cast<const double2*>(C.tw.p);
    c.n_fam = P->n_fam;
    c.box_stride = (int64_t)R * P->ld;
    c.q_max = P->q_max.p;
    const int n = C.n;
    double* ws = P->streamed ? static_cast<double*>(P->ws) : C.ws.p;
    const size_t ws_values = (P->streamed ? P->ws_bytes : C.ws.n * sizeof(double)) / sizeof(double2);
    // Sequences: the families, or their charge columns as real ones: of a single family, and
    // where the workspace holds no plane of a complex one (every row of a chunk pays the whole
    // forward y axis, and a real plane is half as large: streamed 2e5 points, p = 4, depth 5,
    // 12.95 ms as complex sequences, 9.10 as real ones, 10.86 from dense tables)
    const bool columns = R == 2 && (P->n_fam == 1 || 2 * (size_t)chunk_values(P, n, 1) * n > ws_values);
    const int n_seq = columns ? 2 * P->n_fam : P->n_fam;
    if (columns) R = 1;
    c.seq_fam = P->n_fam > 1;
    c.seq_stride = c.seq_fam ? fam_stride : P->ld;
    const int nkx = R == 2 ? n : (n + 1) / 2;
    // sequences together when a plane of both fits, else one after the other; whole planes
    // of frequencies, or rows of one plane where not even one fits
    int nf = n_seq;
    if ((columns && P->n_fam > 1) || 2 * (size_t)chunk_values(P, nkx, nf) * n > ws_values) nf = 1;
    const size_t row = 2 * (size_t)chunk_values(P, nkx, nf);
    const int planes = (int)std::min<size_t>(n, ws_values / (row * n));
    const int rows = planes ? n : (int)std::min<size_t>(n, ws_values / row);
    if (rows < 1) throw Error{HFMM_ERR_STATE, "convolution M2L: workspace too small"};
    const int dz = std::max(planes, 1);
    const int PT = 256;
    // children per CTA of the transforms: eight where four CTAs an SM remain (the latency of
    // their short stages is the rest of the time), else four (half the 128-byte lines) while
    // those fit at all. 1e6 points, p = 8, forward / inverse: 3.45 / 4.78 ms with eight,
    // 3.33 / 3.99 with four, 5.8 with two; p = 6 (36 KB with eight): 127 / 155 us and 142 / 173
    int CH = 8;
    while (CH > 4 && transform_smem(c.p, c.n_s, R, CH, rows) > SMEM_MAX / 4) CH /= 2;
    while (CH > 1 && transform_smem(c.p, c.n_s, R, CH, rows) > SMEM_MAX) CH /= 2;
    // few slots: fewer children a CTA on the inverse (its kz sum stays in one CTA), segments of
    // kz on the forward, towards three CTAs an SM (72 slots, p = 8: 81 and 98 us with one)
    const int64_t want = 3 * sm_count();
    int CHi = CH;
    while (CHi > 1 && (int64_t)c.n_slots * (8 / CHi) * nf < want) CHi /= 2;
    const int segs = (int)std::max<int64_t>(1, want / ((int64_t)(c.n_slots + 1) * (8 / CH) * nf));
    const size_t smem = transform_smem(c.p, c.n_s, R, CH, rows), smem_i = transform_smem(c.p, c.n_s, R, CHi, rows);
    using Kernel = void (*)(ConvCall);
    Kernel fwd = nullptr;
    switch ((c.p + 3) / 4) {
        case 1: fwd = R == 2 ? k_conv_fwd<2, 1> : k_conv_fwd<1, 1>; break;
        case 2: fwd = R == 2 ? k_conv_fwd<2, 2> : k_conv_fwd<1, 2>; break;
        case 3: fwd = R == 2 ? k_conv_fwd<2, 3> : k_conv_fwd<1, 3>; break;
        default: fwd = R == 2 ? k_conv_fwd<2, 0> : k_conv_fwd<1, 0>; break;
    }
    const Kernel inv = R == 2 ? k_conv_inv<2> : k_conv_inv<1>;
    allow_smem(fwd);
    allow_smem(inv);
    auto mul = C.half ? k_conv_mul<true> : k_conv_mul<false>;
    for (int f = 0; f < n_seq; f += nf) {
        const int fam = columns ? f / 2 : f;
        const int64_t off = fam * fam_stride + (columns ? f % 2 * (int64_t)P->ld : 0);
        c.dens = P->equiv.p + off;
        c.check = P->check.p + off;
        c.K = reinterpret_cast<const double2*>(C.K.p) + (int64_t)fam * n * n * ((n + 1) / 2) * N_DISP;
        c.first = 1;
        for (int kz = 0; kz < n; kz += dz)
            for (int ky = 0; ky < n; ky += rows) {
                c.kz0 = kz;
                c.kz1 = std::min(n, kz + dz);
                c.ky0 = ky;
                c.ky1 = std::min(n, ky + rows);
                c.rows = (c.kz1 - c.kz0) * (c.ky1 - c.ky0);
                c.X = reinterpret_cast<double2*>(ws);
                c.Y = c.X + (int64_t)c.rows * chunk_values(P, nkx, nf);
                c.CH = CH;
                c.n_seg = std::min(segs, c.kz1 - c.kz0);
                HFMM_LAUNCH(fwd, dim3((unsigned)(c.n_slots + 1), (unsigned)(8 / CH), (unsigned)(nf * c.n_seg)), PT,
                            smem, s, c);
                HFMM_LAUNCH(mul, dim3((unsigned)((int64_t)c.rows * nkx * c.n_groups), (unsigned)nf),
                            32 * CONV_WARPS, 0, s, c, nkx);
                c.CH = CHi;
                HFMM_LAUNCH(inv, dim3((unsigned)c.n_slots, (unsigned)(8 / CHi), (unsigned)nf), PT, smem_i, s, c);
                c.first = 0;
            }
    }
}

}  // namespace hfmm
