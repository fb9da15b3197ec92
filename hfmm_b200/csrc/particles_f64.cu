// FP64 particle kernels of the plain path: P2M, P2L, L2P, M2P, P2P, the charge
// gather into leaf-major order and the final complex combine.
//
// Every kernel evaluates both Helmholtz components from one sincos per pair
// (family 0: cos(kr)/r, family 1: sin(kr)/r, HFMM.py:25-27) for R charge
// columns at once, and optionally the field -grad phi with the weights
// (cos + kr sin)/r^3 and (sin - kr cos)/r^3 (HFMM.py:29-40).
// Particles are in Morton-sorted order, so each leaf is a contiguous slice of
// the SoA position arrays (the role of _build_padded, near.py:589-598, without
// the padded copy).
#include "hfmm_internal.cuh"
#include "particles.cuh"

#include <algorithm>
#include <type_traits>

namespace hfmm {

namespace {

constexpr int STAGE = 128;   // particles staged in shared memory per pass

// Check potentials of one leaf at its upward check surface (phases.py:118-124).
// Also P2L (phases.py:1755-1769) when `surf` is the equivalent surface of a
// target box and the sources are the particles of its X-list leaves.
template <int NF, int R, bool FAST>
__global__ void __launch_bounds__(512) k_surface_from_particles(
    EvalView v, const int32_t* __restrict__ tgt_boxes, const int32_t* __restrict__ off,
    const int32_t* __restrict__ srcs, const double* __restrict__ surf, int only_level,
    double* check, int64_t fam_stride, int accumulate) {
    __shared__ double sx[STAGE], sy[STAGE], sz[STAGE], sq[R][STAGE];
    const int row = blockIdx.x;
    const int b = tgt_boxes[row];
    const int lvl = v.lvls[b];
    if (lvl < 2 || (only_level >= 0 && lvl != only_level)) return;
    const double h = v.hbox[b];
    const double cx = v.centre[b], cy = v.centre[v.nb + b], cz = v.centre[2 * v.nb + b];
    const int e0 = off ? off[row] : 0, e1 = off ? off[row + 1] : 1;
    for (int j0 = 0; j0 < v.n_s; j0 += blockDim.x) {
        const int j = j0 + threadIdx.x;
        const bool jok = j < v.n_s;
        double px = 0, py = 0, pz = 0;
        if (jok) {
            px = surf[j] * h + cx;
            py = surf[v.n_s + j] * h + cy;
            pz = surf[2 * v.n_s + j] * h + cz;
        }
        double acc[NF][R];
#pragma unroll
        for (int f = 0; f < NF; ++f)
#pragma unroll
            for (int r = 0; r < R; ++r) acc[f][r] = 0.0;
        for (int e = e0; e < e1; ++e) {
            const int sb = srcs ? srcs[e] : b;
            const int s0 = v.leaf_start[sb], cnt = v.counts[sb];
            for (int p0 = 0; p0 < cnt; p0 += STAGE) {
                __syncthreads();
                for (int i = threadIdx.x; i < STAGE && p0 + i < cnt; i += blockDim.x) {
                    int64_t gi = s0 + p0 + i;
                    sx[i] = v.pos_s[gi];
                    sy[i] = v.pos_s[v.n + gi];
                    sz[i] = v.pos_s[2 * v.n + gi];
#pragma unroll
                    for (int r = 0; r < R; ++r) sq[r][i] = v.q_s[r * v.n + gi];
                }
                __syncthreads();
                if (jok) {
                    const int np = min(STAGE, cnt - p0);
#pragma unroll 2
                    for (int i = 0; i < np; ++i) {
                        double dx = px - sx[i], dy = py - sy[i], dz = pz - sz[i];
                        double r2 = dx * dx + dy * dy + dz * dz;
                        double ir = FAST ? rsqrt_normal(r2) : rsqrt(r2);
                        double sn, cs;
                        if (FAST) sincos_reduced64(v.k * (r2 * ir), &sn, &cs);
                        else kernel_pair64(v.yukawa, v.k * (r2 * ir), &sn, &cs);
                        double wc = cs * ir, ws = sn * ir;
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            acc[0][r] += sq[r][i] * wc;
                            if (NF == 2) acc[NF - 1][r] += sq[r][i] * ws;
                        }
                    }
                }
            }
        }
        if (jok) {
#pragma unroll
            for (int f = 0; f < NF; ++f)
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    double* o = check + f * fam_stride + ((int64_t)b * R + r) * v.ld + j;
                    *o = accumulate ? *o + acc[f][r] : acc[f][r];
                }
        }
    }
}

// Particle potentials (and field) from surface densities: L2P (phases.py:1571-1582,
// downward equivalent surface R_CHECK of the leaf itself) and M2P (phases.py:1101-1140,
// upward equivalent surface R_EQUIV of each W-list source box). One CTA per target leaf
// and 16 of its particles; a group of GL lanes shares a particle, each lane taking every
// GL-th surface point, and reduces over GL lanes only. Bound by FP64 operations (56 a pair
// with complex charges and the field) once the work is spread: a W list has up to four
// times the mean length and a leaf three times the mean count, so a CTA per leaf left one
// long CTA running (M2P of 2e5 adaptive points, 28 % of the FP64 rate).
constexpr int GL = 8, L2P_THREADS = 128, L2P_CHUNK = L2P_THREADS / GL;
template <int NF, int R, bool FIELD, bool FAST>
__global__ void __launch_bounds__(L2P_THREADS) k_particles_from_surface(
    EvalView v, const int32_t* __restrict__ tgt_leaves, const int32_t* __restrict__ off,
    const int32_t* __restrict__ srcs, const double* __restrict__ surf,
    const double* __restrict__ dens, int64_t fam_stride, int n_chunk, double* pot, double* fld) {
    extern __shared__ double sh[];
    double* dn = sh;                          // [NF][R][n_s]
    double* ex = sh + NF * R * v.n_s;         // [3][n_s]
    const int row = blockIdx.x / n_chunk;
    const int t = tgt_leaves[row];
    if (v.lvls[t] < 2 && !off) return;        // L2P: no local expansion above level 2
    const int s0 = v.leaf_start[t], cnt = v.counts[t];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int grp = lane / GL, gl = lane % GL;   // particle slot of the warp, lane within it
    const int e0 = off ? off[row] : 0, e1 = off ? off[row + 1] : 1;
    constexpr int NC = PairSums<NF, R, FIELD>::NC, NA = PairSums<NF, R, FIELD>::N;
    for (int i0 = blockIdx.x % n_chunk * L2P_CHUNK; i0 < cnt; i0 += n_chunk * L2P_CHUNK) {
        const int i = i0 + warp * (32 / GL) + grp;
        const bool act = i < cnt;
        const int64_t gi = s0 + (act ? i : 0);
        const double x = v.pos_s[gi], y = v.pos_s[v.n + gi], z = v.pos_s[2 * v.n + gi];
        double acc[NA];
#pragma unroll
        for (int q = 0; q < NA; ++q) acc[q] = 0.0;
        for (int e = e0; e < e1; ++e) {
            const int sb = srcs ? srcs[e] : t;
            const double h = v.hbox[sb];
            const double c[3] = {v.centre[sb], v.centre[v.nb + sb], v.centre[2 * v.nb + sb]};
            if (e1 - e0 > 1 || i0 < L2P_CHUNK * n_chunk) {   // a single source stays for every chunk
                __syncthreads();
                for (int j = threadIdx.x; j < v.n_s; j += L2P_THREADS) {
#pragma unroll
                    for (int a = 0; a < 3; ++a) ex[a * v.n_s + j] = surf[a * v.n_s + j] * h + c[a];
#pragma unroll
                    for (int f = 0; f < NF; ++f)
#pragma unroll
                        for (int r = 0; r < R; ++r)
                            dn[(f * R + r) * v.n_s + j] = dens[f * fam_stride + ((int64_t)sb * R + r) * v.ld + j];
                }
                __syncthreads();
            }
            if (act)
#pragma unroll 2
                for (int j = gl; j < v.n_s; j += GL) {
                    const double dx = x - ex[j], dy = y - ex[v.n_s + j], dz = z - ex[2 * v.n_s + j];
                    const double r2 = dx * dx + dy * dy + dz * dz;
                    double d[NF][R];
#pragma unroll
                    for (int f = 0; f < NF; ++f)
#pragma unroll
                        for (int r = 0; r < R; ++r) d[f][r] = dn[(f * R + r) * v.n_s + j];
                    pair64<NF, R, FIELD, FAST>(v.yukawa, v.k, dx, dy, dz, r2, d, acc);
                }
        }
#pragma unroll
        for (int q = 0; q < NA; ++q)
#pragma unroll
            for (int o = GL / 2; o > 0; o >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
        if (gl == 0 && act) {
#pragma unroll
            for (int q = 0; q < NC; ++q) pot[q * v.n + gi] += acc[q];
            if (FIELD)
#pragma unroll
                for (int q = 0; q < NC * 3; ++q) fld[q * v.n + gi] += acc[NC + q];
        }
    }
}

// Near field over the U list + self pair of each target leaf (near.py:193-312),
// with the "pair" coincidence floor (near.py:252-261):
// d2 <= (16 eps)^2 (rmax_t + rmax_s)^2 counts as coincident and contributes 0.
// Bound by FP64 operations (54 a pair with complex charges and the field). One CTA per
// target leaf, its four warps taking every fourth source leaf, 32 sources staged at a time
// in the warp's own slice; 32 / G targets a pass with G lanes each on the sources, G chosen
// per leaf (p2p_lanes). One thread per target of a 128-thread CTA before left most lanes
// idle on leaves of 15 to 60 points. The warps' sums are added in warp order.
// ROOT (EvalView::root): the last bit of r matters where k r is large. One leaf of 1,200 points
// in a unit cube, error of the potential without / with it / with sqrt and a division: k = 10
// 7.4 / 7.0 / 9.6e-16, 30 1.30 / 1.11 / 1.31e-15, 100 3.92 / 3.26 / 3.33e-15, 1000 3.82 / 3.15 /
// 3.15e-14; it costs 5 % of the smallest call and 0.8 % of 1e6 points, p = 8 (13 % of a call that
// the general form's near field bounds), so it runs from k x extent = 25 on.
constexpr int P2P_WARPS = 4;
template <int NF, int R, bool FIELD, bool FAST, bool ROOT>
__global__ void __launch_bounds__(32 * P2P_WARPS) k_p2p(EvalView v, const int32_t* __restrict__ leaves,
                                                      const int32_t* __restrict__ off,
                                                      const int32_t* __restrict__ srcs, double* pot,
                                                      double* fld) {
    constexpr int NC = PairSums<NF, R, FIELD>::NC, NA = PairSums<NF, R, FIELD>::N;
    __shared__ double stage[P2P_WARPS][3 + R][32];
    __shared__ double part[P2P_WARPS - 1][NA][32];
    const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = leaves[row];
    const int s0t = v.leaf_start[t], cnt_t = v.counts[t];
    const double rt = v.rmax[t];
    const int e0 = off[row], e1 = off[row + 1];
    const double C16 = 1.2621774483536189e-29;   // (16 * 2^-52)^2
    const int G = p2p_lanes(cnt_t), TG = 32 / G;
    const int tg = lane & (TG - 1), sub = lane / TG;
    double(&st)[3 + R][32] = stage[warp];
    for (int i0 = 0; i0 < cnt_t; i0 += TG) {
        const int i = i0 + tg;
        const bool act = i < cnt_t;
        const int64_t gt = s0t + (act ? i : 0);
        const double x = v.pos_s[gt], y = v.pos_s[v.n + gt], z = v.pos_s[2 * v.n + gt];
        double acc[NA];
#pragma unroll
        for (int q = 0; q < NA; ++q) acc[q] = 0.0;
        for (int e = e0 + warp; e < e1; e += P2P_WARPS) {
            const int sb = srcs[e];
            const int s0 = v.leaf_start[sb], cnt = v.counts[sb];
            const double rs = __dadd_rn(rt, v.rmax[sb]);
            const double thr = __dmul_rn(C16, __dmul_rn(rs, rs));
            for (int p0 = 0; p0 < cnt; p0 += 32) {
                const int np = min(32, cnt - p0);
                __syncwarp();
                if (lane < np) {
                    const int64_t gi = s0 + p0 + lane;
                    st[0][lane] = v.pos_s[gi];
                    st[1][lane] = v.pos_s[v.n + gi];
                    st[2][lane] = v.pos_s[2 * v.n + gi];
#pragma unroll
                    for (int r = 0; r < R; ++r) st[3 + r][lane] = v.q_s[r * v.n + gi];
                }
                __syncwarp();
                // a coincident source counts as one at zero charge
                auto sources = [&](auto fast) {
                    constexpr bool F = decltype(fast)::value;
#pragma unroll 2
                    for (int k = sub; k < np; k += G) {
                        const double dx = x - st[0][k], dy = y - st[1][k], dz = z - st[2][k];
                        const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
                        const bool far = d2 > thr;
                        double q[NF][R];
#pragma unroll
                        for (int f = 0; f < NF; ++f)
#pragma unroll
                            for (int r = 0; r < R; ++r) q[f][r] = far ? st[3 + r][k] : 0.0;
                        pair64<NF, R, FIELD, F, ROOT>(v.yukawa, v.k, dx, dy, dz, far ? d2 : 1.0, q, acc);
                    }
                };
                if (FAST && thr >= 1e-290) sources(std::true_type());
                else sources(std::false_type());
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
            for (int w = 0; w < P2P_WARPS - 1; ++w)
#pragma unroll
                for (int q = 0; q < NA; ++q) acc[q] += part[w][q][lane];
#pragma unroll
            for (int q = 0; q < NC; ++q) pot[q * v.n + gt] = acc[q];
            if (FIELD)
#pragma unroll
                for (int q = 0; q < NC * 3; ++q) fld[q * v.n + gt] = acc[NC + q];
        }
    }
}

// Charges in leaf-major order; q_max (nullable) is raised to the bits of the largest real and
// imaginary magnitude (infinities and NaN the largest bits there are)
__global__ void k_gather_q(int64_t n, const int32_t* __restrict__ sidx, const double* __restrict__ q_re,
                           const double* __restrict__ q_im, double* q_s, unsigned long long* q_max) {
    __shared__ unsigned long long most[2];
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    unsigned long long m[2] = {0, 0};
    if (i < n) {
        const int64_t o = sidx[i];
        const double re = q_re[o], im = q_im ? q_im[o] : 0.0;
        q_s[i] = re;
        if (q_im) q_s[n + i] = im;
        m[0] = (unsigned long long)__double_as_longlong(re) & ~(1ull << 63);
        m[1] = (unsigned long long)__double_as_longlong(im) & ~(1ull << 63);
    }
    if (!q_max) return;
    if (threadIdx.x < 2) most[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, m[c], o);
            m[c] = v > m[c] ? v : m[c];
        }
        if ((threadIdx.x & 31) == 0 && m[c]) atomicMax(&most[c], m[c]);
    }
    __syncthreads();
    if (threadIdx.x < 2 && most[threadIdx.x]) atomicMax(q_max + threadIdx.x, most[threadIdx.x]);
}

// The particles' sums, back to input order
template <int NC, bool FIELD>
__global__ void k_combine(int64_t n, const int32_t* __restrict__ sidx, const double* __restrict__ pot,
                          const double* __restrict__ fld, double* phi, double* E) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    int64_t o = sidx[i];
    phi[2 * o] = pot[i];
    phi[2 * o + 1] = NC == 2 ? pot[n + i] : 0.0;
    if (FIELD) {
        for (int a = 0; a < 3; ++a) {
            E[(o * 3 + a) * 2] = fld[a * n + i];
            E[(o * 3 + a) * 2 + 1] = NC == 2 ? fld[(3 + a) * n + i] : 0.0;
        }
    }
}

inline int nblk(int64_t n, int t) { return (int)std::max<int64_t>(1, ceil_div(n, t)); }

// threads of a surface kernel: one per surface point in as few passes as possible
// (n_s = 296 at p = 8 takes 320 threads in one pass, not 256 + 40 in two)
inline int surface_threads(int n_s) {
    const int passes = (int)ceil_div(n_s, 512);
    return (int)std::min<int64_t>(512, round_up(ceil_div(n_s, passes), 32));
}

template <int NF, int R, bool FIELD, bool FAST>
void particles_impl(const ParticlePass& p, cudaStream_t s) {
    const EvalView& v = p.v;
    switch (p.op) {
        case ParticleOp::P2M:
            HFMM_LAUNCH((k_surface_from_particles<NF, R, FAST>), p.nrows, surface_threads(v.n_s), 0, s, v,
                        p.rows, p.off, p.srcs, p.surf, -1, p.out, p.fam_stride, 0);
            break;
        case ParticleOp::P2L:
            HFMM_LAUNCH((k_surface_from_particles<NF, R, FAST>), p.nrows, surface_threads(v.n_s), 0, s, v,
                        p.rows, p.off, p.srcs, p.surf, p.level, p.out, p.fam_stride, 1);
            break;
        case ParticleOp::L2P:
        case ParticleOp::M2P: {
            size_t smem = (size_t)(NF * R + 3) * v.n_s * sizeof(double);
            auto kern = k_particles_from_surface<NF, R, FIELD, FAST>;
            allow_smem(kern);
            // M2P, and L2P of few leaves (under two waves of CTAs): the chunks of a leaf in CTAs
            // of their own, up to eight. L2P of many leaves: one CTA a leaf, which then loads its
            // densities once (1e6 points, p = 8: 1.56 against 1.80 ms; 512 leaves: 63 against 51 us)
            const bool spread = p.off || p.nrows < 2 * 7 * sm_count();
            const int nch = spread ? (int)std::min<int64_t>(8, ceil_div(std::max(p.maxleaf, 1), L2P_CHUNK)) : 1;
            HFMM_LAUNCH(kern, (unsigned)(p.nrows * nch), L2P_THREADS, smem, s, v, p.rows, p.off, p.srcs, p.surf,
                        p.dens, p.fam_stride, nch, p.pot, p.fld);
            break;
        }
        case ParticleOp::P2P:
            if (v.root)
                HFMM_LAUNCH((k_p2p<NF, R, FIELD, FAST, true>), p.nrows, 32 * P2P_WARPS, 0, s, v, p.rows, p.off, p.srcs,
                            p.pot, p.fld);
            else
                HFMM_LAUNCH((k_p2p<NF, R, FIELD, FAST, false>), p.nrows, 32 * P2P_WARPS, 0, s, v, p.rows, p.off, p.srcs,
                            p.pot, p.fld);
            break;
        case ParticleOp::COMBINE:
            HFMM_LAUNCH((k_combine<PairSums<NF, R, FIELD>::NC, FIELD>), nblk(v.n, 256), 256, 0, s, v.n, p.rows, p.pot,
                        p.fld, p.phi, p.E);
            break;
    }
}

template <int NF, int R, bool FIELD>
void particles_mode(const ParticlePass& p, cudaStream_t s) {
    if (NF == 2 && p.v.fast) particles_impl<NF, R, FIELD, NF == 2>(p, s);
    else particles_impl<NF, R, FIELD, false>(p, s);
}

}  // namespace

void gather_charges(int64_t n, const int32_t* sidx, const double* q_re, const double* q_im,
                    double* q_s, unsigned long long* q_max, cudaStream_t s) {
    HFMM_LAUNCH(k_gather_q, nblk(n, 256), 256, 0, s, n, sidx, q_re, q_im, q_s, q_max);
}

void particles_f64(const ParticlePass& p, cudaStream_t s) {
    if (p.nrows == 0 && p.op != ParticleOp::COMBINE) return;
    const int key = (p.nf - 1) * 4 + (p.R - 1) * 2 + (p.field ? 1 : 0);
    switch (key) {
        case 0: particles_mode<1, 1, false>(p, s); break;
        case 1: particles_mode<1, 1, true>(p, s); break;
        case 2: particles_mode<1, 2, false>(p, s); break;
        case 3: particles_mode<1, 2, true>(p, s); break;
        case 4: particles_mode<2, 1, false>(p, s); break;
        case 5: particles_mode<2, 1, true>(p, s); break;
        case 6: particles_mode<2, 2, false>(p, s); break;
        case 7: particles_mode<2, 2, true>(p, s); break;
        default: throw Error{HFMM_ERR_ARG, "particles_f64: bad configuration"};
    }
}

}  // namespace hfmm
