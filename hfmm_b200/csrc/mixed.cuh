// Mixed-precision (two FP16 planes on tcgen05) M2L: shared declarations.
#pragma once
#include "hfmm_internal.cuh"

#include <cuda.h>
#include <cuda_fp16.h>

#include <atomic>
#include <cstring>

#include <string>
#include <vector>

namespace hfmm {

// TMA descriptors of the planes of one level's M2L tables (316 non-adjacent displacements,
// [z][m][k] FP16), per kernel family, and in grid mode of its dense density grid (5-D).
struct MixedMaps {
    CUtensorMap a[2][2], b[2][2];
};

struct MixedCall {
    const int32_t* tile_tgt;       // ntiles x (128 / R) target boxes, -1 padded
    int ntiles;
    const int32_t* src_tab;        // nb x 351 source boxes (-1 = none)
    const int32_t* disp_compact;   // 343: displacement -> M2L table index (-1 = adjacent)
    const uint16_t* B;             // equivalent densities' planes, [plane][fam][box][R][ld] FP16
    int64_t b_plane;               // elements between planes
    const unsigned long long* b_max[2];   // per family: bits of each column's largest density
    double a_scale[2];             // per family: the scale of A's planes
    double* out;                   // check potentials [fam][box][R][ld], FP64
    int R, ld, n_fam;
    int ldk, ldm;                  // rectangular tables: K extent (B rows) and M extent (out
                                   // rows); 0 = ld. A tables are [count][ldm][ldk]
    int fold2;                     // log2 of the k-chunks per FP32 accumulation unit (0: 12 MMAs, 1: 24)
    int valid;                     // rows and columns of A that can be nonzero: K stops there,
                                   // and a row block with at most 64 runs the M = 64 MMA shape
    int64_t fam_stride, out_fam_stride, nb;
    int64_t src_lo, src_hi;        // valid source boxes [src_lo, src_hi) (0, nb when unset)
    int* err;
    uint64_t wait_ns;              // limit of each bounded wait (0: 2 s); set by m2l_split
    int starve;                    // test only: leave stage 0 without its gather arrivals
    // grid mode (complete level, R = 2): B comes from the dense density grid by TMA, one
    // strided 4 x 4 x 4 box per displacement; tile_tgt then holds grid tiles and
    // tile_org each tile's grid origin (x, y, z)
    int grid;
    const int32_t* tile_org;
};

// Wait limit and starvation switch of the next M2L launches (hfmm_debug_m2l_wait):
// a test makes a bounded wait run out on purpose and checks the error status. Atomic:
// a hook call may come from another thread than the evaluate that reads it.
extern std::atomic<uint64_t> g_m2l_wait_ns;
extern std::atomic<int> g_m2l_starve;

// The two FP16 planes of a scaled value: hi its rounding, lo the rounding of the rest (exact in
// FP64). The scale, a power of two, puts the largest magnitude of an operand (of one charge
// column of the densities: a small column keeps its bits beside a large one) in [2^13, 2^14):
// a value down to 2^-16 of that keeps the full 22 bits, a smaller one is off by at most 2^-25
// in scaled units, 2^-38 of the largest.
__device__ __forceinline__ void split2(double x, uint16_t (&p)[2]) {
    const __half h = __float2half_rn((float)x);
    p[0] = __half_as_ushort(h);
    p[1] = __half_as_ushort(__float2half_rn((float)(x - (double)__half2float(h))));
}

// That scale from the largest magnitude's bits; 1 where there is none (zero, infinite, NaN or
// outside the range whose scale is a normal number).
__host__ __device__ __forceinline__ double plane_scale(unsigned long long most) {
    const int e = (int)(most >> 52);   // biased exponent: 2^(e - 1023) <= magnitude
    if (e < 30 || e > 2000) return 1.0;
    const unsigned long long bits = (unsigned long long)(2046 + 13 - e) << 52;   // 2^(13 - (e - 1023))
    double s;
#ifdef __CUDA_ARCH__
    s = __longlong_as_double((long long)bits);
#else
    memcpy(&s, &bits, sizeof(s));
#endif
    return s;
}

// Do planes with one scale a level serve this plan's densities? Their absolute error is 2^-38 of
// the level's largest, everywhere. Under a kernel that falls like 1 / r the field of the largest
// hides it, in two cases not:
//  * A screened kernel leaves clusters some screening lengths apart their own results, and the
//    weaker cluster's are lost. Mixed against FP64 on the weaker of two clusters across the
//    domain, charges 2^14 to 2^36 apart, p = 8, depth 6 and 10 (TF32 halves had 1.3e-6 at most):
//    kappa x extent 2: 7.9e-7, 3: 1.4e-6, 4: 6.5e-6, 6: 1.6e-4, 12: 0.6.
//  * The field -grad phi of a faraway strong cluster falls like 1 / r^2, the error's like 1 / (box
//    side)^2: on small boxes the error shows. Clusters of sigma 0.0005, depth 10, low rank, field
//    on the weaker: Laplace 3e-5 (TF32 halves 5e-7), Helmholtz k x extent = 1 1e-5 (8e-7), 3 and
//    more the same (1e-5: the tables' own error, sin family); sigma 0.004 (boxes of level 8)
//    3e-6 (7e-7), depth 6 the same.
// There the M2L runs in FP64. By convolution one family of it is as fast or faster: 5e5 points,
// p = 8, kappa = 20, whole evaluate, real / complex charges: low-rank planes 6.7 / 10.1 ms, dense
// planes 13.8 / 22.1, FP64 M2L 8.3 / 15.3 (TF32 halves 11.9 / 16.2 and 18.6 / 30.5); 20,000
// points 2.6 / 2.6 with dense planes, 0.41 / 0.56 without.
inline bool planes_hold(const hfmm_plan* P) {
    const double kd = (P->k < 0.0 ? -P->k : P->k) * P->extent;
    if (P->yukawa && kd > 2.0) return false;
    return P->md < 8 || (!P->yukawa && kd >= 3.0);
}

// Maps of the two planes of tables [count][ldm][ld] (ldm 0: ld), `plane` apart, and of a grid
// [plane][x][y][z][2][ckld]: rows and K values from `valid` on are zeros, which the loads
// then fill in instead of reading
void make_table_maps(CUtensorMap (&map)[2], const uint16_t* base, size_t plane, int valid, int ld, int count,
                     int ldm = 0);
void make_grid_maps(CUtensorMap (&map)[2], const uint16_t* base, int valid, int ckld, int G);
// rows of ld FP64 values, row i of charge column i % R, each column's largest magnitude's bits at
// most[column] -> their FP16 planes, `plane` elements apart; absmax raises most[column] to it
void split_planes(const double* src, const unsigned long long* most, uint16_t* out, int64_t plane, int64_t rows,
                  int ld, int R, cudaStream_t s);
void absmax(const double* src, int64_t rows, int ld, int R, unsigned long long* most, cudaStream_t s);
double table_scale(const double* table, int64_t rows, int ld);   // plane_scale of the largest entry
// a complete level's densities [box][2][ckld] (boxes in level order from m_id) -> planes of
// the dense grid [x][y][z][2][ckld] of side G
void split_planes_grid(const double* src, const unsigned long long* most, const uint64_t* m_id, int64_t n_boxes,
                       int G, int ckld, uint16_t* out, cudaStream_t s);
// process-wide: 1 (default) lets complete levels use grid mode, 0 forces the gather
extern std::atomic<int> g_m2l_grid;
void split_transpose_tables(const double* at, double scale, uint16_t* out, int ld, int count);
void m2l_split(const MixedMaps& maps, const MixedCall& c, cudaStream_t s);

// the low-rank mixed M2L call of one plan, level and family for R charge columns
MixedCall cx_call(hfmm_plan* P, int l, int f, int R);

// One work item of the queued M2L: a tile x one 128-row block of calls[call].
struct M2LItem {
    int call, tile, mblock;
};
// Persistent M2L over items (sorted by the caller), n_ctas resident CTAs; `next` is a
// device int the launch resets. calls, maps and items live in device memory. The wait
// limit comes from g_m2l_wait_ns at launch; starve (a test switch) leaves every CTA's
// first stage unfilled.
void m2l_queue(const MixedCall* calls, const MixedMaps* maps, const M2LItem* items, int n_items,
               int* next, int R, int n_ctas, cudaStream_t s, int starve = 0);
// The work list of a queued M2L over the plans given: every (plan, level, family)
// low-rank call with its tensor maps, one item per tile and 128-row block, largest
// first (cost: K values per entry, 0.6 for a block of at most 64 live rows). Returns
// "" when it applies, else why not (32-bit gather offsets would overflow).
std::string queue_items(hfmm_plan* const* plans, int n_plans, int R, std::vector<MixedCall>& calls,
                        std::vector<MixedMaps>& maps, std::vector<M2LItem>& items);
// A plan's own queued M2L for R charge columns, built and uploaded at finalize.
struct PlanQueue {
    DevBuf<MixedCall> calls;
    DevBuf<MixedMaps> maps;
    DevBuf<M2LItem> items;
    DevBuf<int> next;
    int n_items = 0;
};
void plan_queue_build(hfmm_plan* P);     // both charge-column counts
void plan_queue_release(hfmm_plan* P);
size_t m2l_queue_smem();
size_t m2l_split_smem();

}  // namespace hfmm
