// The FP64 M2L by convolution (m2l_conv.cu): the kernels' call parameters.
#pragma once
#include "hfmm_internal.cuh"

namespace hfmm {

struct ConvCall {
    int p, n, n_s, ld;                // order, transform length 2p - 1, surface points, row length
    int n_slots, n_groups, CH;        // slots (the zero slot follows), groups, children per CTA
    int kz0, kz1, ky0, ky1, rows;     // the chunk's frequencies; rows = its (kz, ky) pairs
    int n_seg;                        // kz segments of the forward transform's CTAs
    int first;                        // the first chunk stores the check potentials, others add
    int n_fam, seq_fam;               // families of spectra; 1: sequence i takes family i's, 0: family 0's
    const int32_t *child, *nbr, *pos, *line_off, *line_k;
    const int4* groups;
    const double2 *tw, *K;            // e^{2 pi i m / n} as (cos, sin); the spectra
    // Sequence i, box b: R columns from i * seq_stride + b * box_stride on. A sequence is one
    // family's complex column (R = 2) or one real column (R = 1)
    const double* dens;
    double* check;
    int64_t seq_stride, box_stride;
    const unsigned long long* q_max;  // R = 2: bits of the largest real and imaginary charge
    double2 *X, *Y;                   // [sequence][row][kx][slot][child]
};

}  // namespace hfmm
