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
    int n_fam;
    const int32_t *child, *nbr, *pos, *line_off, *line_k;
    const int4* groups;
    const double2 *tw, *K;            // e^{2 pi i m / n} as (cos, sin); the spectra
    const double* dens;               // [fam][box][R][ld]
    double* check;
    int64_t fam_stride;
    double2 *X, *Y;                   // [fam][row][kx][slot][child]
};

}  // namespace hfmm
