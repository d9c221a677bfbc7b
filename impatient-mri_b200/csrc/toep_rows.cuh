// Pruned F^H F engine of 2-D images on mixed-radix lengths (see toep_rows.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstddef>

namespace imp {

// An image of ns x nf voxels (f fastest) runs on transforms of es x ef points,
// the next lengths of the engine's table (the zero padding covers the rest).
struct ToepRowsPlan {
    int ns = 0, nf = 0, es = 0, ef = 0;
    int C = 0, L1 = 0;     // coils, segments
    int chunk = 1;         // (segment, coil) transforms per launch
    int e_s = -1, e_f = -1;  // table entries of the two lengths
    size_t b1_elems() const { return (size_t)chunk * ns * 2 * ef; }
    size_t q_elems() const { return (size_t)4 * es * ef; }  // one segment's spectrum
    int launches() const { return 3 * ((L1 * C + chunk - 1) / chunk); }  // per application
};

// False when a side is longer than the table's longest length.
bool toep_rows_plan(int ns, int nf, int C, int L1, ToepRowsPlan *p);

// Twiddle tables of both axes (device memory of the caller's to free).
cudaError_t toep_rows_twiddles(const ToepRowsPlan &p, float2 **tw_s, float2 **tw_f);

// fftbuf [nl][2es][2ef] = the kernels Q_l of nl segments (reference layout,
// [nl][2ns][2nf] split re/im, displacement zero at (ns, nf)), each at its
// displacements modulo the grid.
cudaError_t toep_rows_embed(const ToepRowsPlan &p, float2 *fftbuf, const float *q_r,
                            const float *q_i, int nl, cudaStream_t st);
// qf2 [nl][2es][2ef] in parity-major order from the natural-order spectra, scaled.
cudaError_t toep_rows_qf(const ToepRowsPlan &p, float2 *qf2, const float2 *qf, float scale, int nl,
                         cudaStream_t st);

// q = sum_{l,c} conj(e_l S_c) crop(IFFT(Qf_l FFT(pad(e_l S_c x)))); sens [C][N],
// eph [L1][N], qf2 [L1][q_elems].  Every kernel returns at once when *done.
cudaError_t toep_rows_apply(const ToepRowsPlan &p, float2 *q, const float2 *x, const float2 *sens,
                            const float2 *eph, float2 *b1, const float2 *qf2, const int *done,
                            const float2 *tw_s, const float2 *tw_f, cudaStream_t st);

}  // namespace imp
