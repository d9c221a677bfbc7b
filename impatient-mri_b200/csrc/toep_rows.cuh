// Pruned F^H F engine on mixed-radix lengths (see toep_rows.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstddef>

namespace imp {

// An image of ns x nm x nf voxels (f fastest; 2-D: nm = 1) runs on transforms of
// es x em x ef points, the next lengths of the engine's table (the zero padding
// covers the rest).
struct ToepRowsPlan {
    int ns = 0, nm = 1, nf = 0, es = 0, em = 1, ef = 0;
    int C = 0, L1 = 0;     // coils, segments
    int chunk = 1;         // (segment, coil) transforms per launch
    int e_s = -1, e_m = -1, e_f = -1;  // table entries of the lengths
    // spectrum of one transform before the slow axis, and of its rows alone
    size_t job_elems() const { return (size_t)ns * (nm > 1 ? 2 * em : 1) * 2 * ef; }
    size_t row_elems() const { return nm > 1 ? (size_t)ns * nm * 2 * ef : 0; }
    size_t b0_elems() const { return (size_t)chunk * row_elems(); }
    size_t b1_elems() const { return (size_t)chunk * job_elems(); }
    // one segment's spectrum
    size_t q_elems() const { return (size_t)2 * es * (nm > 1 ? 2 * em : 1) * 2 * ef; }
    int launches() const {  // per application
        return (nm > 1 ? 5 : 3) * ((L1 * C + chunk - 1) / chunk);
    }
};

// False when a side is longer than the table's longest length.
bool toep_rows_plan(int ns, int nm, int nf, int C, int L1, ToepRowsPlan *p);

// Twiddle tables of the axes s, m (3-D only), f (device memory, the caller's to free).
cudaError_t toep_rows_twiddles(const ToepRowsPlan &p, float2 *tw[3]);

// fftbuf [nl][2es][2em][2ef] = the kernels Q_l of nl segments (reference layout,
// [nl][2ns][2nm][2nf] split re/im, displacement zero at (ns, nm, nf)), each at its
// displacements modulo the grid.
cudaError_t toep_rows_embed(const ToepRowsPlan &p, float2 *fftbuf, const float *q_r,
                            const float *q_i, int nl, cudaStream_t st);
// qf2 [nl][2es][2em][2ef] in parity-major order from the natural-order spectra, scaled.
cudaError_t toep_rows_qf(const ToepRowsPlan &p, float2 *qf2, const float2 *qf, float scale, int nl,
                         cudaStream_t st);

// q = sum_{l,c} conj(e_l S_c) crop(IFFT(Qf_l FFT(pad(e_l S_c x)))); sens [C][N],
// eph [L1][N], qf2 [L1][q_elems].  Every kernel returns at once when *done.
cudaError_t toep_rows_apply(const ToepRowsPlan &p, float2 *q, const float2 *x, const float2 *sens,
                            const float2 *eph, float2 *b0, float2 *b1, const float2 *qf2,
                            const int *done, float2 *const tw[3], cudaStream_t st);

}  // namespace imp
