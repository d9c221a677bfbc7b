// Two-pass register FFT of one grid axis, n = R1 R2 (see grid_fft2.cu).
#pragma once
#include <cuda_runtime.h>

namespace imp {

// One axis pass: the lines of a block and the outputs it keeps.  Lines of a
// strided axis are consecutive columns (compact indices over the kept faster
// coordinates); those of the contiguous axis (S == 1) are whole lines.
struct AxisArgs {
    long long S;       // element stride of the axis (product of the faster lengths)
    int n, ln;         // axis length and its log2 (when a power of two)
    int cw, lcw, rs;   // lines per block (power of two), log2(cw), tile row stride
    int nst;           // stages
    unsigned char rad[24];
    // Pruning.  Outputs kept along this axis: j < klo or j >= n - khi (klo = n:
    // all).  Lines: only those whose coordinates along the faster axes are kept
    // there, enumerated compactly: nf faster axes (outer first) with kept
    // ranges [0, flo) and [fg - fhi, fg); Sc = product of their kept counts.
    int klo, khi;
    int nf;
    int flo[2], fhi[2], fg[2];
    long long Sc;
    long long lines;   // lines in all (the last block may be partial: contiguous axis)
};

// Offset (within S) of compact line index ic over the kept faster coordinates.
__device__ __forceinline__ long long line_offset(const AxisArgs &p, long long ic) {
    auto ex = [](long long c, int lo, int hi, int g) -> long long {
        return c < lo ? c : c + (g - lo - hi);
    };
    if (p.nf == 0) return ic;
    if (p.nf == 1) return ex(ic, p.flo[0], p.fhi[0], p.fg[0]);
    const long long inner = p.flo[1] + p.fhi[1];
    const long long y = ic / inner, z = ic - y * inner;
    return ex(y, p.flo[0], p.fhi[0], p.fg[0]) * p.fg[1] + ex(z, p.flo[1], p.fhi[1], p.fg[1]);
}

// Largest number of lines per block of the two-pass kernel for axis length n
// (0: no instantiation of that length).
int fft2_lines(int n);
// Exponent of entry i < n of its twiddle table exp(-2 pi i e / n) (fft2_lines(n) > 0).
int fft2_twiddle_exp(int n, int i);
// Mean gain of its register transforms, which the table's entries are divided by.
double fft2_gain(int n);
// Launches it with p.cw lines per block (a power of two, at most fft2_lines).
cudaError_t fft2_launch(float2 *data, const AxisArgs &p, const float2 *tw, bool inverse,
                        cudaStream_t st);
// Opts every instantiation into its shared memory on the current device.
cudaError_t fft2_setup();

}  // namespace imp
