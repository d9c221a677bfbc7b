// Two-pass register FFT of one grid axis, n = R1 R2 with R1 <= R2 <= 32.
//
//   pass 1: thread (line, j1) loads x[j1 + R1 j2] for every j2 straight from
//           global memory, takes the R2-point DFT over j2, multiplies output
//           k2 by w_n^{j1 k2} and stores it to shared memory at (j1, k2);
//   pass 2: thread (line, k2) reads its R1 values, takes the R1-point DFT over
//           j1 and stores X[k2 + R2 k1] straight to global memory (only the
//           outputs that the caller keeps).
// Consecutive threads take consecutive columns of a strided axis (cw of them,
// 64 bytes and up) and consecutive elements of a line of the contiguous one,
// so both global passes are coalesced.
//
// What bounds it: the pass moves 16 bytes per point (8 in, 8 out), HBM- or
// L2-bound when enough loads are in flight; every thread issues its R2 loads
// before it uses one.  The Stockham kernel that takes the remaining lengths
// goes through shared memory once per radix and stages its loads and stores
// there as well (two or three more round trips and barriers per pass).
#include "common.cuh"
#include "fft_reg.cuh"
#include "grid_fft2.cuh"

#include <algorithm>

namespace imp {

namespace {

constexpr int kT2 = 256;

// Lines per block: a tile of about 4096 elements (33 KB, six blocks of 256
// threads per SM), at least 8 lines (64-byte runs of a strided axis), at most 64.
constexpr int lines_of(int n) {
    int c = 64;
    while (c > 8 && c * n > 4096) c /= 2;
    return c;
}

// Shared-memory strides (float2).  Strided axis: element (j1, k2, c) at
// j1 (R2 cw + pad) + k2 cw + c; the 16 / cw values of j1 that a half-warp
// writes at once must fall on different bank pairs, which R2 cw + pad = cw
// (mod 16) gives.  Contiguous axis: element (c, j1, k2) at (c R1 + j1) P + k2
// with P odd, so that the j1 of a half-warp do.
__host__ __device__ constexpr int pad_of(int R2, int cw) {
    return cw >= 16 ? 0 : (((1 - R2) * cw) % 16 + 16) % 16;
}
__host__ __device__ constexpr int odd_row(int R2) { return R2 | 1; }

template <int R1, int R2>
constexpr size_t smem2(int cw) {
    const size_t a = (size_t)R1 * (R2 * cw + 16), b = (size_t)cw * R1 * odd_row(R2);
    return sizeof(float2) * (a > b ? a : b);
}

template <int R1, int R2>
__global__ void __launch_bounds__(kT2) k_fft2(float2 *__restrict__ data, const AxisArgs p,
                                              const float2 *__restrict__ tw, const bool inv) {
    // tw[k2 R1 + j1] = w_n^{j1 k2}: the threads of a warp read neighbouring entries
    extern __shared__ float2 sm[];
    constexpr int n = R1 * R2;
    const bool contig = p.S == 1;
    const int cw = p.cw;
    const long long l0 = (long long)blockIdx.x * cw;
    const long long o = contig ? 0 : l0 / p.Sc;
    float2 *base = contig ? data + l0 * n : data + o * n * p.S + line_offset(p, l0 - o * p.Sc);
    const long long jst = p.S, cst = contig ? n : 1;
    const int left = contig ? (int)min((long long)cw, p.lines - l0) : cw;  // lines of this block
    const int s1 = contig ? odd_row(R2) : R2 * cw + pad_of(R2, cw);  // stride of j1
    const int s2 = contig ? 1 : cw;                                  // stride of k2
    const int sc = contig ? R1 * odd_row(R2) : 1;                    // stride of the line
    for (int it = threadIdx.x; it < R1 * cw; it += blockDim.x) {
        const int c = contig ? it / R1 : it & (cw - 1);
        const int j1 = contig ? it - c * R1 : it >> p.lcw;
        if (c >= left) continue;
        const float2 *src = base + c * cst + j1 * jst;
        float2 v[R2];
#pragma unroll
        for (int q = 0; q < R2; ++q) v[q] = src[(long long)(q * R1) * jst];
#pragma unroll
        for (int q = 0; q < R2; ++q) v[q] = fftr::swap_ri(v[q], inv);
        fftr::dft<R2>(v);
        float2 *dst = sm + j1 * s1 + c * sc;
        dst[0] = v[0];
#pragma unroll
        for (int q = 1; q < R2; ++q) dst[q * s2] = cmul(v[q], __ldg(&tw[q * R1 + j1]));
    }
    __syncthreads();
    for (int it = threadIdx.x; it < R2 * cw; it += blockDim.x) {
        const int c = contig ? it / R2 : it & (cw - 1);
        const int k2 = contig ? it - c * R2 : it >> p.lcw;
        if (c >= left) continue;
        const float2 *src = sm + k2 * s2 + c * sc;
        float2 v[R1];
#pragma unroll
        for (int q = 0; q < R1; ++q) v[q] = src[q * s1];
        fftr::dft<R1>(v);
        float2 *dst = base + c * cst + k2 * jst;
#pragma unroll
        for (int q = 0; q < R1; ++q) {
            const int j = k2 + R2 * q;
            if (j < p.klo || j >= n - p.khi)
                dst[(long long)(q * R2) * jst] = fftr::swap_ri(v[q], inv);
        }
    }
}

struct Entry {
    int n, r2;
    size_t (*smem)(int);
    void (*kern)(float2 *, const AxisArgs, const float2 *, const bool);
};

#define E2(A, B) {A * B, B, smem2<A, B>, k_fft2<A, B>}
// The lengths with a balanced split into register radices.
const Entry kEntries[] = {
    E2(2, 4),   E2(3, 4),   E2(4, 4),   E2(4, 5),   E2(4, 6),   E2(4, 7),   E2(6, 6),
    E2(4, 8),   E2(5, 8),   E2(6, 8),   E2(7, 8),   E2(8, 8),   E2(8, 9),   E2(8, 10),
    E2(8, 12),  E2(8, 14),  E2(10, 12), E2(8, 16),  E2(12, 12), E2(10, 16), E2(12, 14),
    E2(12, 16), E2(10, 20), E2(12, 18), E2(14, 16), E2(15, 16), E2(16, 16), E2(14, 20),
    E2(16, 18), E2(16, 20), E2(14, 24), E2(18, 20), E2(16, 24), E2(14, 28), E2(20, 20),
    E2(18, 24), E2(16, 28), E2(20, 24), E2(18, 28), E2(16, 32), E2(20, 28), E2(24, 24),
    E2(20, 32), E2(24, 28), E2(24, 32), E2(28, 28), E2(28, 32), E2(32, 32),
};
#undef E2

const Entry *entry_of(int n) {
    for (const Entry &e : kEntries)
        if (e.n == n) return &e;
    return nullptr;
}

}  // namespace

int fft2_lines(int n) { return entry_of(n) ? lines_of(n) : 0; }

int fft2_twiddle_exp(int n, int i) {
    const int r1 = n / entry_of(n)->r2;
    return (i % r1) * (i / r1);
}

double fft2_gain(int n) {
    const int r2 = entry_of(n)->r2;
    return 1.0 + fftr::dft_gain(n / r2) + fftr::dft_gain(r2);
}

cudaError_t fft2_setup() {
    for (const Entry &e : kEntries) {
        if (e.smem(lines_of(e.n)) <= 48 * 1024) continue;
        const cudaError_t r = cudaFuncSetAttribute(
            (const void *)e.kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
            (int)e.smem(lines_of(e.n)));
        if (r != cudaSuccess) return r;
    }
    return cudaSuccess;
}

cudaError_t fft2_launch(float2 *data, const AxisArgs &p, const float2 *tw, bool inverse,
                        cudaStream_t st) {
    const Entry *e = entry_of(p.n);
    if (!e || p.cw < 1 || p.cw > lines_of(p.n) || (p.cw & (p.cw - 1)))
        return cudaErrorInvalidValue;
    const long long blocks = (p.lines + p.cw - 1) / p.cw;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    // few lines per block (a strided axis whose kept runs are short): no idle warps
    const int threads = std::min(kT2, (e->r2 * p.cw + 31) / 32 * 32);
    e->kern<<<(unsigned)blocks, threads, e->smem(p.cw), st>>>(data, p, tw, inverse);
    return cudaGetLastError();
}

}  // namespace imp
