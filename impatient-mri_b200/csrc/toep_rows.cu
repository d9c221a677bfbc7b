// Pruned F^H F engine of 2-D and 3-D images on mixed-radix lengths.
//
// Along each axis of length n the zero-padded 2n-point transform splits by
// output parity a into two n-point transforms of x[j] w_2n^{a j}; the inverse
// restricted to [0, n) is the parity sum of two n-point inverses (the doubled
// grid never exists).  With n = R1 R2 (R1, R2 <= 32), j = j1 + R1 j2 and
// k = k2 + R2 k1, an n-point line is an R2-point register DFT per j1, the
// twiddle w_2n^{j1 (2 k2 + a)} (it carries the parity's j1 part; the rest,
// w_{2 R2}^{a j2}, is a compile-time constant) and an R1-point register DFT
// per k2.  An image is [s][m][f] (2-D: one m).  Kernels per chunk of (segment,
// coil) transforms:
//   k_row_fwd  rows along f: forms S_c e_l x from global memory in registers,
//              both parities, writes [s][m][a][kf];
//   k_mid_fwd  3-D: columns along m, both parities, writes [s][a][km][...];
//   k_col      columns along s, in place: both parities forward, x Qf_l,
//              inverse, parity sum;
//   k_mid_inv  3-D: columns along m: inverse, parity sum;
//   k_row_inv  rows along f: inverse, parity sum, conj(e_l S_c), summed over the
//              block's transforms in registers and over the cluster's blocks in
//              distributed shared memory.
// Every first DFT reads global memory straight into registers and every last
// one writes it from registers, so a row kernel makes one trip through shared
// memory and the column kernel two.  The inverse transforms run as forward
// ones on values with real and imaginary parts exchanged.
//
// What bounds it: issue and latency at 16 to 24 warps per SM (the register DFTs
// take 64 registers for 32 points), not memory (20 to 60 % of DRAM).  512x512 x 32
// coils, one application: rows forward 48 us, columns 143, rows inverse 80 (a plane
// engine of line passes in shared memory: 75, 175, 114).  256x256x32 x 4 coils, one
// segment: 56, 91 (middle forward), 259, 79, 71 us (plane engine 176, 273, 202).
//
// Sides that are no length of the table run on the next one: rows and columns
// past the image are zero on input and dropped on output, Q_l sits at its
// displacements on the larger grid, and the result is the same sum.
#include "common.cuh"
#include "fft_reg.cuh"
#include "toep_rows.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <vector>

namespace imp {

namespace cg = cooperative_groups;

namespace {

constexpr int kColW = 8;  // columns per block of k_col (64-byte rows)

__host__ __device__ constexpr int cmax(int a, int b) { return a > b ? a : b; }

// Row kernels: thread (row, j1) in the R2-point passes, (row, a, k2) in the
// R1-point ones.  PS rows per block, about 128 threads.
template <int R1, int R2>
struct RowShape {
    static constexpr int n = R1 * R2;
    static constexpr int per_row = cmax(R1, 2 * R2);
    static constexpr int PS = cmax(1, 128 / per_row);
    static constexpr int T = (PS * per_row + 31) / 32 * 32;
    // element (row, a, j1, k2) at (row 2 + a) A + j1 P + k2: P odd so that the
    // j1 of a half-warp fall on different bank pairs, A = R2 (mod 16) so that
    // the two parities of short k2 runs do
    static constexpr int P = R2 | 1;
    static constexpr int A = R1 * P + ((R2 - R1 * P) % 16 + 16) % 16;
    static constexpr size_t smem = sizeof(float2) * (size_t)PS * 2 * A;
};

template <int R2, int Q>
__device__ __forceinline__ void half_twist(float2 (&v)[R2]) {  // v[q] *= w_{2 R2}^q
    if constexpr (Q < R2) {
        v[Q] = fftr::mulw<Q, 2 * R2>(v[Q]);
        half_twist<R2, Q + 1>(v);
    }
}

// tables: twA[(a R2 + k2) R1 + j1] (threads over j1), then
//         twB[(j1 2 + a) R2 + k2]  (threads over k2), both w_2n^{j1 (2 k2 + a)}
template <int R1, int R2>
__global__ void __launch_bounds__(RowShape<R1, R2>::T)
    k_row_fwd(float2 *__restrict__ b1, const float2 *__restrict__ x,
              const float2 *__restrict__ sens, const float2 *__restrict__ eph, int ns, int nf,
              int C, int job0, const float2 *__restrict__ tw, const int *__restrict__ done) {
    using S = RowShape<R1, R2>;
    extern __shared__ float2 sm[];
    if (done && *done) return;
    const int s0 = blockIdx.x * S::PS;
    const int job = job0 + blockIdx.y, l = job / C, c = job - l * C;
    {
        const int row = threadIdx.x / R1, j1 = threadIdx.x - row * R1, s = s0 + row;
        if (row < S::PS && s < ns) {
            const size_t at = (size_t)s * nf + j1, N = (size_t)ns * nf;
            const float2 *sc = sens + (size_t)c * N + at, *ec = eph + (size_t)l * N + at;
            float2 v[R2], t[R2];
#pragma unroll
            for (int q = 0; q < R2; ++q) {
                v[q] = make_float2(0.f, 0.f);
                if (j1 + R1 * q < nf)
                    v[q] = cmul(cmul(__ldg(&sc[R1 * q]), __ldg(&ec[R1 * q])),
                                __ldg(&x[at + R1 * q]));
            }
            float2 *dst = sm + (row * 2) * S::A + j1 * S::P;
#pragma unroll
            for (int q = 0; q < R2; ++q) t[q] = v[q];
            fftr::dft<R2>(t);
            dst[0] = t[0];
#pragma unroll
            for (int q = 1; q < R2; ++q) dst[q] = cmul(t[q], __ldg(&tw[q * R1 + j1]));
            half_twist<R2, 1>(v);
            fftr::dft<R2>(v);
#pragma unroll
            for (int q = 0; q < R2; ++q)
                dst[S::A + q] = cmul(v[q], __ldg(&tw[(R2 + q) * R1 + j1]));
        }
    }
    __syncthreads();
    const int ra = threadIdx.x / R2, k2 = threadIdx.x - ra * R2, a = ra & 1, row = ra >> 1;
    const int s = s0 + row;
    if (row < S::PS && s < ns) {
        const float2 *src = sm + ra * S::A + k2;
        float2 v[R1];
#pragma unroll
        for (int q = 0; q < R1; ++q) v[q] = src[q * S::P];
        fftr::dft<R1>(v);
        float2 *dst = b1 + ((size_t)blockIdx.y * ns + s) * (2 * S::n) + a * S::n + k2;
#pragma unroll
        for (int q = 0; q < R1; ++q) dst[R2 * q] = v[q];
    }
}

// blockIdx.y = cluster rank: the block takes transforms job0 + rank, + csize, ...
template <int R1, int R2>
__global__ void __launch_bounds__(RowShape<R1, R2>::T)
    k_row_inv(float2 *__restrict__ out, const float2 *__restrict__ b1,
              const float2 *__restrict__ sens, const float2 *__restrict__ eph, int ns, int nf,
              int C, int job0, int njobs, int first, const float2 *__restrict__ tw,
              const int *__restrict__ done) {
    using S = RowShape<R1, R2>;
    extern __shared__ float2 sm[];
    cg::cluster_group cluster = cg::this_cluster();
    const bool skip = done && *done;
    const int rank = blockIdx.y, csize = gridDim.y;
    const int s0 = blockIdx.x * S::PS;
    const size_t N = (size_t)ns * nf;
    const float2 *twB = tw + 2 * S::n;
    const int ra = threadIdx.x / R2, k2 = threadIdx.x - ra * R2, a = ra & 1;
    const bool in1 = (ra >> 1) < S::PS && s0 + (ra >> 1) < ns;
    const int row = threadIdx.x / R1, j1 = threadIdx.x - row * R1, s = s0 + row;
    const bool in2 = row < S::PS && s < ns;
    const size_t at = (size_t)s * nf + j1;
    float2 y[R2];
#pragma unroll
    for (int q = 0; q < R2; ++q) y[q] = make_float2(0.f, 0.f);
    if (!skip) {
        for (int i = rank; i < njobs; i += csize) {
            const int job = job0 + i, l = job / C, c = job - l * C;
            if (in1) {
                const float2 *src = b1 + ((size_t)i * ns + s0 + (ra >> 1)) * (2 * S::n) +
                                    a * S::n + k2;
                float2 v[R1];
#pragma unroll
                for (int q = 0; q < R1; ++q) v[q] = src[R2 * q];
#pragma unroll
                for (int q = 0; q < R1; ++q) v[q] = fftr::swap_ri(v[q], true);
                fftr::dft<R1>(v);
                float2 *dst = sm + ra * S::A + k2;
                dst[0] = v[0];
#pragma unroll
                for (int q = 1; q < R1; ++q)
                    dst[q * S::P] = cmul(v[q], __ldg(&twB[(q * 2 + a) * R2 + k2]));
            }
            __syncthreads();
            if (in2) {
                const float2 *src = sm + (row * 2) * S::A + j1 * S::P;
                float2 t[R2], u[R2];
#pragma unroll
                for (int q = 0; q < R2; ++q) t[q] = src[q];
                fftr::dft<R2>(t);
#pragma unroll
                for (int q = 0; q < R2; ++q) u[q] = src[S::A + q];
                fftr::dft<R2>(u);
                half_twist<R2, 1>(u);
                const float2 *sc = sens + (size_t)c * N + at, *ec = eph + (size_t)l * N + at;
#pragma unroll
                for (int q = 0; q < R2; ++q)
                    if (j1 + R1 * q < nf) {
                        const float2 val = make_float2(t[q].y + u[q].y, t[q].x + u[q].x);
                        const float2 z =
                            cmulc(cmul(__ldg(&sc[R1 * q]), __ldg(&ec[R1 * q])), val);
                        y[q].x += z.x;
                        y[q].y += z.y;
                    }
            }
            __syncthreads();
        }
        if (in2) {  // partial sums over the work area: element (row, f) at row n + f
#pragma unroll
            for (int q = 0; q < R2; ++q) sm[row * S::n + j1 + R1 * q] = y[q];
        }
    }
    cluster.sync();
    if (!skip) {
        const int e_all = S::PS * S::n, share = (e_all + csize - 1) / csize;
        const int e1 = min(e_all, (rank + 1) * share);
        for (int e = rank * share + threadIdx.x; e < e1; e += S::T) {
            const int r = e / S::n, f = e - r * S::n;
            if (f >= nf || s0 + r >= ns) continue;
            float2 sum = make_float2(0.f, 0.f);
            for (int k = 0; k < csize; ++k) {
                const float2 v = cluster.map_shared_rank(sm, k)[e];
                sum.x += v.x;
                sum.y += v.y;
            }
            const size_t o = (size_t)(s0 + r) * nf + f;
            if (!first) {
                sum.x += out[o].x;
                sum.y += out[o].y;
            }
            out[o] = sum;
        }
    }
    cluster.sync();  // no block leaves while another still reads its sums
}

template <int R1, int R2>
struct ColShape {
    static constexpr int n = R1 * R2, W = kColW;
    static constexpr int T = W * cmax(R1, 2 * R2);
    // element (a, j1, k2, w) at ((a R1 + j1) P + k2) W + w, P odd: the two j1 of a
    // half-warp fall on different bank halves
    static constexpr int P = R2 | 1;
    static constexpr size_t smem = sizeof(float2) * (size_t)2 * R1 * P * W;
};

// Block = (column group, transform).  Columns [cg W, + W) of the transform, in
// place.  `jobs_x`: the transform is the faster block index, so that the coils of
// a segment read the same columns of Qf_l close in time (3-D, where Qf_l exceeds
// the L2; in 2-D the neighbouring columns first are faster, 6.51 against 6.62 ms
// for 20 updates at 512x512 x 32 coils).
// Threads per SM that the registers are budgeted for: 16-point transforms fit 80 registers
// and 24 warps (256x256x32 x 4 coils: 28.1 ms per reconstruction, 28.2 with 16 warps),
// longer ones take up to 128 and 16 warps (512x512: 6.5 ms for 20 updates, 8.9 with 24);
// shorter ones need no budget and blocks that do not divide it keep what is left.
template <int R1, int R2>
__global__ void __launch_bounds__(ColShape<R1, R2>::T,
                                  cmax(1, (R1 == 16 ? 768 : 512) / ColShape<R1, R2>::T))
    k_col(float2 *__restrict__ b1, const float2 *__restrict__ qf2, int ns, int ncol, int C,
          int job0, int jobs_x, const float2 *__restrict__ tw, const int *__restrict__ done) {
    using S = ColShape<R1, R2>;
    constexpr int W = S::W, P = S::P, n = S::n;
    extern __shared__ float2 sm[];
    if (done && *done) return;
    const unsigned cgrp = jobs_x ? blockIdx.y : blockIdx.x;
    const int job = (int)(jobs_x ? blockIdx.x : blockIdx.y);
    const int l = (job0 + job) / C;
    const int w = threadIdx.x % W, tj = threadIdx.x / W;
    const size_t col0 = (size_t)cgrp * W + w;
    float2 *col = b1 + (size_t)job * ns * ncol + col0;
    const float2 *twB = tw + 2 * n;
    if (tj < R1) {
        const int j1 = tj;
        float2 v[R2], t[R2];
#pragma unroll
        for (int q = 0; q < R2; ++q) {
            v[q] = make_float2(0.f, 0.f);
            if (j1 + R1 * q < ns) v[q] = col[(size_t)(j1 + R1 * q) * ncol];
        }
        float2 *dst = sm + j1 * P * W + w;
#pragma unroll
        for (int q = 0; q < R2; ++q) t[q] = v[q];
        fftr::dft<R2>(t);
        dst[0] = t[0];
#pragma unroll
        for (int q = 1; q < R2; ++q) dst[q * W] = cmul(t[q], __ldg(&tw[q * R1 + j1]));
        half_twist<R2, 1>(v);
        fftr::dft<R2>(v);
        dst += R1 * P * W;
#pragma unroll
        for (int q = 0; q < R2; ++q) dst[q * W] = cmul(v[q], __ldg(&tw[(R2 + q) * R1 + j1]));
    }
    __syncthreads();
    if (tj < 2 * R2) {
        const int a = tj / R2, k2 = tj - a * R2;
        float2 *p = sm + (a * R1 * P + k2) * W + w;
        float2 z[R1];
#pragma unroll
        for (int q = 0; q < R1; ++q) z[q] = p[q * P * W];
        fftr::dft<R1>(z);
        const float2 *qc = qf2 + (size_t)l * 2 * n * ncol + (size_t)(a * n + k2) * ncol + col0;
#pragma unroll
        for (int q = 0; q < R1; ++q)
            z[q] = fftr::swap_ri(cmul(z[q], __ldg(&qc[(size_t)(R2 * q) * ncol])), true);
        fftr::dft<R1>(z);
        p[0] = z[0];
#pragma unroll
        for (int q = 1; q < R1; ++q)
            p[q * P * W] = cmul(z[q], __ldg(&twB[(q * 2 + a) * R2 + k2]));
    }
    __syncthreads();
    if (tj < R1) {
        const int j1 = tj;
        const float2 *src = sm + j1 * P * W + w;
        float2 t[R2], u[R2];
#pragma unroll
        for (int q = 0; q < R2; ++q) t[q] = src[q * W];
        fftr::dft<R2>(t);
        src += R1 * P * W;
#pragma unroll
        for (int q = 0; q < R2; ++q) u[q] = src[q * W];
        fftr::dft<R2>(u);
        half_twist<R2, 1>(u);
#pragma unroll
        for (int q = 0; q < R2; ++q)
            if (j1 + R1 * q < ns)
                col[(size_t)(j1 + R1 * q) * ncol] =
                    make_float2(t[q].y + u[q].y, t[q].x + u[q].x);
    }
}

// Columns along m of one s-plane: in [m][w] (row stride ncol) -> both parities
// [a][km][w].  blockIdx.x = column group, .y = s, .z = transform.
template <int R1, int R2>
__global__ void __launch_bounds__(ColShape<R1, R2>::T)
    k_mid_fwd(float2 *__restrict__ b1, const float2 *__restrict__ b0, int nm, int ncol,
              const float2 *__restrict__ tw, const int *__restrict__ done) {
    using S = ColShape<R1, R2>;
    constexpr int W = S::W, P = S::P, n = S::n;
    extern __shared__ float2 sm[];
    if (done && *done) return;
    const int w = threadIdx.x % W, tj = threadIdx.x / W;
    const size_t plane = (size_t)blockIdx.z * gridDim.y + blockIdx.y;
    if (tj < R1) {
        const int j1 = tj;
        const float2 *src = b0 + plane * nm * ncol + blockIdx.x * W + w;
        float2 v[R2], t[R2];
#pragma unroll
        for (int q = 0; q < R2; ++q) {
            v[q] = make_float2(0.f, 0.f);
            if (j1 + R1 * q < nm) v[q] = src[(size_t)(j1 + R1 * q) * ncol];
        }
        float2 *dst = sm + j1 * P * W + w;
#pragma unroll
        for (int q = 0; q < R2; ++q) t[q] = v[q];
        fftr::dft<R2>(t);
        dst[0] = t[0];
#pragma unroll
        for (int q = 1; q < R2; ++q) dst[q * W] = cmul(t[q], __ldg(&tw[q * R1 + j1]));
        half_twist<R2, 1>(v);
        fftr::dft<R2>(v);
        dst += R1 * P * W;
#pragma unroll
        for (int q = 0; q < R2; ++q) dst[q * W] = cmul(v[q], __ldg(&tw[(R2 + q) * R1 + j1]));
    }
    __syncthreads();
    if (tj < 2 * R2) {
        const int a = tj / R2, k2 = tj - a * R2;
        const float2 *src = sm + (a * R1 * P + k2) * W + w;
        float2 z[R1];
#pragma unroll
        for (int q = 0; q < R1; ++q) z[q] = src[q * P * W];
        fftr::dft<R1>(z);
        float2 *dst = b1 + (plane * 2 * n + (size_t)a * n + k2) * ncol + blockIdx.x * W + w;
#pragma unroll
        for (int q = 0; q < R1; ++q) dst[(size_t)(R2 * q) * ncol] = z[q];
    }
}

// The inverse of k_mid_fwd: both parities back to the nm rows of the image.
template <int R1, int R2>
__global__ void __launch_bounds__(ColShape<R1, R2>::T)
    k_mid_inv(float2 *__restrict__ b0, const float2 *__restrict__ b1, int nm, int ncol,
              const float2 *__restrict__ tw, const int *__restrict__ done) {
    using S = ColShape<R1, R2>;
    constexpr int W = S::W, P = S::P, n = S::n;
    extern __shared__ float2 sm[];
    if (done && *done) return;
    const int w = threadIdx.x % W, tj = threadIdx.x / W;
    const size_t plane = (size_t)blockIdx.z * gridDim.y + blockIdx.y;
    const float2 *twB = tw + 2 * n;
    if (tj < 2 * R2) {
        const int a = tj / R2, k2 = tj - a * R2;
        const float2 *src = b1 + (plane * 2 * n + (size_t)a * n + k2) * ncol + blockIdx.x * W + w;
        float2 z[R1];
#pragma unroll
        for (int q = 0; q < R1; ++q) z[q] = src[(size_t)(R2 * q) * ncol];
#pragma unroll
        for (int q = 0; q < R1; ++q) z[q] = fftr::swap_ri(z[q], true);
        fftr::dft<R1>(z);
        float2 *dst = sm + (a * R1 * P + k2) * W + w;
        dst[0] = z[0];
#pragma unroll
        for (int q = 1; q < R1; ++q)
            dst[q * P * W] = cmul(z[q], __ldg(&twB[(q * 2 + a) * R2 + k2]));
    }
    __syncthreads();
    if (tj < R1) {
        const int j1 = tj;
        const float2 *src = sm + j1 * P * W + w;
        float2 t[R2], u[R2];
#pragma unroll
        for (int q = 0; q < R2; ++q) t[q] = src[q * W];
        fftr::dft<R2>(t);
        src += R1 * P * W;
#pragma unroll
        for (int q = 0; q < R2; ++q) u[q] = src[q * W];
        fftr::dft<R2>(u);
        half_twist<R2, 1>(u);
        float2 *dst = b0 + plane * nm * ncol + blockIdx.x * W + w;
#pragma unroll
        for (int q = 0; q < R2; ++q)
            if (j1 + R1 * q < nm)
                dst[(size_t)(j1 + R1 * q) * ncol] = make_float2(t[q].y + u[q].y, t[q].x + u[q].x);
    }
}

// Sizes of a doubled grid and of the one it is placed on (2-D: middle sizes 1).
struct Grids {
    int n0, n1, n2;  // image axes doubled
    int e0, e1, e2;  // engine lengths doubled
};

// blockIdx.y = index along the slowest axis, .z = segment
__global__ void k_embed(float2 *__restrict__ buf, const float *__restrict__ qr,
                        const float *__restrict__ qi, Grids g) {
    const unsigned plane = (unsigned)g.n1 * g.n2;
    const size_t src = ((size_t)blockIdx.z * g.n0 + blockIdx.y) * plane;
    auto place = [](int i, int n, int e) {  // displacement i - n / 2 modulo e
        return n == 1 ? 0 : (i < n / 2 ? i - n / 2 + e : i - n / 2);
    };
    buf += ((size_t)blockIdx.z * g.e0 + place((int)blockIdx.y, g.n0, g.e0)) * g.e1 * g.e2;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < plane;
         i += gridDim.x * blockDim.x) {
        const unsigned m = i / (unsigned)g.n2, f = i - m * g.n2;
        buf[(size_t)place((int)m, g.n1, g.e1) * g.e2 + place((int)f, g.n2, g.e2)] =
            make_float2(qr[src + i], qi[src + i]);
    }
}

// Natural order -> parity-major along every axis (index (k & 1) e + (k >> 1)), scaled.
__global__ void k_qf_parity(float2 *__restrict__ qf2, const float2 *__restrict__ qf, Grids g,
                            float scale) {
    const unsigned plane = (unsigned)g.e1 * g.e2;
    auto par = [](unsigned k, int e) { return e == 1 ? 0u : (k & 1u) * (e / 2) + (k >> 1); };
    qf += ((size_t)blockIdx.z * g.e0 + blockIdx.y) * plane;
    qf2 += ((size_t)blockIdx.z * g.e0 + par(blockIdx.y, g.e0)) * plane;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < plane;
         i += gridDim.x * blockDim.x) {
        const unsigned m = i / (unsigned)g.e2, f = i - m * g.e2;
        const float2 v = qf[i];
        qf2[(size_t)par(m, g.e1) * g.e2 + par(f, g.e2)] = make_float2(v.x * scale, v.y * scale);
    }
}

struct Entry {
    int n, r1, r2;
    int ps, t_row, t_col;
    size_t sm_row, sm_col;
    decltype(&k_row_fwd<8, 4>) fwd;
    decltype(&k_row_inv<8, 4>) inv;
    decltype(&k_col<8, 4>) col;
    decltype(&k_mid_fwd<8, 4>) mid_fwd;
    decltype(&k_mid_inv<8, 4>) mid_inv;
};

#define ER(A, B)                                                                              \
    {A * B, A, B, RowShape<A, B>::PS, RowShape<A, B>::T, ColShape<A, B>::T, RowShape<A, B>::smem, \
     ColShape<A, B>::smem, k_row_fwd<A, B>, k_row_inv<A, B>, k_col<A, B>, k_mid_fwd<A, B>,        \
     k_mid_inv<A, B>}
// Lengths at most a fifth apart (from 20); R1 about 2 R2, so that the R1 threads of a line
// in the one pass and the 2 R2 of the other keep the same block busy.
const Entry kTable[] = {
    ER(2, 2),   ER(4, 2),   ER(4, 3),   ER(4, 4),   ER(5, 4),   ER(6, 4),   ER(7, 4),
    ER(8, 4),   ER(10, 4),  ER(8, 6),   ER(14, 4),  ER(8, 8),   ER(10, 8),  ER(12, 8),  ER(14, 8),
    ER(16, 8),  ER(16, 9),  ER(16, 10), ER(16, 12), ER(20, 10), ER(20, 12), ER(16, 16),
    ER(24, 12), ER(20, 16), ER(24, 14), ER(24, 16), ER(25, 16), ER(28, 16), ER(30, 16),
    ER(32, 16), ER(32, 18), ER(32, 20), ER(32, 24), ER(32, 28), ER(32, 32),
};
#undef ER

int entry_for(int n) {
    int best = -1;
    for (int i = 0; i < (int)(sizeof(kTable) / sizeof(kTable[0])); ++i)
        if (kTable[i].n >= n && (best < 0 || kTable[i].n < kTable[best].n)) best = i;
    return best;
}

cudaError_t smem_opt(const Entry &e) {
    cudaError_t r = cudaFuncSetAttribute((const void *)e.fwd,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)e.sm_row);
    if (r == cudaSuccess)
        r = cudaFuncSetAttribute((const void *)e.inv, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)e.sm_row);
    if (r == cudaSuccess)
        r = cudaFuncSetAttribute((const void *)e.col, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)e.sm_col);
    for (const void *k : {(const void *)e.mid_fwd, (const void *)e.mid_inv})
        if (r == cudaSuccess)
            r = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)e.sm_col);
    return r;
}

cudaError_t twiddles(const Entry &e, float2 **tw) {
    const int n = e.n;
    std::vector<float2> h(4 * (size_t)n);
    for (int a = 0; a < 2; ++a) {
        // the register transforms' mean gain, parity 1 with the half twist's
        double gain = 1.0 + fftr::dft_gain(e.r1) + fftr::dft_gain(e.r2);
        for (int q = 0; a && q < e.r2; ++q) gain += fftr::mulw_gain(q, 2 * e.r2) / e.r2;
        for (int k2 = 0; k2 < e.r2; ++k2)
            for (int j1 = 0; j1 < e.r1; ++j1) {
                const double ang =
                    -3.14159265358979323846264338327950288 * ((double)j1 * (2 * k2 + a)) / n;
                const float2 w =
                    make_float2((float)(std::cos(ang) / gain), (float)(std::sin(ang) / gain));
                h[(size_t)(a * e.r2 + k2) * e.r1 + j1] = w;
                h[2 * (size_t)n + (size_t)(j1 * 2 + a) * e.r2 + k2] = w;
            }
    }
    cudaError_t r = cudaMalloc(tw, sizeof(float2) * h.size());
    if (r != cudaSuccess) return r;
    return cudaMemcpy(*tw, h.data(), sizeof(float2) * h.size(), cudaMemcpyHostToDevice);
}

Grids grids(const ToepRowsPlan &p) {
    const bool three = p.nm > 1;
    return Grids{2 * p.ns, three ? 2 * p.nm : 1, 2 * p.nf, 2 * p.es, three ? 2 * p.em : 1, 2 * p.ef};
}

// blocks along x for a plane of n elements, rows x segs planes
dim3 plane_grid(size_t n, int rows, int segs) {
    const size_t want = 148 * 16, planes = (size_t)rows * segs;
    const size_t x = std::max<size_t>(1, std::min((n + 255) / 256, want / planes + 1));
    return dim3((unsigned)x, rows, segs);
}

}  // namespace

bool toep_rows_plan(int ns, int nm, int nf, int C, int L1, ToepRowsPlan *plan) {
    ToepRowsPlan p;
    p.ns = ns;
    p.nm = nm;
    p.nf = nf;
    p.C = C;
    p.L1 = L1;
    p.e_s = entry_for(ns);
    p.e_m = nm > 1 ? entry_for(nm) : 0;
    p.e_f = entry_for(nf);
    if (ns < 1 || nm < 1 || nf < 1 || C < 1 || L1 < 1 || L1 > 65535 || p.e_s < 0 || p.e_m < 0 ||
        p.e_f < 0)
        return false;
    p.es = kTable[p.e_s].n;
    p.em = nm > 1 ? kTable[p.e_m].n : 1;
    p.ef = kTable[p.e_f].n;
    // Half spectra of at most 320 MB: the kernels are bound by issue and latency, not by
    // memory, so chunks that fit the L2 only add launches and tails (512x512 x 32 coils, 20
    // updates: 6.54 ms in one chunk of 134 MB, 6.90 in 64 MB chunks, 7.33 in 32 MB ones).
    // A whole number of coil sets where they fit, for the reuse of Qf_l in k_col.
    const size_t job = sizeof(float2) * p.job_elems();
    const size_t fit = std::max<size_t>(1, ((size_t)320 << 20) / job);
    const size_t jobs = (size_t)L1 * C;
    const size_t parts = (jobs + fit - 1) / fit;
    size_t chunk = (jobs + parts - 1) / parts;
    if (chunk > (size_t)C) chunk = std::min(fit / C * C, (chunk + C - 1) / C * C);
    else if (fit >= (size_t)C) chunk = C;
    p.chunk = (int)std::min<size_t>(std::max<size_t>(chunk, 1), 65535);
    for (int e : {p.e_s, p.e_m, p.e_f})
        if (smem_opt(kTable[e]) != cudaSuccess) return false;
    *plan = p;
    return true;
}

cudaError_t toep_rows_twiddles(const ToepRowsPlan &p, float2 *tw[3]) {
    const int e[3] = {p.e_s, p.e_m, p.e_f};
    for (int a = 0; a < 3; ++a)
        if (a != 1 || p.nm > 1) {
            const cudaError_t r = twiddles(kTable[e[a]], &tw[a]);
            if (r != cudaSuccess) return r;
        }
    return cudaSuccess;
}

cudaError_t toep_rows_embed(const ToepRowsPlan &p, float2 *fftbuf, const float *q_r,
                            const float *q_i, int nl, cudaStream_t st) {
    if (p.es != p.ns || p.em != p.nm || p.ef != p.nf) {
        const cudaError_t e = cudaMemsetAsync(fftbuf, 0, sizeof(float2) * p.q_elems() * nl, st);
        if (e != cudaSuccess) return e;
    }
    const Grids g = grids(p);
    k_embed<<<plane_grid((size_t)g.n1 * g.n2, g.n0, nl), 256, 0, st>>>(fftbuf, q_r, q_i, g);
    return cudaGetLastError();
}

cudaError_t toep_rows_qf(const ToepRowsPlan &p, float2 *qf2, const float2 *qf, float scale, int nl,
                         cudaStream_t st) {
    const Grids g = grids(p);
    k_qf_parity<<<plane_grid((size_t)g.e1 * g.e2, g.e0, nl), 256, 0, st>>>(qf2, qf, g, scale);
    return cudaGetLastError();
}

cudaError_t toep_rows_apply(const ToepRowsPlan &p, float2 *q, const float2 *x, const float2 *sens,
                            const float2 *eph, float2 *b0, float2 *b1, const float2 *qf2,
                            const int *done, float2 *const tw[3], cudaStream_t st) {
    const Entry &es = kTable[p.e_s], &em = kTable[p.e_m], &ef = kTable[p.e_f];
    const bool three = p.nm > 1;
    const int rows = p.ns * p.nm, cols = 2 * p.ef, ncol = (three ? 2 * p.em : 1) * cols;
    const unsigned groups = (unsigned)((rows + ef.ps - 1) / ef.ps);
    float2 *rbuf = three ? b0 : b1;  // the rows' spectra
    const int jobs = p.L1 * p.C;
    for (int j0 = 0; j0 < jobs; j0 += p.chunk) {
        const int nj = std::min(p.chunk, jobs - j0);
        ef.fwd<<<dim3(groups, nj), ef.t_row, ef.sm_row, st>>>(rbuf, x, sens, eph, rows, p.nf, p.C,
                                                             j0, tw[2], done);
        const dim3 mid(cols / kColW, p.ns, nj);
        if (three)
            em.mid_fwd<<<mid, em.t_col, em.sm_col, st>>>(b1, b0, p.nm, cols, tw[1], done);
        const bool jobs_x = three && ncol / kColW <= 65535;
        const dim3 gc = jobs_x ? dim3(nj, ncol / kColW) : dim3(ncol / kColW, nj);
        es.col<<<gc, es.t_col, es.sm_col, st>>>(b1, qf2, p.ns, ncol, p.C, j0, jobs_x ? 1 : 0,
                                               tw[0], done);
        if (three)
            em.mid_inv<<<mid, em.t_col, em.sm_col, st>>>(b0, b1, p.nm, cols, tw[1], done);
        // cluster over the transforms: enough ranks for some sixteen blocks per SM (at
        // most 8, the portable cluster size), as many as give every one the same number
        // of transforms; a block of a 3-D image takes them all (256x256x32 x 4: 96 us
        // per launch with one each, for the cluster's barriers and the exchange)
        const int want = std::min(8, std::max(1, (int)((148 * 16 + groups - 1) / groups)));
        const int most = std::min(want, nj);
        const int rounds = (nj + most - 1) / most, cs = (nj + rounds - 1) / rounds;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(groups, cs);
        cfg.blockDim = dim3(ef.t_row);
        cfg.dynamicSmemBytes = ef.sm_row;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1;
        attr[0].val.clusterDim.y = cs;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, ef.inv, q, (const float2 *)rbuf, sens, eph,
                                                 rows, p.nf, p.C, j0, nj, j0 == 0 ? 1 : 0,
                                                 (const float2 *)tw[2], done);
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

}  // namespace imp
