// Pruned F^H F engine of 2-D images on mixed-radix lengths.
//
// Along each axis of length n the zero-padded 2n-point transform splits by
// output parity a into two n-point transforms of x[j] w_2n^{a j}; the inverse
// restricted to [0, n) is the parity sum of two n-point inverses (the doubled
// grid never exists).  With n = R1 R2 (R1, R2 <= 32), j = j1 + R1 j2 and
// k = k2 + R2 k1, an n-point line is an R2-point register DFT per j1, the
// twiddle w_2n^{j1 (2 k2 + a)} (it carries the parity's j1 part; the rest,
// w_{2 R2}^{a j2}, is a compile-time constant) and an R1-point register DFT
// per k2.  Three kernels per chunk of (segment, coil) transforms:
//   k_row_fwd  rows along f: forms S_c e_l x from global memory in registers,
//              both parities, writes [s][a][k];
//   k_col      columns along s, in place: both parities forward, x Qf_l,
//              inverse, parity sum;
//   k_row_inv  rows along f: inverse, parity sum, conj(e_l S_c), summed over the
//              block's transforms in registers and over the cluster's blocks in
//              distributed shared memory.
// Every first DFT reads global memory straight into registers and every last
// one writes it from registers, so a row kernel makes one trip through shared
// memory and the column kernel two.  The inverse transforms run as forward
// ones on values with real and imaginary parts exchanged.
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

// Columns [blockIdx.x W, + W) of the transform blockIdx.y, in place.
template <int R1, int R2>
__global__ void __launch_bounds__(ColShape<R1, R2>::T, cmax(1, 512 / ColShape<R1, R2>::T))
    k_col(float2 *__restrict__ b1, const float2 *__restrict__ qf2, int ns, int ncol, int C,
          int job0, const float2 *__restrict__ tw, const int *__restrict__ done) {
    using S = ColShape<R1, R2>;
    constexpr int W = S::W, P = S::P, n = S::n;
    extern __shared__ float2 sm[];
    if (done && *done) return;
    const int l = (job0 + blockIdx.y) / C;
    const int w = threadIdx.x % W, tj = threadIdx.x / W;
    float2 *col = b1 + (size_t)blockIdx.y * ns * ncol + blockIdx.x * W + w;
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
        const float2 *qc = qf2 + (size_t)l * 2 * n * ncol + (size_t)(a * n + k2) * ncol +
                           blockIdx.x * W + w;
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

__global__ void k_embed(float2 *__restrict__ buf, const float *__restrict__ qr,
                        const float *__restrict__ qi, int ns, int nf, int es, int ef) {
    const size_t G = (size_t)4 * ns * nf;
    buf += (size_t)blockIdx.y * 4 * es * ef;
    qr += blockIdx.y * G;
    qi += blockIdx.y * G;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < G;
         i += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(i / (2 * nf)), y = (int)(i % (2 * nf));
        const int dx = x - ns, dy = y - nf;  // displacement
        const size_t o = (size_t)(dx < 0 ? dx + 2 * es : dx) * (2 * ef) + (dy < 0 ? dy + 2 * ef : dy);
        buf[o] = make_float2(qr[i], qi[i]);
    }
}

// [2es][2ef] natural order -> row (as es + ks), column (af ef + kf), scaled
__global__ void k_qf_parity(float2 *__restrict__ qf2, const float2 *__restrict__ qf, int es,
                            int ef, float scale) {
    const size_t G = (size_t)4 * es * ef;
    qf2 += blockIdx.y * G;
    qf += blockIdx.y * G;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < G;
         i += (size_t)gridDim.x * blockDim.x) {
        const int ks = (int)(i / (2 * ef)), kf = (int)(i % (2 * ef));
        const float2 v = qf[i];
        qf2[(size_t)((ks & 1) * es + (ks >> 1)) * (2 * ef) + (kf & 1) * ef + (kf >> 1)] =
            make_float2(v.x * scale, v.y * scale);
    }
}

struct Entry {
    int n, r1, r2;
    int ps, t_row, t_col;
    size_t sm_row, sm_col;
    decltype(&k_row_fwd<8, 4>) fwd;
    decltype(&k_row_inv<8, 4>) inv;
    decltype(&k_col<8, 4>) col;
};

#define ER(A, B)                                                                              \
    {A * B, A, B, RowShape<A, B>::PS, RowShape<A, B>::T, ColShape<A, B>::T, RowShape<A, B>::smem, \
     ColShape<A, B>::smem, k_row_fwd<A, B>, k_row_inv<A, B>, k_col<A, B>}
// Lengths at most a fifth apart; R1 about 2 R2, so that the R1 threads of a line
// in the one pass and the 2 R2 of the other keep the same block busy.
const Entry kTable[] = {
    ER(4, 4),   ER(8, 4),   ER(8, 6),   ER(8, 8),   ER(10, 8),  ER(12, 8),  ER(14, 8),
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
    return r;
}

cudaError_t twiddles(const Entry &e, float2 **tw) {
    const int n = e.n;
    std::vector<float2> h(4 * (size_t)n);
    for (int a = 0; a < 2; ++a)
        for (int k2 = 0; k2 < e.r2; ++k2)
            for (int j1 = 0; j1 < e.r1; ++j1) {
                const double ang =
                    -3.14159265358979323846264338327950288 * ((double)j1 * (2 * k2 + a)) / n;
                const float2 w = make_float2((float)std::cos(ang), (float)std::sin(ang));
                h[(size_t)(a * e.r2 + k2) * e.r1 + j1] = w;
                h[2 * (size_t)n + (size_t)(j1 * 2 + a) * e.r2 + k2] = w;
            }
    cudaError_t r = cudaMalloc(tw, sizeof(float2) * h.size());
    if (r != cudaSuccess) return r;
    return cudaMemcpy(*tw, h.data(), sizeof(float2) * h.size(), cudaMemcpyHostToDevice);
}

unsigned blocks_for(size_t n) { return (unsigned)std::min<size_t>((n + 255) / 256, 148 * 16); }

}  // namespace

bool toep_rows_plan(int ns, int nf, int C, int L1, ToepRowsPlan *plan) {
    ToepRowsPlan p;
    p.ns = ns;
    p.nf = nf;
    p.C = C;
    p.L1 = L1;
    p.e_s = entry_for(ns);
    p.e_f = entry_for(nf);
    if (ns < 1 || nf < 1 || C < 1 || L1 < 1 || p.e_s < 0 || p.e_f < 0) return false;
    p.es = kTable[p.e_s].n;
    p.ef = kTable[p.e_f].n;
    // Half spectra of at most 256 MB: the kernels are bound by issue and latency, not by
    // memory, so chunks that fit the L2 only add launches and tails (512x512 x 32 coils, 20
    // updates: 6.54 ms in one chunk of 134 MB, 6.90 in 64 MB chunks, 7.33 in 32 MB ones).
    const size_t job = sizeof(float2) * (size_t)ns * 2 * p.ef;
    const size_t fit = std::max<size_t>(1, ((size_t)256 << 20) / job);
    const size_t jobs = (size_t)L1 * C;
    const size_t parts = (jobs + fit - 1) / fit;
    p.chunk = (int)std::min<size_t>((jobs + parts - 1) / parts, 65535);
    if (smem_opt(kTable[p.e_s]) != cudaSuccess || smem_opt(kTable[p.e_f]) != cudaSuccess)
        return false;
    *plan = p;
    return true;
}

cudaError_t toep_rows_twiddles(const ToepRowsPlan &p, float2 **tw_s, float2 **tw_f) {
    const cudaError_t e = twiddles(kTable[p.e_s], tw_s);
    return e != cudaSuccess ? e : twiddles(kTable[p.e_f], tw_f);
}

cudaError_t toep_rows_embed(const ToepRowsPlan &p, float2 *fftbuf, const float *q_r,
                            const float *q_i, int nl, cudaStream_t st) {
    if (p.es != p.ns || p.ef != p.nf) {
        const cudaError_t e = cudaMemsetAsync(fftbuf, 0, sizeof(float2) * p.q_elems() * nl, st);
        if (e != cudaSuccess) return e;
    }
    k_embed<<<dim3(blocks_for((size_t)4 * p.ns * p.nf), nl), 256, 0, st>>>(
        fftbuf, q_r, q_i, p.ns, p.nf, p.es, p.ef);
    return cudaGetLastError();
}

cudaError_t toep_rows_qf(const ToepRowsPlan &p, float2 *qf2, const float2 *qf, float scale, int nl,
                         cudaStream_t st) {
    k_qf_parity<<<dim3(blocks_for(p.q_elems()), nl), 256, 0, st>>>(qf2, qf, p.es, p.ef, scale);
    return cudaGetLastError();
}

cudaError_t toep_rows_apply(const ToepRowsPlan &p, float2 *q, const float2 *x, const float2 *sens,
                            const float2 *eph, float2 *b1, const float2 *qf2, const int *done,
                            const float2 *tw_s, const float2 *tw_f, cudaStream_t st) {
    const Entry &es = kTable[p.e_s], &ef = kTable[p.e_f];
    const unsigned groups = (unsigned)((p.ns + ef.ps - 1) / ef.ps);
    const int jobs = p.L1 * p.C;
    for (int j0 = 0; j0 < jobs; j0 += p.chunk) {
        const int nj = std::min(p.chunk, jobs - j0);
        ef.fwd<<<dim3(groups, nj), ef.t_row, ef.sm_row, st>>>(b1, x, sens, eph, p.ns, p.nf, p.C,
                                                             j0, tw_f, done);
        es.col<<<dim3(2 * p.ef / kColW, nj), es.t_col, es.sm_col, st>>>(
            b1, qf2, p.ns, 2 * p.ef, p.C, j0, tw_s, done);
        // cluster over the transforms: as many ranks as give every one the same
        // number of them (at most 8, the portable cluster size)
        const int rounds = (nj + 7) / 8, cs = (nj + rounds - 1) / rounds;
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
        const cudaError_t e =
            cudaLaunchKernelEx(&cfg, ef.inv, q, (const float2 *)b1, sens, eph, p.ns, p.nf, p.C, j0,
                               nj, j0 == 0 ? 1 : 0, tw_f, done);
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

}  // namespace imp
