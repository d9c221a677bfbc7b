// Toeplitz reconstruction path on B200.
//
//   Q_l   = deapod(crop(IFFT(KB-grid_{2k}(h_l(t)))))          toeplitz/computeQ.cmem.cu:401-754
//   F^H d = sum_c conj(S_c) sum_l e^{+i w (tau l + t0)}
//             deapod(crop(IFFT(KB-grid_k(h_l(t) d_c))))      toeplitz/computeFH.cmem.cu:469-1129
//   A^H A p = sum_c conj(S_c) sum_l e^{+i w tau_l}
//             crop(IFFT(Qf_l . FFT(pad(e^{-i w tau_l} S_c p)))) / G   toeplitz/recon.cu:1113-1465
//   CG on (A^H A + lambda D^H W D) x = F^H d from x = 0, best-residual
//   iterate returned                                          toeplitz/recon.cu:1724-2191
//
// B200 design (not a translation of the reference kernels):
// * gridding is a scatter of each sample's separable KB footprint with vector
//   float2 atomics straight into the ifftshifted position of the FFT buffer,
//   one warp per sample (the lanes on contiguous cells), for the (at most two)
//   time segments whose Hanning window covers the sample -- no CPU binning, no
//   overflow path, no host round trips; the inverse transform is cropped to the
//   cells the post kernels read;
// * every shift / crop / deapodisation / phase / SENSE step is an index map
//   fused into the kernels around the FFTs; the FFTs are this library's own
//   (the pruned mixed-radix F^H F engine of toep_rows.cu, the mixed-radix grid
//   transform of grid_fft.cu for the gridding grids, Qf_l and the zero-padded
//   chain of sides longer than the engine's longest length);
// * Qf_l, sensitivities and phase factors stay resident in HBM; one CG
//   iteration (FFT chain + FP64 CG scalars, best-iterate tracking and the
//   tolerance stop all on the device) is captured once as a CUDA graph.
#include "../../include/impatient_b200.h"
#include "common.cuh"
#include "io.h"
#include "toeplitz.cuh"
#include "tv.cuh"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <string>
#include <sys/stat.h>
#include <vector>

namespace imp {

namespace {

constexpr float kPiF = 3.1415926535897932384626433832795029f;
constexpr float kKW = 4.0f;  // kernel width
constexpr int kVB = 256;
constexpr int kTBlocks = 296;
constexpr int kMaxTaps = 12;

enum { T_PQ = 0, T_RR = 1, T_NORM = 2, T_SCAL = 3 };
// scalars (after the three partial slabs): beta2[2], resBest, normFhd, cur, done
struct TScal {
    double beta2[2];
    double res_best;
    double norm_fhd;
    int cur;
    int done;
    double tol;   // stop when sqrt(|r|^2 / |F^H d|^2) < tol
    int iters;    // CG updates performed since the solve started
    unsigned arrive;  // k_t_dir blocks done with this update (the last one finishes it)
};

__device__ __forceinline__ TScal *scal(double *dots) {
    return reinterpret_cast<TScal *>(dots + T_SCAL * kTBlocks);
}

// Modified Bessel I0 (Abramowitz & Stegun 9.8.1, 9.8.2).
__device__ __forceinline__ float bessi0f(float x) {
    const float ax = fabsf(x);
    if (ax < 3.75f) {
        float y = x / 3.75f;
        y *= y;
        return 1.0f + y * (3.5156229f + y * (3.0899424f + y * (1.2067492f + y * (0.2659732f +
                                         y * (0.360768e-1f + y * 0.45813e-2f)))));
    }
    const float y = 3.75f / ax;
    return (expf(ax) * rsqrtf(ax)) *
           (0.39894228f + y * (0.1328592e-1f + y * (0.225319e-2f + y * (-0.157565e-2f + y * (
                                0.916281e-2f + y * (-0.2057706e-1f + y * (0.2635537e-1f + y * (
                                                       -0.1647633e-1f + y * 0.392377e-2f))))))));
}

// KB weight at distance d (image-grid units): toeplitz/GPU_kernels.cu:270-300.
__device__ __forceinline__ float kb_weight(float d, float beta) {
    if (d > 0.5f * kKW) return 0.f;
    const float a = 1.0f - (4.0f / (kKW * kKW)) * d * d;
    if (!(a >= 0.f)) return 0.f;
    return bessi0f(beta * sqrtf(a)) * (1.0f / kKW);
}

__device__ __forceinline__ float hanning(float t, float tau, int l, float t0) {
    const float x = t - tau * (float)l - t0;
    return fabsf(x) < tau ? 0.5f + 0.5f * cosf(kPiF * x / tau) : 0.f;
}

// KB transform shape for deapodisation: toeplitz/gridding_utils.cu:60-110.
__device__ __forceinline__ float kb_transform(float u, float beta) {
    const float e = kPiF * kPiF * kKW * kKW * u * u - beta * beta;
    if (e > 0.f) {
        const float s = sqrtf(e);
        return sinf(s) / s;
    }
    if (e < 0.f) {
        const float s = sqrtf(-e);
        return sinhf(s) / s;
    }
    return 1.f;
}

// Scatter gridding, one warp per sample: each sample's separable KB footprint
// is added into the ifftshifted position (X - gs/2) mod gs of every cell X it
// covers (ready for the inverse FFT), for a batch of grids at once: segments
// [l0, l0 + nl) x coils [0, nc) of dr / di, grid (l - l0) nc + c at
// `cells` elements each.  Without data (Q: the samples' real window values) a
// grid holds two segments, 2 m in the real and 2 m + 1 in the imaginary part,
// the latter scaled by segw's pair_scale (l0 even, nc 1, L1 segments in all).  A sample's footprint, indices and KB weights are
// formed once for the (at most two) segments whose Hanning window covers it
// and for all coils, whose values the lanes load in parallel; one launch per
// (segment, coil) had recomputed them each time and was too short to fill the
// GPU (256x256, 16 coils, 13 segments: 208 launches of 14 us).  The lanes take
// the cells of the footprint's two fastest-varying axes (z and y in 3-D, y and
// x in 2-D; up to 9 x 9 at OS 2), so one atomic instruction of the warp updates
// a few contiguous runs of a grid instead of 32 scattered cells, and the outer
// axis is looped.  No unit is full: with one value per sample (Q of 128x128x32) the
// SMs issue at 65 % and the L2 is at 43 %; with 16 coils the L1's atomic path is at
// 62 %, behind long waits for the coils' values.
constexpr int kGridWarps = 8;
constexpr int kGridCoils = 32;  // coils per launch at most

// Sum of the samples' window values per segment: how strong each segment's Q is.
// Neighbouring samples are nearly always of the same segments: one addition per warp
// then (a shared-memory addition per lane loops: Q of 128x128x32 3.29 ms against 3.17;
// this kernel takes 18 us of it, for 524288 samples).
constexpr int kSegShared = 1024;
__global__ void k_seg_weights(float *w, const float *t, int M, float tau, float t0, int L1) {
    __shared__ float sh[kSegShared];
    const bool own = L1 <= kSegShared;
    float *sum = own ? sh : w;
    if (own)
        for (int l = threadIdx.x; l < L1; l += blockDim.x) sh[l] = 0.f;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int s0 = blockIdx.x * blockDim.x + threadIdx.x - lane; s0 < M;
         s0 += gridDim.x * blockDim.x) {
        const float ts = __ldg(&t[min(s0 + lane, M - 1)]), xs = (ts - t0) / tau;
        const bool in = s0 + lane < M && tau > 0.f && xs > -2.f && xs < (float)L1 + 1.f;
        const int la = in ? (int)floorf(xs) - 1 : INT_MIN;  // windows la .. la + 3
        int same;
        __match_all_sync(~0u, la, &same);
        if (same && la == INT_MIN) continue;
        for (int d = 0; d < 4; ++d) {
            const int l = la + d;
            float h = in && l >= 0 && l < L1 ? hanning(ts, tau, l, t0) : 0.f;
            if (same)
                for (int o = 16; o; o >>= 1) h += __shfl_xor_sync(~0u, h, o);
            if (h != 0.f && (!same || lane == 0)) atomicAdd(&sum[l], h);
        }
    }
    __syncthreads();
    if (own)
        for (int l = threadIdx.x; l < L1; l += blockDim.x)
            if (sh[l] != 0.f) atomicAdd(&w[l], sh[l]);
}

// Power of two (or with sign -1 its inverse) that brings the second of two segments that
// share a grid to the strength of the first, of weights w.x and w.y.  Each segment's Q then
// has the accuracy of a grid of its own; without it one of 1e-4 of its partner's weight
// came out 7.9e-5 from 64 bits instead of 1.1e-5, and one without samples not zero.
__device__ __forceinline__ float pair_scale(float2 w, int sign) {
    if (!(w.x > 0.f && w.y > 0.f)) return 1.f;
    const int k = (__float_as_int(w.x) >> 23) - (__float_as_int(w.y) >> 23);
    return __int_as_float((127 + sign * min(max(k, -60), 60)) << 23);
}

// ONE: a single value per sample and step (nc 1), kept in registers (the coil
// loop's shared-memory read per cell costs: Q of 128x128x32 3.41 -> 3.09 ms).
// D3: a 3-D grid; the axes' roles are compile-time, their arrays in registers.
// The samples are strided over kGridBlocks resident blocks per SM.
constexpr int kGridBlocks = 6;
template <bool ONE, bool D3>
__global__ void __launch_bounds__(kGridWarps * 32, kGridBlocks)
    k_grid_w(float2 *grid, size_t cells, const float *kx, const float *ky, const float *kz,
             const float *t, const float *dr, const float *di, int M, GridSpec g, float tau,
             float t0, int l0, int nl, int nc, int L1, const float2 *segw) {
    __shared__ float wsh[kGridWarps][3][kMaxTaps];
    __shared__ float2 vsh[ONE ? 1 : kGridWarps][kGridCoils];
    if (!(tau > 0.f)) return;  // every window is empty
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float(&ws)[3][kMaxTaps] = wsh[wid];
    float2(&vs)[kGridCoils] = vsh[ONE ? 0 : wid];
    const float inv_os = 1.0f / g.os;
    // loop axis A, lane axes B (slower) and Cc (faster)
    constexpr int A = D3 ? 0 : 2, B = D3 ? 1 : 0, Cc = D3 ? 2 : 1;
    for (int s = blockIdx.x * kGridWarps + wid; s < M; s += gridDim.x * kGridWarps) {
        // segments around t: every lane reads the same sample, so all of this is warp-uniform
        const float ts = __ldg(&t[s]);
        const float xs = (ts - t0) / tau;
        if (!(xs > (float)l0 - 2.f && xs < (float)(l0 + nl) + 1.f)) continue;
        const int lf = (int)floorf(xs);
        // Q: step m stands for the segments 2 m and 2 m + 1 (real and imaginary part)
        const int la = dr ? max(l0, lf - 1) : max(l0, lf - 1) >> 1;
        const int lb = dr ? min(l0 + nl, lf + 3) : (min(l0 + nl, lf + 3) + 1) >> 1;
        bool ready = false;
        int lo[3], cnt[3];
        for (int l = la; l < lb; ++l) {
            const float h = hanning(ts, tau, dr ? l : 2 * l, t0);
            float h1 = !dr && 2 * l + 1 < L1 ? hanning(ts, tau, 2 * l + 1, t0) : 0.f;
            if (h == 0.f && h1 == 0.f) continue;
            if (!dr && h1 != 0.f) h1 *= pair_scale(__ldg(&segw[l]), 1);
            float2 v1 = make_float2(h, h1);
            if constexpr (ONE) {
                if (dr) {
                    v1 = make_float2(h * __ldg(&dr[s]), h * (di ? __ldg(&di[s]) : 0.f));
                    if (v1.x == 0.f && v1.y == 0.f) continue;
                }
            } else {
                __syncwarp();  // the previous segment's values have been read
                for (int c = lane; c < nc; c += 32) {
                    const size_t i = (size_t)c * M + s;
                    vs[c] = make_float2(h * __ldg(&dr[i]), h * (di ? __ldg(&di[i]) : 0.f));
                }
            }
            if (!ready) {
                ready = true;
                const float k3[3] = {__ldg(&kx[s]), __ldg(&ky[s]), D3 ? __ldg(&kz[s]) : 0.f};
                float cc[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    if (a == 2 && !D3) {
                        lo[2] = 0;
                        cnt[2] = 1;
                        cc[2] = 0.f;
                        continue;
                    }
                    const float c = g.os * (g.kscale * k3[a] + 0.5f * (float)g.img[a]);
                    const float r = 0.5f * kKW * g.os;
                    int a0 = (int)ceilf(c - r), a1 = (int)floorf(c + r);
                    a0 = max(a0, 0);
                    a1 = min(a1, g.gs[a] - 1);
                    a1 = min(a1, a0 + kMaxTaps - 1);
                    lo[a] = a0;
                    cnt[a] = max(a1 - a0 + 1, 0);
                    cc[a] = c;
                }
                for (int q = lane; q < 3 * kMaxTaps; q += 32) {
                    const int a = q / kMaxTaps, j = q - a * kMaxTaps;
                    if (j < cnt[a])
                        ws[a][j] = (a == 2 && !D3)
                                       ? 1.f
                                       : kb_weight(fabsf(cc[a] - (float)(lo[a] + j)) * inv_os,
                                                   g.beta);
                }
            }
            __syncwarp();
            // A covered cell's shifted index is lo + j - gs / 2 modulo gs; with + (gs + 1) / 2
            // instead it is below 2 gs and wraps at most once (one conditional subtraction, no
            // division per cell).  gs is odd where an axis' oversampled length, rounded up in
            // FP32, passes the multiple of four it was made for (z: 61 for 38 at 1.5).  The loop
            // axis steps by a fixed stride and wraps once.  (Aligned pairs of cells as 16-byte
            // atomics measured no faster: 5.32 against 5.22 ms for Q of 128x128x32 when a grid
            // held one segment.)
            float2 *gl = grid + (size_t)(l - (dr ? l0 : l0 >> 1)) * nc * cells;
            const int nbc = cnt[B] * cnt[Cc];
            int a0 = D3 ? lo[A] + (g.gs[A] + 1) / 2 : 0;
            if (a0 >= g.gs[A]) a0 -= g.gs[A];
            const size_t astride = D3 ? (size_t)g.gs[1] * g.gs[2] : 0;
            const size_t awrap = astride * g.gs[A];
            const int rowlen = D3 ? g.gs[2] : g.gs[1];  // stride of axis B
            for (int p = lane; p < nbc; p += 32) {
                const int jb = p / cnt[Cc], jc = p - jb * cnt[Cc];
                const float wbc = ws[B][jb] * ws[Cc][jc];
                if (wbc == 0.f) continue;
                int ib = lo[B] + jb + (g.gs[B] + 1) / 2;
                if (ib >= g.gs[B]) ib -= g.gs[B];
                int ic = lo[Cc] + jc + (g.gs[Cc] + 1) / 2;
                if (ic >= g.gs[Cc]) ic -= g.gs[Cc];
                size_t cell = (size_t)a0 * astride + (size_t)ib * rowlen + ic;
                int ia = a0;
                for (int ja = 0; ja < cnt[A]; ++ja) {
                    const float ww = wbc * ws[A][ja];
                    if (ww != 0.f) {
                        if constexpr (ONE)
                            atomicAdd(&gl[cell], make_float2(ww * v1.x, ww * v1.y));
                        else
                            for (int c = 0; c < nc; ++c) {
                                const float2 v = vs[c];
                                atomicAdd(&gl[(size_t)c * cells + cell],
                                          make_float2(ww * v.x, ww * v.y));
                            }
                    }
                    cell += astride;
                    if (++ia == g.gs[A]) {
                        ia = 0;
                        cell -= awrap;
                    }
                }
            }
        }
        __syncwarp();  // the next sample overwrites ws
    }
}

struct NV {
    int v[3];
};

// Voxel coordinates (x, y, z) of a voxel-order index (2-D [x][y], 3-D
// [y][x][z]); indices below 2^32 with 32-bit divisions, which cost a fraction
// of a 64-bit one.
template <typename U>
__device__ __forceinline__ void vox_xyz_u(U q, const int nv[3], bool is3d, int &x, int &y, int &z) {
    if (!is3d) {
        const U c = q / (unsigned)nv[1];
        x = (int)c;
        y = (int)(q - c * (unsigned)nv[1]);
        z = 0;
    } else {
        const U yx = q / (unsigned)nv[2], r = yx / (unsigned)nv[1];
        z = (int)(q - yx * (unsigned)nv[2]);
        y = (int)r;
        x = (int)(yx - r * (unsigned)nv[1]);
    }
}
__device__ __forceinline__ void vox_xyz(size_t q, const int nv[3], bool is3d, int &x, int &y,
                                        int &z) {
    if (q >> 32) vox_xyz_u<unsigned long long>(q, nv, is3d, x, y, z);
    else vox_xyz_u<unsigned>((unsigned)q, nv, is3d, x, y, z);
}

// (i + n / 2) mod n of an even n, i < n
__device__ __forceinline__ int half_turn(int i, int n) {
    return i < n / 2 ? i + n / 2 : i - n / 2;
}

// Where image voxel (x, y, z) of a gridding problem sits after the inverse FFT
// (fftshift and crop of the centre), where its negative does, and its
// deapodisation factor.
struct GridAt {
    size_t idx, neg;
    float s;
};
__device__ __forceinline__ GridAt grid_at(const GridSpec &g, int x, int y, int z) {
    const int c[3] = {x, y, z};
    GridAt r{0, 0, 1.f};
    float kern = 1.f;
    for (int a = 0; a < 3; ++a) {
        // the centred crop, shifted: c - img/2 modulo gs
        int j = c[a] - g.img[a] / 2;
        if (j < 0) j += g.gs[a];
        r.idx = r.idx * g.gs[a] + j;
        r.neg = r.neg * g.gs[a] + (j ? g.gs[a] - j : 0);
        if (a < 2 || g.is3d)
            kern *= kb_transform(((float)c[a] - 0.5f * (float)g.img[a]) / (float)g.img[a], g.beta);
    }
    const float osd = g.is3d ? g.os * g.os * g.os : g.os * g.os;
    r.s = 1.0f / (kern * osd);
    return r;
}

// Q_l of nl segments from the inverse-FFT'd grids of two segments each, in the
// reference layout.  The gridded windows are real, so each segment's transform
// F is Hermitian and G = F_0 + i F_1 separates into F_0 = (G(r) + conj G(-r)) / 2
// and F_1 = (G(r) - conj G(-r)) / 2i: half the transforms and scatters.  A
// voxel's indices and deapodisation (sinh per axis) serve all segments.  segw: the
// weights of these segments, two per grid; one without samples gives zeros.
__global__ void k_q_post(const float2 *A, size_t cells, GridSpec g, NV n2, float *qr, float *qi,
                         size_t G2, int nl, const float2 *segw) {
    // n2: the 2N grid in voxel axis order
    const int nv[3] = {n2.v[0], n2.v[1], n2.v[2]};
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < G2;
         q += (size_t)gridDim.x * blockDim.x) {
        int x, y, z;
        vox_xyz(q, nv, g.is3d, x, y, z);
        const GridAt at = grid_at(g, x, y, z);
        const float s = 0.5f * at.s;
        for (int l = 0; l < nl; l += 2) {
            const float2 *Al = A + (size_t)(l >> 1) * cells;
            const float2 v = Al[at.idx], m = Al[at.neg], w = __ldg(&segw[l >> 1]);
            const float s0 = w.x > 0.f ? s : 0.f;
            qr[(size_t)l * G2 + q] = (v.x + m.x) * s0;
            qi[(size_t)l * G2 + q] = (v.y - m.y) * s0;
            if (l + 1 < nl) {
                const float s1 = w.y > 0.f ? s * pair_scale(w, -1) : 0.f;
                qr[(size_t)(l + 1) * G2 + q] = (v.y + m.y) * s1;
                qi[(size_t)(l + 1) * G2 + q] = (m.x - v.x) * s1;
            }
        }
    }
}

// Q_l given in the reference layout -> ifftshifted FFT input.
__global__ void k_q_shift(const float *qr, const float *qi, NV n2, bool is3d, float2 *fftbuf,
                          size_t G2) {
    const int nv[3] = {n2.v[0], n2.v[1], n2.v[2]};
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < G2;
         q += (size_t)gridDim.x * blockDim.x) {
        int x, y, z;
        vox_xyz(q, nv, is3d, x, y, z);
        size_t o;
        if (!is3d)
            o = (size_t)half_turn(x, nv[0]) * nv[1] + half_turn(y, nv[1]);
        else
            o = ((size_t)half_turn(y, nv[0]) * nv[1] + half_turn(x, nv[1])) * nv[2] +
                half_turn(z, nv[2]);
        fftbuf[o] = make_float2(qr[q], qi[q]);
    }
}

// F^H d accumulation of a batch of grids, segments [l0, l0 + nl) x nc coils:
// acc += sum_l e^{+i w tau_l} sum_c conj(S_c) image_{l,c}.
__global__ void k_fh_post(const float2 *A, size_t cells, GridSpec g, NV nv3, size_t N,
                          const float2 *sens, const float2 *eph, float2 *acc, int nl, int nc) {
    const int nv[3] = {nv3.v[0], nv3.v[1], nv3.v[2]};
    for (size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x; r < N;
         r += (size_t)gridDim.x * blockDim.x) {
        int x, y, z;
        vox_xyz(r, nv, g.is3d, x, y, z);
        const GridAt at = grid_at(g, x, y, z);
        float2 a = acc[r];
        for (int l = 0; l < nl; ++l) {
            const float2 *Al = A + (size_t)l * nc * cells + at.idx;
            float2 u = make_float2(0.f, 0.f);
#pragma unroll 4
            for (int c = 0; c < nc; ++c) {
                const float2 w = cmulc(sens[(size_t)c * N + r], Al[(size_t)c * cells]);
                u.x += w.x;
                u.y += w.y;
            }
            const float2 ve = cmulc(eph[(size_t)l * N + r], make_float2(u.x * at.s, u.y * at.s));
            a.x += ve.x;  // eph = exp(-i w tau_l)
            a.y += ve.y;
        }
        acc[r] = a;
    }
}

__global__ void k_eph(float2 *eph, const float *fm, size_t N, int L1, float tau, float t0) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)L1 * N;
         i += (size_t)gridDim.x * blockDim.x) {
        const int l = (int)(i / N);
        const size_t r = i % N;
        const double arg = -(double)(fm ? fm[r] : 0.f) * ((double)tau * l + (double)t0);
        double s, c;
        sincos(arg, &s, &c);
        eph[i] = make_float2((float)c, (float)s);
    }
}

__global__ void k_pack_sens_c(float2 *sens, const float *sr, const float *si, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        sens[i] = sr ? make_float2(sr[i], si ? si[i] : 0.f) : make_float2(1.f, 0.f);
}

// FFT-buffer index of image voxel q in the zero-padded, ifftshifted 2N grid:
// per axis (q + N/2 + N) mod 2N (recon.cu:325-421 and the half-rotation shifts).
__device__ __forceinline__ size_t pad_index(size_t q, const int nv[3], bool is3d) {
    int x, y, z;
    vox_xyz(q, nv, is3d, x, y, z);
    if (!is3d) {
        const int ox = (x + nv[0] / 2 + nv[0]) % (2 * nv[0]);
        const int oy = (y + nv[1] / 2 + nv[1]) % (2 * nv[1]);
        return (size_t)ox * (2 * nv[1]) + oy;
    }
    const int oy = (y + nv[0] / 2 + nv[0]) % (2 * nv[0]);
    const int ox = (x + nv[1] / 2 + nv[1]) % (2 * nv[1]);
    const int oz = (z + nv[2] / 2 + nv[2]) % (2 * nv[2]);
    return ((size_t)oy * (2 * nv[1]) + ox) * (2 * nv[2]) + oz;
}

// pad[c][o(q)] = S_c[q] p[q] exp(-i w tau_l)[q]
__global__ void k_pad(float2 *pad, const float2 *p, const float2 *sens, const float2 *eph_l,
                      NV nv, bool is3d, size_t N, size_t G2, int C, const double *dots) {
    if (dots && scal(const_cast<double *>(dots))->done) return;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < N;
         q += (size_t)gridDim.x * blockDim.x) {
        const size_t o = pad_index(q, nv.v, is3d);
        const float2 pe = cmul(p[q], eph_l[q]);
        for (int c = 0; c < C; ++c) pad[(size_t)c * G2 + o] = cmul(sens[(size_t)c * N + q], pe);
    }
}

__global__ void k_mulq(float2 *big, const float2 *qf, size_t G2, int C, const double *dots) {
    if (dots && scal(const_cast<double *>(dots))->done) return;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)C * G2;
         i += (size_t)gridDim.x * blockDim.x)
        big[i] = cmul(big[i], qf[i % G2]);
}

// acc[q] (+)= conj(exp(-i w tau_l)) sum_c conj(S_c) big[c][o(q)] / G2
__global__ void k_crop_acc(float2 *acc, const float2 *big, const float2 *sens,
                           const float2 *eph_l, NV nv, bool is3d, size_t N, size_t G2, int C,
                           int first, float scale, const double *dots) {
    if (dots && scal(const_cast<double *>(dots))->done) return;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < N;
         q += (size_t)gridDim.x * blockDim.x) {
        const size_t o = pad_index(q, nv.v, is3d);
        float2 s = make_float2(0.f, 0.f);
        for (int c = 0; c < C; ++c) {
            const float2 u = cmulc(sens[(size_t)c * N + q], big[(size_t)c * G2 + o]);
            s.x += u.x;
            s.y += u.y;
        }
        float2 v = cmulc(eph_l[q], s);
        v.x *= scale;
        v.y *= scale;
        if (!first) {
            const float2 a = acc[q];
            v.x += a.x;
            v.y += a.y;
        }
        acc[q] = v;
    }
}

// q += lambda D^H W D p (pen 1) or lambda C^T W C p (pen 2, y = W C p formed
// beforehand); partial Re<p, q>
__global__ void __launch_bounds__(kVB) k_t_tvdot(float2 *__restrict__ q,
                                                 const float2 *__restrict__ p,
                                                 const float *__restrict__ w, int N, Grid3 gd,
                                                 int pen, float lambda, RegView reg,
                                                 double *dots) {
    __shared__ double sh[33];
    if (scal(dots)->done) return;
    double loc = 0.0;
#pragma unroll 4
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < N; r += gridDim.x * blockDim.x) {
        float2 v = q[r];
        if (pen) {
            const float2 t = pen == 2 ? reg_ct_at(reg, r) : dhwd_at(p, w, r, gd);
            v.x += lambda * t.x;
            v.y += lambda * t.y;
            q[r] = v;
        }
        const float2 pv = p[r];
        loc += (double)pv.x * v.x + (double)pv.y * v.y;
    }
    const double b = block_sum(loc, sh);
    if (threadIdx.x == 0) dots[T_PQ * kTBlocks + blockIdx.x] = b;
}

// alpha = beta2 / Re<p,q>; x += alpha p; r -= alpha q; partial |r|^2
__global__ void __launch_bounds__(kVB) k_t_update(float2 *__restrict__ x, float2 *__restrict__ r,
                                                  const float2 *__restrict__ p,
                                                  const float2 *__restrict__ q, int N,
                                                  double *dots) {
    __shared__ double sh[33];
    TScal *S = scal(dots);
    if (S->done) return;
    const double pq = sum_partials(dots + T_PQ * kTBlocks, kTBlocks, sh);
    const float alpha = (float)(S->beta2[S->cur] / pq);
    double loc = 0.0;
#pragma unroll 4
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const float2 pv = p[i], qv = q[i];
        float2 xv = x[i], rv = r[i];
        xv.x += alpha * pv.x;
        xv.y += alpha * pv.y;
        rv.x -= alpha * qv.x;
        rv.y -= alpha * qv.y;
        x[i] = xv;
        r[i] = rv;
        loc += (double)rv.x * rv.x + (double)rv.y * rv.y;
    }
    const double b = block_sum(loc, sh);
    if (threadIdx.x == 0) dots[T_RR * kTBlocks + blockIdx.x] = b;
}

// p = r + (beta2_new / beta2) p; best-residual tracking.  The last block to
// finish (arrival counter) closes the update: best residual, beta2 swap,
// iteration count and the stopping test (recon.cu:2107-2112).  Every block
// has read the scalars it uses before it arrives, so the update of the
// scalars cannot race with those reads.
__global__ void __launch_bounds__(kVB) k_t_dir(float2 *__restrict__ p,
                                               const float2 *__restrict__ r,
                                               const float2 *__restrict__ x,
                                               float2 *__restrict__ best, int N, double *dots) {
    __shared__ double sh[33];
    TScal *S = scal(dots);
    if (S->done) return;
    const double bnew = sum_partials(dots + T_RR * kTBlocks, kTBlocks, sh);
    const int cur = S->cur;
    const double bold = S->beta2[cur];
    const float ratio = (float)(bnew / bold);
    const bool better = bnew < S->res_best;
#pragma unroll 4
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const float2 rv = r[i], pv = p[i];
        p[i] = make_float2(rv.x + ratio * pv.x, rv.y + ratio * pv.y);
        if (better) best[i] = x[i];
    }
    __syncthreads();  // the block's reads of the scalars are done
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&S->arrive, 1u) == gridDim.x - 1) {
            __threadfence();
            S->beta2[cur ^ 1] = bnew;
            if (bnew < S->res_best) S->res_best = bnew;
            S->cur = cur ^ 1;
            S->iters += 1;
            if (sqrt(bnew / S->norm_fhd) < S->tol) S->done = 1;
            S->arrive = 0;
        }
    }
}

__global__ void k_t_setup(double *dots, double tol) {
    TScal *S = scal(dots);
    S->tol = tol;
    S->iters = 0;
    S->arrive = 0;
}

// TV-pass start: r = fhd - q; p = r; partial |r|^2
__global__ void __launch_bounds__(kVB) k_t_init(float2 *r, float2 *p, const float2 *fhd,
                                                const float2 *q, int N, double *dots) {
    __shared__ double sh[33];
    double loc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const float2 f = fhd[i], qv = q[i];
        const float2 rv = make_float2(f.x - qv.x, f.y - qv.y);
        r[i] = rv;
        p[i] = rv;
        loc += (double)rv.x * rv.x + (double)rv.y * rv.y;
    }
    const double b = block_sum(loc, sh);
    if (threadIdx.x == 0) dots[T_RR * kTBlocks + blockIdx.x] = b;
}

__global__ void __launch_bounds__(kVB) k_t_init_finish(double *dots) {
    __shared__ double sh[33];
    const double rr = sum_partials(dots + T_RR * kTBlocks, kTBlocks, sh);
    if (threadIdx.x == 0) {
        TScal *S = scal(dots);
        S->cur = 0;
        S->beta2[0] = rr;
        S->res_best = rr;
        S->done = 0;
    }
}

__global__ void __launch_bounds__(kVB) k_t_norm(const float2 *f, int N, double *dots) {
    __shared__ double sh[33];
    double loc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const float2 v = f[i];
        loc += (double)v.x * v.x + (double)v.y * v.y;
    }
    const double b = block_sum(loc, sh);
    if (threadIdx.x == 0) dots[T_NORM * kTBlocks + blockIdx.x] = b;
}

__global__ void __launch_bounds__(kVB) k_t_norm_finish(double *dots) {
    __shared__ double sh[33];
    const double n = sum_partials(dots + T_NORM * kTBlocks, kTBlocks, sh);
    if (threadIdx.x == 0) scal(dots)->norm_fhd = n;
}

__global__ void k_soa2c(float2 *o, const float *r, const float *i, size_t n) {
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x)
        o[k] = make_float2(r[k], i[k]);
}

__global__ void k_c2soa(float *r, float *i, const float2 *o, size_t n) {
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x) {
        r[k] = o[k].x;
        i[k] = o[k].y;
    }
}

__global__ void k_fillf(float *w, float v, size_t n) {
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x)
        w[k] = v;
}

int gridn(size_t n) {
    return (int)std::min<size_t>(std::max<size_t>((n + kVB - 1) / kVB, 1), 148 * 16);
}

float beatty_beta(float os) {
    const float v = (os - 0.5f) * (os - 0.5f) * (kKW * kKW * 4.0f) / (os * os) - 0.8f;
    return kPiF * std::sqrt(v);
}

}  // namespace

// The output crop the post kernels read after the inverse transform of a
// gridding grid, as half-lengths per FFT axis (grid_image_value: along each
// axis the image's img/2 cells on either side of index 0).
struct Crop {
    int lo[3], hi[3];
};
// negatives: the crop's negatives are read too (index img/2 joins; eight, so
// that the kept runs stay multiples of the transform's column groups).
static Crop crop_of(const GridSpec &g, bool negatives) {
    Crop c{{0, 0, 0}, {0, 0, 0}};
    const int first = g.is3d ? 0 : 1;
    for (int a = first; a < 3; ++a) {
        const int h = g.img[a - first] / 2;
        c.lo[a] = negatives ? h + 8 : h;
        c.hi[a] = h;
    }
    return c;
}

// Blocks of the warp-per-sample gridding: one wave (grid-stride over the samples).
static unsigned grid_blocks() { return 148u * kGridBlocks; }

GridSpec grid_spec(const int img[3], float os, bool beta_after_rounding, float kscale) {
    GridSpec g;
    for (int a = 0; a < 3; ++a) g.img[a] = img[a];
    g.is3d = img[2] > 1;
    const float beta_before = beatty_beta(os);
    float osr;
    if (!g.is3d)
        osr = 2.0f * std::ceil((os * (float)img[0]) / 2.0f) / (float)img[0];
    else
        osr = 4.0f * std::ceil((os * (float)img[2]) / 4.0f) / (float)img[2];
    g.os = osr;
    g.beta = beta_after_rounding ? beatty_beta(osr) : beta_before;
    g.gs[0] = (int)std::ceil(osr * (float)img[0]);
    g.gs[1] = (int)std::ceil(osr * (float)img[1]);
    if (g.gs[0] % 2) g.gs[0] += 1;
    if (g.gs[1] % 2) g.gs[1] += 1;
    g.gs[2] = g.is3d ? (int)std::ceil(osr * (float)img[2]) : 1;
    g.kscale = kscale;
    return g;
}

#define T_TRY(x)                                \
    do {                                        \
        cudaError_t e_ = (x);                   \
        if (e_ != cudaSuccess) return e_;       \
    } while (0)

ToepSolver::~ToepSolver() { release(); }

static void free_plan(GridFft *f) {
    grid_fft_destroy(f);
    *f = GridFft();
}

void ToepSolver::release() {
    release_cg();
    free_plan(&gfq_);
    free_plan(&gff_);
    for (void *b : {(void *)sens_, (void *)eph_, (void *)fm_, (void *)fhd_, (void *)t_,
                    (void *)grid_, (void *)segw_})
        if (b) cudaFree(b);
    segw_ = nullptr;
    sens_ = eph_ = fhd_ = grid_ = nullptr;
    fm_ = t_ = nullptr;
    grid_cells_ = 0;
    ready_ = false;
}

// What F^H F and the CG hold beside the set-up.
void ToepSolver::release_cg() {
    if (g_iter_) cudaGraphExecDestroy(g_iter_);
    g_iter_ = nullptr;
    free_plan(&gf2_);
    free_plan(&gf1_);
    reg_.release();
    void *bufs[] = {qf_, big_, x_,  r_,  p_,  q_,     best_,  w_,
                    dots_, qf2_, b0_, b1_, tw_[0], tw_[1], tw_[2]};
    for (void *b : bufs)
        if (b) cudaFree(b);
    qf_ = big_ = x_ = r_ = p_ = q_ = best_ = nullptr;
    qf2_ = b0_ = b1_ = tw_[0] = tw_[1] = tw_[2] = nullptr;
    w_ = nullptr;
    dots_ = nullptr;
    rows_ = false;
    cg_ready_ = false;
}

cudaError_t ToepSolver::setup(const ToepConfig &cfg, const float *t, const float *fm,
                              const float *sensi_r, const float *sensi_i, unsigned *dev_err,
                              cudaStream_t st) {
    // Same sizes and stream: keep buffers, FFT plans and (same CG terms) the
    // captured iteration graph; only the per-call inputs are refreshed.
    const bool like = st == st_ && cfg.q_only == cfg_.q_only && cfg.nx == cfg_.nx &&
                      cfg.ny == cfg_.ny && cfg.nz == cfg_.nz && cfg.C == cfg_.C &&
                      cfg.M == cfg_.M && (int)cfg.ntime_segs == L_;
    const bool same_shape = ready_ && like;
    ready_ = false;  // until this set-up is complete
    if (!like) lean_ = 0;
    if (same_shape) {
        if (g_iter_ && (cfg.fd != cfg_.fd || cfg.lambda != cfg_.lambda ||
                        cfg.use_graphs != cfg_.use_graphs)) {
            cudaGraphExecDestroy(g_iter_);
            g_iter_ = nullptr;
        }
        cfg_ = cfg;
        err_ = dev_err;
        float tb[2] = {0.f, 0.f};
        T_TRY(cudaMemcpyAsync(&tb[0], t, sizeof(float), cudaMemcpyDeviceToHost, st));
        T_TRY(cudaMemcpyAsync(&tb[1], t + cfg.M - 1, sizeof(float), cudaMemcpyDeviceToHost, st));
        T_TRY(cudaStreamSynchronize(st));
        tau_ = cfg.ntime_segs > 0.f ? (tb[1] - tb[0]) / cfg.ntime_segs : (tb[1] - tb[0]);
        t0_ = tb[0];
        const int L1 = L_ + 1, C = cfg.C;
        T_TRY(cudaMemcpyAsync(t_, t, sizeof(float) * cfg.M, cudaMemcpyDeviceToDevice, st));
        launches_ = 0;
        if (!cfg.q_only) {
            k_pack_sens_c<<<gridn((size_t)C * N_), kVB, 0, st>>>(sens_, sensi_r, sensi_i,
                                                                (size_t)C * N_);
            k_eph<<<gridn((size_t)L1 * N_), kVB, 0, st>>>(eph_, fm, N_, L1, tau_, t0_);
            launches_ = 2;
            T_TRY(cudaGetLastError());
        }
        if (cfg.cg) T_TRY(prepare_cg());
        ready_ = true;
        return cudaSuccess;
    }
    release();
    // a doubled side that no grid transform takes is refused, whatever the call
    for (int d : {cfg.nx, cfg.ny, cfg.nz})
        if (d > 1 && !grid_fft_length_ok(2 * d)) return cudaErrorInvalidValue;
    cfg_ = cfg;
    st_ = st;
    err_ = dev_err;
    L_ = (int)cfg.ntime_segs;
    const bool is3d = cfg.nz > 1;
    N_ = (size_t)cfg.nx * cfg.ny * cfg.nz;
    if (!is3d) {
        nv[0] = cfg.nx;
        nv[1] = cfg.ny;
        nv[2] = 1;
        n2[0] = 2 * cfg.nx;
        n2[1] = 2 * cfg.ny;
        n2[2] = 1;
    } else {
        nv[0] = cfg.ny;
        nv[1] = cfg.nx;
        nv[2] = cfg.nz;
        n2[0] = 2 * cfg.ny;
        n2[1] = 2 * cfg.nx;
        n2[2] = 2 * cfg.nz;
    }
    G2_ = (size_t)n2[0] * n2[1] * n2[2];
    // tau = (t[M-1] - t[0]) / L (toeplitz/computeFH.cmem.cu:1227-1229)
    float tb[2] = {0.f, 0.f};
    T_TRY(cudaMemcpyAsync(&tb[0], t, sizeof(float), cudaMemcpyDeviceToHost, st));
    T_TRY(cudaMemcpyAsync(&tb[1], t + cfg.M - 1, sizeof(float), cudaMemcpyDeviceToHost, st));
    T_TRY(cudaStreamSynchronize(st));
    tau_ = cfg.ntime_segs > 0.f ? (tb[1] - tb[0]) / cfg.ntime_segs : (tb[1] - tb[0]);
    t0_ = tb[0];
    const int L1 = L_ + 1, C = cfg.C;
    T_TRY(cudaMalloc(&t_, sizeof(float) * cfg.M));
    T_TRY(cudaMemcpyAsync(t_, t, sizeof(float) * cfg.M, cudaMemcpyDeviceToDevice, st));
    launches_ = 0;
    if (cfg.q_only) {
        T_TRY(cudaMalloc(&segw_, sizeof(float2) * (L_ / 2 + 1)));
        ready_ = true;
        return cudaSuccess;
    }
    T_TRY(cudaMalloc(&sens_, sizeof(float2) * C * N_));
    T_TRY(cudaMalloc(&eph_, sizeof(float2) * L1 * N_));
    if (cfg.cg) T_TRY(prepare_cg());
    T_TRY(cudaMalloc(&fhd_, sizeof(float2) * N_));
    k_pack_sens_c<<<gridn((size_t)C * N_), kVB, 0, st>>>(sens_, sensi_r, sensi_i, (size_t)C * N_);
    k_eph<<<gridn((size_t)L1 * N_), kVB, 0, st>>>(eph_, fm, N_, L1, tau_, t0_);
    T_TRY(cudaGetLastError());
    launches_ = 2;
    ready_ = true;
    return cudaSuccess;
}

// Buffers and plans of F^H F and the CG, and the -reg matrix of cfg_; kept from the first
// call that needs them on (F^H d does not: 64x64 x 4 coils, first call 0.93 -> 0.53 ms).
cudaError_t ToepSolver::prepare_cg() {
    if (!cg_ready_) T_TRY(build_cg());
    cg_ready_ = true;
    return set_reg();
}

// After a call that ran out of memory: gives back what it can, so that the same call needs
// less.  1: gridding grids one at a time, F^H F with one transform and one Qf_l at a time;
// 2: F^H F on the zero-padded chain, whose transforms are no longer than the doubled image.
bool ToepSolver::shrink() {
    if (lean_ >= (cfg_.q_only ? 1 : 2)) return false;
    ++lean_;
    release_cg();
    if (grid_) cudaFree(grid_);
    grid_ = nullptr;
    grid_cells_ = 0;
    return true;
}

cudaError_t ToepSolver::build_cg() {
    release_cg();
    const bool is3d = cfg_.nz > 1;
    const int L1 = L_ + 1, C = cfg_.C;
    // Sides up to the engine's longest length run on the pruned mixed-radix
    // engine; others (and IMP_TOEP_PADDED=1) use the zero-padded chain on the
    // grid transform.
    const char *force_padded = std::getenv("IMP_TOEP_PADDED");
    const bool pruned = lean_ < 2 && !(force_padded && force_padded[0] == '1');
    rows_ = pruned && toep_rows_plan(nv[0], is3d ? nv[1] : 1, is3d ? nv[2] : nv[1], C, L1, &rp_);
    if (rows_) {
        if (lean_) rp_.chunk = 1;
        qf_segs_ = lean_ ? 1 : (int)std::min<size_t>(
            L1, std::max<size_t>(1, ((size_t)128 << 20) / (sizeof(float2) * rp_.q_elems())));
        T_TRY(cudaMalloc(&qf_, sizeof(float2) * rp_.q_elems() * qf_segs_));
        T_TRY(cudaMalloc(&qf2_, sizeof(float2) * rp_.q_elems() * L1));
        if (rp_.b0_elems()) T_TRY(cudaMalloc(&b0_, sizeof(float2) * rp_.b0_elems()));
        T_TRY(cudaMalloc(&b1_, sizeof(float2) * rp_.b1_elems()));
        T_TRY(toep_rows_twiddles(rp_, tw_));
    } else {
        T_TRY(cudaMalloc(&qf_, sizeof(float2) * L1 * G2_));
        T_TRY(cudaMalloc(&big_, sizeof(float2) * C * G2_));
    }
    for (float2 **b : {&x_, &r_, &p_, &q_, &best_}) T_TRY(cudaMalloc(b, sizeof(float2) * N_));
    T_TRY(cudaMalloc(&w_, sizeof(float) * N_));
    T_TRY(cudaMalloc(&dots_, sizeof(double) * (T_SCAL * kTBlocks + 8)));
    T_TRY(cudaMemsetAsync(dots_, 0, sizeof(double) * (T_SCAL * kTBlocks + 8), st_));
    // the 2N grid: batched over the coils for the zero-padded chain, single
    // for Qf_l (2-D grids are [n2[0]][n2[1]], 3-D [n2[0]][n2[1]][n2[2]])
    int d0 = is3d ? n2[0] : 1, d1 = is3d ? n2[1] : n2[0], d2 = is3d ? n2[2] : n2[1];
    if (rows_) {  // the engine's lengths
        d0 = is3d ? 2 * rp_.es : 1;
        d1 = is3d ? 2 * rp_.em : 2 * rp_.es;
        d2 = 2 * rp_.ef;
    } else {
        T_TRY(grid_fft_create(&gf2_, d0, d1, d2, C));
    }
    T_TRY(grid_fft_create(&gf1_, d0, d1, d2, 1));
    return cudaSuccess;
}

// Plan of one grid and room for `batch` of them.
cudaError_t ToepSolver::ensure_grid_plan(const GridSpec &g, GridFft *plan, int batch) {
    const int d0 = g.is3d ? g.gs[0] : 1, d1 = g.is3d ? g.gs[1] : g.gs[0];
    const int d2 = g.is3d ? g.gs[2] : g.gs[1];
    const bool planned = plan->tw[0] || plan->tw[1] || plan->tw[2];
    if (!planned || plan->n[0] != d0 || plan->n[1] != d1 || plan->n[2] != d2)
        T_TRY(grid_fft_create(plan, d0, d1, d2, 1));
    const size_t need = g.cells() * batch;
    if (need > grid_cells_) {
        if (grid_) cudaFree(grid_);
        grid_ = nullptr;
        grid_cells_ = 0;
        T_TRY(cudaMalloc(&grid_, sizeof(float2) * need));
        grid_cells_ = need;
    }
    return cudaSuccess;
}

// Gridding grids per batch: as many as half of the L2 holds (the scatter's
// atomics, the transform and the crop then stay in L2), at least one.
static size_t grid_batch(const GridSpec &g, bool lean) {
    return lean ? 1 : std::max<size_t>(1, ((size_t)64 << 20) / (sizeof(float2) * g.cells()));
}

cudaError_t ToepSolver::compute_q(const float *kx, const float *ky, const float *kz,
                                  float *q_out_r, float *q_out_i) {
    const bool is3d = cfg_.nz > 1;
    const int img[3] = {2 * cfg_.nx, 2 * cfg_.ny, is3d ? 2 * cfg_.nz : 1};
    const GridSpec g = grid_spec(img, cfg_.os_q, true, 2.0f);
    // two segments per grid
    const int nb = (int)std::min<size_t>(grid_batch(g, lean_ > 0), L_ / 2 + 1);
    T_TRY(ensure_grid_plan(g, &gfq_, nb));
    const NV n2d{{n2[0], n2[1], n2[2]}};
    const Crop crop = crop_of(g, true);
    T_TRY(cudaMemsetAsync(segw_, 0, sizeof(float2) * (L_ / 2 + 1), st_));
    k_seg_weights<<<std::min((cfg_.M + kVB - 1) / kVB, 148 * 6), kVB, 0, st_>>>(
        reinterpret_cast<float *>(segw_), t_, cfg_.M, tau_, t0_, L_ + 1);
    T_TRY(cudaGetLastError());
    ++launches_;
    for (int l = 0; l <= L_; l += 2 * nb) {
        const int nl = std::min(2 * nb, L_ + 1 - l), ng = (nl + 1) / 2;
        T_TRY(cudaMemsetAsync(grid_, 0, sizeof(float2) * g.cells() * ng, st_));
        auto scatter = g.is3d ? k_grid_w<true, true> : k_grid_w<true, false>;
        scatter<<<grid_blocks(), kGridWarps * 32, 0, st_>>>(
            grid_, g.cells(), kx, ky, kz, t_, nullptr, nullptr, cfg_.M, g, tau_, t0_, l, nl, 1,
            L_ + 1, segw_);
        T_TRY(cudaGetLastError());
        T_TRY(grid_fft_exec_cropped(gfq_, grid_, true, crop.lo, crop.hi, st_, ng));
        k_q_post<<<gridn(G2_), kVB, 0, st_>>>(grid_, g.cells(), g, n2d, q_out_r + (size_t)l * G2_,
                                             q_out_i + (size_t)l * G2_, G2_, nl,
                                             segw_ + l / 2);
        T_TRY(cudaGetLastError());
        launches_ += 2 + gfq_.passes();
    }
    return cudaStreamSynchronize(st_);
}

cudaError_t ToepSolver::load_q(const float *q_r, const float *q_i) {
    if (rows_) {
        for (int l = 0; l <= L_; l += qf_segs_) {
            const int nl = std::min(qf_segs_, L_ + 1 - l);
            T_TRY(toep_rows_embed(rp_, qf_, q_r + (size_t)l * G2_, q_i + (size_t)l * G2_, nl, st_));
            T_TRY(grid_fft_exec_cropped(gf1_, qf_, false, nullptr, nullptr, st_, nl));
            T_TRY(toep_rows_qf(rp_, qf2_ + (size_t)l * rp_.q_elems(), qf_,
                               1.0f / (float)rp_.q_elems(), nl, st_));
            launches_ += 2 + gf1_.passes();
        }
        return cudaStreamSynchronize(st_);
    }
    const NV n2d{{n2[0], n2[1], n2[2]}};
    for (int l = 0; l <= L_; ++l) {
        float2 *qf_l = qf_ + (size_t)l * G2_;
        k_q_shift<<<gridn(G2_), kVB, 0, st_>>>(q_r + (size_t)l * G2_, q_i + (size_t)l * G2_, n2d,
                                              cfg_.nz > 1, qf_l, G2_);
        T_TRY(cudaGetLastError());
        T_TRY(grid_fft_exec(gf1_, qf_l, false, st_));
        launches_ += 1 + gf1_.passes();
    }
    return cudaStreamSynchronize(st_);
}

cudaError_t ToepSolver::compute_fhd(const float *kx, const float *ky, const float *kz,
                                    const float *kd_r, const float *kd_i, float *fhd_r,
                                    float *fhd_i) {
    const int img[3] = {cfg_.nx, cfg_.ny, cfg_.nz};
    const GridSpec g = grid_spec(img, cfg_.os_fh, false, 1.0f);
    // batches of coils x segments: the coils of a launch share each sample's weights
    const size_t room = grid_batch(g, lean_ > 0);
    const int nc_b = (int)std::min<size_t>(room, std::min(cfg_.C, kGridCoils));
    const int nl_b = (int)std::min<size_t>(std::max<size_t>(room / nc_b, 1), L_ + 1);
    T_TRY(ensure_grid_plan(g, &gff_, nc_b * nl_b));
    const NV nvd{{nv[0], nv[1], nv[2]}};
    const Crop crop = crop_of(g, false);
    T_TRY(cudaMemsetAsync(fhd_, 0, sizeof(float2) * N_, st_));
    for (int c = 0; c < cfg_.C; c += nc_b)
        for (int l = 0; l <= L_; l += nl_b) {
            const int nc = std::min(nc_b, cfg_.C - c), nl = std::min(nl_b, L_ + 1 - l);
            T_TRY(cudaMemsetAsync(grid_, 0, sizeof(float2) * g.cells() * nc * nl, st_));
            auto scatter = nc == 1 ? (g.is3d ? k_grid_w<true, true> : k_grid_w<true, false>)
                                   : (g.is3d ? k_grid_w<false, true> : k_grid_w<false, false>);
            scatter<<<grid_blocks(), kGridWarps * 32, 0, st_>>>(
                grid_, g.cells(), kx, ky, kz, t_, kd_r + (size_t)c * cfg_.M,
                kd_i + (size_t)c * cfg_.M, cfg_.M, g, tau_, t0_, l, nl, nc, L_ + 1, nullptr);
            T_TRY(cudaGetLastError());
            T_TRY(grid_fft_exec_cropped(gff_, grid_, true, crop.lo, crop.hi, st_, nc * nl));
            k_fh_post<<<gridn(N_), kVB, 0, st_>>>(grid_, g.cells(), g, nvd, N_,
                                                 sens_ + (size_t)c * N_, eph_ + (size_t)l * N_,
                                                 fhd_, nl, nc);
            T_TRY(cudaGetLastError());
            launches_ += 2 + gff_.passes();
        }
    if (fhd_r) {
        k_c2soa<<<gridn(N_), kVB, 0, st_>>>(fhd_r, fhd_i, fhd_, N_);
        T_TRY(cudaGetLastError());
        ++launches_;
    }
    return cudaStreamSynchronize(st_);
}

// q = A^H A p over all segments and coils (no TV term)
cudaError_t ToepSolver::apply_aha(const float2 *p, float2 *q) {
    const bool is3d = cfg_.nz > 1;
    NV nvv{{nv[0], nv[1], nv[2]}};
    const int C = cfg_.C;
    const float scale = 1.0f / (float)G2_;
    const double *dots = dots_;
    if (rows_)
        return toep_rows_apply(rp_, q, p, sens_, eph_, b0_, b1_, qf2_, done_flag(), tw_, st_);
    for (int l = 0; l <= L_; ++l) {
        const float2 *eph_l = eph_ + (size_t)l * N_;
        T_TRY(cudaMemsetAsync(big_, 0, sizeof(float2) * C * G2_, st_));
        k_pad<<<gridn(N_), kVB, 0, st_>>>(big_, p, sens_, eph_l, nvv, is3d, N_, G2_, C, dots);
        T_TRY(cudaGetLastError());
        T_TRY(grid_fft_exec(gf2_, big_, false, st_));
        k_mulq<<<gridn((size_t)C * G2_), kVB, 0, st_>>>(big_, qf_ + (size_t)l * G2_, G2_, C, dots);
        T_TRY(cudaGetLastError());
        T_TRY(grid_fft_exec(gf2_, big_, true, st_));
        k_crop_acc<<<gridn(N_), kVB, 0, st_>>>(q, big_, sens_, eph_l, nvv, is3d, N_, G2_, C,
                                              l == 0 ? 1 : 0, scale, dots);
        T_TRY(cudaGetLastError());
    }
    return cudaSuccess;
}

const int *ToepSolver::done_flag() const {
    return reinterpret_cast<const int *>(
        reinterpret_cast<const char *>(dots_ + T_SCAL * kTBlocks) + offsetof(TScal, done));
}

// -reg takes precedence over -fd (toeplitz/recon.cu:1543-1680)
cudaError_t ToepSolver::penalty_dot(float2 *q, const float2 *p) {
    const Grid3 gd{nv[0], nv[1], nv[2]};
    const int pen = reg_.on() ? 2 : cfg_.fd ? 1 : 0;
    if (pen == 2) {
        T_TRY(reg_.apply_cw(p, w_, done_flag(), st_));
        ++launches_;
    }
    k_t_tvdot<<<kTBlocks, kVB, 0, st_>>>(q, p, w_, (int)N_, gd, pen, cfg_.lambda, reg_.view(),
                                        dots_);
    return cudaGetLastError();
}

cudaError_t ToepSolver::set_reg() {
    if (!cfg_.reg) {
        if (reg_.on()) {
            reg_.release();
            if (g_iter_) cudaGraphExecDestroy(g_iter_);
            g_iter_ = nullptr;
        }
        return cudaSuccess;
    }
    const bool was_on = reg_.on();
    bool moved = false;
    T_TRY(reg_.set(*cfg_.reg, (int)N_, st_, &moved));
    if ((moved || !was_on) && g_iter_) {
        cudaGraphExecDestroy(g_iter_);
        g_iter_ = nullptr;
    }
    return cudaSuccess;
}

cudaError_t ToepSolver::cg_iteration() {
    const Grid3 gd{nv[0], nv[1], nv[2]};
    T_TRY(apply_aha(p_, q_));
    T_TRY(penalty_dot(q_, p_));
    k_t_update<<<kTBlocks, kVB, 0, st_>>>(x_, r_, p_, q_, (int)N_, dots_);
    k_t_dir<<<kTBlocks, kVB, 0, st_>>>(p_, r_, x_, best_, (int)N_, dots_);
    return cudaGetLastError();
}

static cudaError_t capture_graph(cudaStream_t st, cudaGraphExec_t *exec,
                                 cudaError_t (ToepSolver::*fn)(), ToepSolver *self) {
    T_TRY(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    cudaError_t body = (self->*fn)();
    cudaGraph_t graph = nullptr;
    cudaError_t end = cudaStreamEndCapture(st, &graph);
    if (body != cudaSuccess) {
        if (graph) cudaGraphDestroy(graph);
        return body;
    }
    if (end != cudaSuccess) return end;
    cudaError_t inst = cudaGraphInstantiate(exec, graph, 0);
    cudaGraphDestroy(graph);
    return inst;
}

cudaError_t ToepSolver::solve(const float *fhd_r, const float *fhd_i, float *x_r, float *x_i) {
    const Grid3 gd{nv[0], nv[1], nv[2]};
    const int N = (int)N_;
    if (fhd_r) {
        k_soa2c<<<gridn(N_), kVB, 0, st_>>>(fhd_, fhd_r, fhd_i, N_);
        T_TRY(cudaGetLastError());
    }
    T_TRY(cudaMemsetAsync(x_, 0, sizeof(float2) * N_, st_));
    T_TRY(cudaMemsetAsync(best_, 0, sizeof(float2) * N_, st_));
    k_fillf<<<gridn(N_), kVB, 0, st_>>>(w_, 1.f, N_);
    k_t_norm<<<kTBlocks, kVB, 0, st_>>>(fhd_, N, dots_);
    k_t_norm_finish<<<1, kVB, 0, st_>>>(dots_);
    k_t_setup<<<1, 1, 0, st_>>>(dots_, 1.0e-16);  // recon.cu:2112
    T_TRY(cudaGetLastError());
    launches_ += 5;
    const int iter_launches = aha_launches() + 3 + (reg_.on() ? 1 : 0);  // one CG iteration
    if (cfg_.use_graphs && !g_iter_) T_TRY(capture_graph(st_, &g_iter_, &ToepSolver::cg_iteration, this));
    for (int tv_i = 0; tv_i < std::max(cfg_.tv ? cfg_.tv_num : 1, 1); ++tv_i) {
        if (tv_i != 0) {
            T_TRY(tv_weight(w_, x_, N, gd, cfg_.tv_eps, st_));
            ++launches_;
        }
        // r = F^H d - A x; p = r; beta2 = resBest = |r|^2   (recon.cu:2036-2057)
        T_TRY(cudaMemsetAsync(reinterpret_cast<char *>(dots_ + T_SCAL * kTBlocks) +
                                  offsetof(TScal, done),
                              0, sizeof(int), st_));
        T_TRY(apply_aha(x_, q_));
        T_TRY(penalty_dot(q_, x_));
        k_t_init<<<kTBlocks, kVB, 0, st_>>>(r_, p_, fhd_, q_, N, dots_);
        k_t_init_finish<<<1, kVB, 0, st_>>>(dots_);
        T_TRY(cudaGetLastError());
        launches_ += aha_launches() + 3;
        for (int it = 0; it < cfg_.cg_num; ++it) {
            if (g_iter_)
                T_TRY(cudaGraphLaunch(g_iter_, st_));
            else
                T_TRY(cg_iteration());
            launches_ += iter_launches;
        }
        if (!cfg_.tv) break;
    }
    k_c2soa<<<gridn(N_), kVB, 0, st_>>>(x_r, x_i, best_, N_);
    T_TRY(cudaGetLastError());
    ++launches_;
    return cudaSuccess;
}

cudaError_t ToepSolver::solve_from(const float *fhd_r, const float *fhd_i, float *x_r,
                                   float *x_i, double tol, int max_iter, int *iters) {
    const Grid3 gd{nv[0], nv[1], nv[2]};
    const int N = (int)N_;
    if (fhd_r) k_soa2c<<<gridn(N_), kVB, 0, st_>>>(fhd_, fhd_r, fhd_i, N_);
    k_soa2c<<<gridn(N_), kVB, 0, st_>>>(x_, x_r, x_i, N_);
    T_TRY(cudaMemcpyAsync(best_, x_, sizeof(float2) * N_, cudaMemcpyDeviceToDevice, st_));
    k_fillf<<<gridn(N_), kVB, 0, st_>>>(w_, 1.f, N_);
    k_t_norm<<<kTBlocks, kVB, 0, st_>>>(fhd_, N, dots_);
    k_t_norm_finish<<<1, kVB, 0, st_>>>(dots_);
    k_t_setup<<<1, 1, 0, st_>>>(dots_, tol);
    T_TRY(cudaGetLastError());
    launches_ += 6;
    if (cfg_.use_graphs && !g_iter_) T_TRY(capture_graph(st_, &g_iter_, &ToepSolver::cg_iteration, this));
    // The kernels return at once while `done` is set (a previous solve may have
    // stopped on its tolerance): clear it before the first A^H A.
    T_TRY(cudaMemsetAsync(reinterpret_cast<char *>(dots_ + T_SCAL * kTBlocks) +
                              offsetof(TScal, done),
                          0, sizeof(int), st_));
    // r = F^H d - A x0; p = r
    T_TRY(apply_aha(x_, q_));
    T_TRY(penalty_dot(q_, x_));
    k_t_init<<<kTBlocks, kVB, 0, st_>>>(r_, p_, fhd_, q_, N, dots_);
    k_t_init_finish<<<1, kVB, 0, st_>>>(dots_);
    T_TRY(cudaGetLastError());
    launches_ += aha_launches() + 3;
    const int iter_launches = aha_launches() + 3 + (reg_.on() ? 1 : 0);
    const TScal *S = reinterpret_cast<const TScal *>(dots_ + T_SCAL * kTBlocks);
    int it = 0;
    while (it < max_iter) {
        const int chunk = std::min(4, max_iter - it);
        for (int k = 0; k < chunk; ++k) {
            if (g_iter_)
                T_TRY(cudaGraphLaunch(g_iter_, st_));
            else
                T_TRY(cg_iteration());
            launches_ += iter_launches;
        }
        it += chunk;
        int done = 0;
        T_TRY(cudaMemcpyAsync(&done, &S->done, sizeof(int), cudaMemcpyDeviceToHost, st_));
        T_TRY(cudaStreamSynchronize(st_));
        if (done) break;
    }
    if (iters) {
        T_TRY(cudaMemcpyAsync(iters, &S->iters, sizeof(int), cudaMemcpyDeviceToHost, st_));
        T_TRY(cudaStreamSynchronize(st_));
    }
    k_c2soa<<<gridn(N_), kVB, 0, st_>>>(x_r, x_i, best_, N_);
    ++launches_;
    return cudaGetLastError();
}

cudaError_t ToepSolver::apply(const float *p_r, const float *p_i, float *q_r, float *q_i) {
    k_soa2c<<<gridn(N_), kVB, 0, st_>>>(p_, p_r, p_i, N_);
    T_TRY(cudaMemsetAsync(dots_ + T_SCAL * kTBlocks, 0, sizeof(TScal), st_));
    T_TRY(apply_aha(p_, q_));
    if (cfg_.fd || reg_.on()) {
        k_fillf<<<gridn(N_), kVB, 0, st_>>>(w_, 1.f, N_);
        T_TRY(penalty_dot(q_, p_));
    }
    k_c2soa<<<gridn(N_), kVB, 0, st_>>>(q_r, q_i, q_, N_);
    return cudaGetLastError();
}

}  // namespace imp

// ============================================================================
// C-ABI of the Toeplitz path
// ============================================================================
#include "context.h"
#include "nudft.cuh"

using imp::DevKeep;
using imp::fail;
using imp::in_less_memory;

namespace {

imp_status toep_args(const imp_toeplitz_options *o, int nx, int ny, int nz, int num_k) {
    if (!o) return fail(IMP_ERR_INVALID_ARG, "null options");
    if (nx <= 0 || ny <= 0 || nz <= 0 || num_k <= 0)
        return fail(IMP_ERR_INVALID_ARG, "nx, ny, nz and num_k must be > 0");
    if (nx % 2 || ny % 2 || (nz > 1 && nz % 2))
        return fail(IMP_ERR_INVALID_ARG, "image sizes must be even (half-rotation shifts)");
    if (o->ntime_segs < 0.f) return fail(IMP_ERR_INVALID_ARG, "ntime_segs must be >= 0");
    if (o->gridOS_Q < 1.f || o->gridOS_Q > 2.f || o->gridOS_FH < 1.f || o->gridOS_FH > 2.f)
        return fail(IMP_ERR_INVALID_ARG, "gridding oversampling factor should be in [1.0,2.0]");
    if (o->cg_num <= 0) return fail(IMP_ERR_INVALID_ARG, "cg_num must be > 0");
    if (o->reg) {
        const char *why = imp::sparse_reg_check(*o->reg, nx * ny * nz);
        if (why[0]) return fail(IMP_ERR_INVALID_ARG, std::string("-reg matrix: ") + why);
    }
    return IMP_OK;
}

imp::ToepConfig toep_cfg(const imp_toeplitz_options *o, int nx, int ny, int nz, int C, int M) {
    imp::ToepConfig c;
    c.nx = nx;
    c.ny = ny;
    c.nz = nz;
    c.C = C;
    c.M = M;
    c.ntime_segs = o->ntime_segs;
    c.os_q = o->gridOS_Q;
    c.os_fh = o->gridOS_FH;
    c.cg_num = o->cg_num;
    c.fd = o->enable_fd != 0;
    c.lambda = o->fd_penalizer;
    c.tv = o->enable_tv != 0;
    c.tv_num = o->enable_tv ? o->tv_num : 1;
    c.tv_eps = o->tv_eps;
    c.reg = o->reg;
    return c;
}

// The same configuration without the CG's penalty terms (Q and F^H d).
imp::ToepConfig toep_cfg_nopen(const imp_toeplitz_options *o, int nx, int ny, int nz, int C,
                               int M) {
    imp::ToepConfig c = toep_cfg(o, nx, ny, nz, C, M);
    c.reg = nullptr;
    return c;
}

imp::ToepSolver &solver_of(imp_context *ctx) {
    if (!ctx->tp) ctx->tp.reset(new imp::ToepSolver());
    return *ctx->tp;
}

// Q is coil-free: it gets its own solver, so that alternating Q and
// F^H d / CG calls (one coil versus num_coil) keep both set up instead of
// rebuilding buffers and FFT plans on every call.
imp::ToepSolver &solver_q_of(imp_context *ctx) {
    if (!ctx->tp_q) ctx->tp_q.reset(new imp::ToepSolver());
    return *ctx->tp_q;
}

imp_status copy_out(imp_context *ctx, float *dst, const float *src, size_t n) {
    IMP_CUDA(cudaMemcpyAsync(dst, src, n * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream),
             "output D2H");
    return IMP_OK;
}

}  // namespace

extern "C" {

void imp_toeplitz_options_default(imp_toeplitz_options *o) {
    if (!o) return;
    std::memset(o, 0, sizeof(*o));
    o->cg_num = 8;
    o->tv_num = 10;
    o->tv_eps = 1e-6f;
    o->ntime_segs = 12.f;
    o->gridOS_Q = 1.125f;
    o->gridOS_FH = 1.5f;
}

imp_status imp_toeplitz_q(imp_context *ctx, const imp_toeplitz_options *opt, float *q_r,
                          float *q_i, const float *kx, const float *ky, const float *kz,
                          const float *t, int num_k, int nx, int ny, int nz) {
    imp_status s = toep_args(opt, nx, ny, nz, num_k);
    if (s != IMP_OK) return s;
    if (!q_r || !q_i || !kx || !ky || !t || (nz > 1 && !kz))
        return fail(IMP_ERR_INVALID_ARG, "null array argument");
    return in_less_memory(ctx, [&]() -> imp_status {
        if ((s = imp::begin(ctx)) != IMP_OK) return s;
        imp::stage_reset(ctx);
        DevKeep keep;
        const float *dkx, *dky, *dkz = nullptr, *dt;
        if ((s = imp::to_device_staged(ctx, kx, num_k, &dkx, nullptr)) ||
            (s = imp::to_device_staged(ctx, ky, num_k, &dky, nullptr)) ||
            (s = imp::to_device_staged(ctx, kz, nz > 1 ? num_k : 0, &dkz, nullptr)) ||
            (s = imp::to_device_staged(ctx, t, num_k, &dt, nullptr)))
            return s;
        imp::ToepSolver &ts = solver_q_of(ctx);
        imp::ToepConfig qcfg = toep_cfg_nopen(opt, nx, ny, nz, 1, num_k);
        qcfg.q_only = true;
        IMP_CUDA(ts.setup(qcfg, dt, nullptr, nullptr, nullptr, ctx->dev_err, ctx->stream),
                 "toeplitz setup");
        const size_t nq = (size_t)ts.segments() * ts.q_elems();
        float *dqr, *dqi;
        bool hr, hi;
        if ((s = imp::out_device_staged(ctx, q_r, nq, &dqr, &hr)) ||
            (s = imp::out_device_staged(ctx, q_i, nq, &dqi, &hi)))
            return s;
        IMP_CUDA(ts.compute_q(dkx, dky, dkz, dqr, dqi), "Q gridding");
        if (hr && (s = copy_out(ctx, q_r, dqr, nq))) return s;
        if (hi && (s = copy_out(ctx, q_i, dqi, nq))) return s;
        s = imp::finish(ctx);
        ctx->launches = ts.launches();
        return s;
    });
}

imp_status imp_toeplitz_fhd(imp_context *ctx, const imp_toeplitz_options *opt, float *fhd_r,
                            float *fhd_i, const float *kdata_r, const float *kdata_i,
                            const float *kx, const float *ky, const float *kz, const float *t,
                            const float *fm, const float *sensi_r, const float *sensi_i,
                            int num_k, int num_coil, int nx, int ny, int nz) {
    imp_status s = toep_args(opt, nx, ny, nz, num_k);
    if (s != IMP_OK) return s;
    if (!fhd_r || !fhd_i || !kdata_r || !kdata_i || !kx || !ky || !t || (nz > 1 && !kz))
        return fail(IMP_ERR_INVALID_ARG, "null array argument");
    if (num_coil <= 0 || (num_coil > 1 && (!sensi_r || !sensi_i)))
        return fail(IMP_ERR_INVALID_ARG, "num_coil > 0 and sensi for num_coil > 1");
    return in_less_memory(ctx, [&]() -> imp_status {
        if ((s = imp::begin(ctx)) != IMP_OK) return s;
        imp::stage_reset(ctx);
        const size_t N = (size_t)nx * ny * nz, M = num_k, C = num_coil;
        DevKeep keep;
        const float *dkx, *dky, *dkz = nullptr, *dt, *dfm = nullptr, *dsr = nullptr;
        const float *dsi = nullptr, *dkr, *dki;
        if ((s = imp::to_device_staged(ctx, kx, M, &dkx, nullptr)) ||
            (s = imp::to_device_staged(ctx, ky, M, &dky, nullptr)) ||
            (s = imp::to_device_staged(ctx, kz, nz > 1 ? M : 0, &dkz, nullptr)) ||
            (s = imp::to_device_staged(ctx, t, M, &dt, nullptr)) ||
            (s = imp::to_device_staged(ctx, fm, N, &dfm, nullptr)) ||
            (s = imp::to_device_staged(ctx, C > 1 ? sensi_r : nullptr, C * N, &dsr, nullptr)) ||
            (s = imp::to_device_staged(ctx, C > 1 ? sensi_i : nullptr, C * N, &dsi, nullptr)) ||
            (s = imp::to_device_staged(ctx, kdata_r, C * M, &dkr, nullptr)) ||
            (s = imp::to_device_staged(ctx, kdata_i, C * M, &dki, nullptr)))
            return s;
        imp::ToepSolver &ts = solver_of(ctx);
        IMP_CUDA(ts.setup(toep_cfg_nopen(opt, nx, ny, nz, num_coil, num_k), dt, dfm, dsr, dsi,
                          ctx->dev_err, ctx->stream),
                 "toeplitz setup");
        float *dfr, *dfi;
        bool hr, hi;
        if ((s = imp::out_device_staged(ctx, fhd_r, N, &dfr, &hr)) ||
            (s = imp::out_device_staged(ctx, fhd_i, N, &dfi, &hi)))
            return s;
        IMP_CUDA(ts.compute_fhd(dkx, dky, dkz, dkr, dki, dfr, dfi), "F^H d gridding");
        if (hr && (s = copy_out(ctx, fhd_r, dfr, N))) return s;
        if (hi && (s = copy_out(ctx, fhd_i, dfi, N))) return s;
        s = imp::finish(ctx);
        ctx->launches = ts.launches();
        return s;
    });
}

static imp_status toeplitz_common(imp_context *ctx, const imp_toeplitz_options *opt,
                                  const float *q_r, const float *q_i, const float *t, int num_k,
                                  const float *fm, const float *sensi_r, const float *sensi_i,
                                  int num_coil, int nx, int ny, int nz, DevKeep &keep,
                                  imp::ToepSolver **out) {
    imp_status s = toep_args(opt, nx, ny, nz, num_k);
    if (s != IMP_OK) return s;
    if (!q_r || !q_i || !t) return fail(IMP_ERR_INVALID_ARG, "null array argument");
    if (num_coil <= 0 || (num_coil > 1 && (!sensi_r || !sensi_i)))
        return fail(IMP_ERR_INVALID_ARG, "num_coil > 0 and sensi for num_coil > 1");
    if ((s = imp::begin(ctx)) != IMP_OK) return s;
    imp::stage_reset(ctx);
    const size_t N = (size_t)nx * ny * nz, C = num_coil;
    const float *dt, *dfm = nullptr, *dsr = nullptr, *dsi = nullptr, *dqr, *dqi;
    if ((s = imp::to_device_staged(ctx, t, num_k, &dt, nullptr)) ||
        (s = imp::to_device_staged(ctx, fm, N, &dfm, nullptr)) ||
        (s = imp::to_device_staged(ctx, num_coil > 1 ? sensi_r : nullptr, C * N, &dsr, nullptr)) ||
        (s = imp::to_device_staged(ctx, num_coil > 1 ? sensi_i : nullptr, C * N, &dsi, nullptr)))
        return s;
    imp::ToepSolver &ts = solver_of(ctx);
    imp::ToepConfig cfg = toep_cfg(opt, nx, ny, nz, num_coil, num_k);
    cfg.cg = true;
    IMP_CUDA(ts.setup(cfg, dt, dfm, dsr, dsi, ctx->dev_err, ctx->stream),
             "toeplitz setup");
    const size_t nq = (size_t)ts.segments() * ts.q_elems();
    if ((s = imp::to_device_staged(ctx, q_r, nq, &dqr, nullptr)) ||
        (s = imp::to_device_staged(ctx, q_i, nq, &dqi, nullptr)))
        return s;
    IMP_CUDA(ts.load_q(dqr, dqi), "Qf");
    *out = &ts;
    return IMP_OK;
}

imp_status imp_toeplitz_recon(imp_context *ctx, const imp_toeplitz_options *opt, float *x_r,
                              float *x_i, const float *fhd_r, const float *fhd_i,
                              const float *q_r, const float *q_i, const float *t, int num_k,
                              const float *fm, const float *sensi_r, const float *sensi_i,
                              int num_coil, int nx, int ny, int nz) {
    if (!x_r || !x_i || !fhd_r || !fhd_i) return fail(IMP_ERR_INVALID_ARG, "null array argument");
    return in_less_memory(ctx, [&]() -> imp_status {
        DevKeep keep;
        imp::ToepSolver *ts = nullptr;
        imp_status s = toeplitz_common(ctx, opt, q_r, q_i, t, num_k, fm, sensi_r, sensi_i, num_coil,
                                       nx, ny, nz, keep, &ts);
        if (s != IMP_OK) return s;
        const size_t N = (size_t)nx * ny * nz;
        const float *dfr, *dfi;
        float *dxr, *dxi;
        bool hr, hi;
        if ((s = imp::to_device_staged(ctx, fhd_r, N, &dfr, nullptr)) ||
            (s = imp::to_device_staged(ctx, fhd_i, N, &dfi, nullptr)) ||
            (s = imp::out_device_staged(ctx, x_r, N, &dxr, &hr)) ||
            (s = imp::out_device_staged(ctx, x_i, N, &dxi, &hi)))
            return s;
        IMP_CUDA(ts->solve(dfr, dfi, dxr, dxi), "toeplitz CG");
        if (hr && (s = copy_out(ctx, x_r, dxr, N))) return s;
        if (hi && (s = copy_out(ctx, x_i, dxi, N))) return s;
        s = imp::finish(ctx);
        ctx->launches = ts->launches();
        return s;
    });
}

imp_status imp_toeplitz_cg(imp_context *ctx, const imp_toeplitz_options *opt, float *x_r,
                           float *x_i, const float *fhd_r, const float *fhd_i, const float *q_r,
                           const float *q_i, const float *t, int num_k, const float *fm,
                           const float *sensi_r, const float *sensi_i, int num_coil, int nx,
                           int ny, int nz, double tol, int max_iter, int *iterations) {
    if (!x_r || !x_i || !fhd_r || !fhd_i) return fail(IMP_ERR_INVALID_ARG, "null array argument");
    if (max_iter < 0 || !(tol >= 0.0)) return fail(IMP_ERR_INVALID_ARG, "max_iter >= 0, tol >= 0");
    if (!opt) return fail(IMP_ERR_INVALID_ARG, "null options");
    imp_toeplitz_options o = *opt;
    o.enable_tv = 0;  // one CG run, no reweighting passes
    return in_less_memory(ctx, [&]() -> imp_status {
        DevKeep keep;
        imp::ToepSolver *ts = nullptr;
        imp_status s = toeplitz_common(ctx, &o, q_r, q_i, t, num_k, fm, sensi_r, sensi_i, num_coil,
                                       nx, ny, nz, keep, &ts);
        if (s != IMP_OK) return s;
        const size_t N = (size_t)nx * ny * nz;
        const float *dfr, *dfi, *dx0r, *dx0i;
        float *dxr, *dxi;
        bool hr, hi;
        if ((s = imp::to_device_staged(ctx, fhd_r, N, &dfr, nullptr)) ||
            (s = imp::to_device_staged(ctx, fhd_i, N, &dfi, nullptr)) ||
            (s = imp::to_device_staged(ctx, x_r, N, &dx0r, nullptr)) ||
            (s = imp::to_device_staged(ctx, x_i, N, &dx0i, nullptr)) ||
            (s = imp::out_device_staged(ctx, x_r, N, &dxr, &hr)) ||
            (s = imp::out_device_staged(ctx, x_i, N, &dxi, &hi)))
            return s;
        const cudaMemcpyKind d2d = cudaMemcpyDeviceToDevice;
        if (hr) IMP_CUDA(cudaMemcpyAsync(dxr, dx0r, N * 4, d2d, ctx->stream), "x0");
        if (hi) IMP_CUDA(cudaMemcpyAsync(dxi, dx0i, N * 4, d2d, ctx->stream), "x0");
        int it = 0;
        IMP_CUDA(ts->solve_from(dfr, dfi, dxr, dxi, tol, max_iter, &it), "toeplitz warm CG");
        if (iterations) *iterations = it;
        if (hr && (s = copy_out(ctx, x_r, dxr, N))) return s;
        if (hi && (s = copy_out(ctx, x_i, dxi, N))) return s;
        s = imp::finish(ctx);
        ctx->launches = ts->launches();
        return s;
    });
}

imp_status imp_grid_fft(imp_context *ctx, float *data_r, float *data_i, int n0, int n1, int n2,
                        int batch, int inverse) {
    if (!data_r || !data_i) return fail(IMP_ERR_INVALID_ARG, "null array argument");
    if (n0 < 1 || n1 < 1 || n2 < 1 || batch < 1)
        return fail(IMP_ERR_INVALID_ARG, "grid sizes and batch must be >= 1");
    const size_t n = (size_t)batch * n0 * n1 * n2;
    if (n > ((size_t)1 << 31)) return fail(IMP_ERR_INVALID_ARG, "grid larger than 2^31 points");
    imp_status s = imp::begin(ctx);
    if (s != IMP_OK) return s;
    imp::GridFft f;
    const cudaError_t pe = imp::grid_fft_create(&f, n0, n1, n2, batch);
    if (pe == cudaErrorInvalidValue)
        return fail(IMP_ERR_UNSUPPORTED, "grid FFT: an axis is longer than 4096 points or has "
                                         "a prime factor above 255");
    IMP_CUDA(pe, "grid FFT plan");
    std::unique_ptr<imp::GridFft, void (*)(imp::GridFft *)> guard(&f, imp::grid_fft_destroy);
    DevKeep keep;
    const float *dr, *di;
    float *odr, *odi;
    bool hr, hi;
    if ((s = imp::to_device(ctx, data_r, n, keep, &dr, nullptr)) ||
        (s = imp::to_device(ctx, data_i, n, keep, &di, nullptr)) ||
        (s = imp::out_device(ctx, data_r, n, keep, &odr, &hr)) ||
        (s = imp::out_device(ctx, data_i, n, keep, &odi, &hi)))
        return s;
    void *buf = nullptr;
    IMP_CUDA(cudaMalloc(&buf, n * sizeof(float2)), "grid FFT buffer");
    keep.emplace_back(buf, [](void *q) { cudaFree(q); });
    float2 *b = (float2 *)buf;
    const cudaStream_t st = ctx->stream;
    imp::k_soa2c<<<imp::gridn(n), imp::kVB, 0, st>>>(b, dr, di, n);
    IMP_CUDA(cudaGetLastError(), "grid FFT pack");
    IMP_CUDA(imp::grid_fft_exec(f, b, inverse != 0, st), "grid FFT");
    imp::k_c2soa<<<imp::gridn(n), imp::kVB, 0, st>>>(odr, odi, b, n);
    IMP_CUDA(cudaGetLastError(), "grid FFT unpack");
    if (hr && (s = copy_out(ctx, data_r, odr, n))) return s;
    if (hi && (s = copy_out(ctx, data_i, odi, n))) return s;
    s = imp::finish(ctx);
    ctx->launches = 2 + f.passes();
    return s;
}

imp_status imp_toeplitz_apply(imp_context *ctx, const imp_toeplitz_options *opt, float *q_out_r,
                              float *q_out_i, const float *p_r, const float *p_i,
                              const float *q_r, const float *q_i, const float *t, int num_k,
                              const float *fm, const float *sensi_r, const float *sensi_i,
                              int num_coil, int nx, int ny, int nz) {
    if (!q_out_r || !q_out_i || !p_r || !p_i)
        return fail(IMP_ERR_INVALID_ARG, "null array argument");
    return in_less_memory(ctx, [&]() -> imp_status {
        DevKeep keep;
        imp::ToepSolver *ts = nullptr;
        imp_status s = toeplitz_common(ctx, opt, q_r, q_i, t, num_k, fm, sensi_r, sensi_i, num_coil,
                                       nx, ny, nz, keep, &ts);
        if (s != IMP_OK) return s;
        const size_t N = (size_t)nx * ny * nz;
        const float *dpr, *dpi;
        float *dor, *doi;
        bool hr, hi;
        if ((s = imp::to_device_staged(ctx, p_r, N, &dpr, nullptr)) ||
            (s = imp::to_device_staged(ctx, p_i, N, &dpi, nullptr)) ||
            (s = imp::out_device_staged(ctx, q_out_r, N, &dor, &hr)) ||
            (s = imp::out_device_staged(ctx, q_out_i, N, &doi, &hi)))
            return s;
        IMP_CUDA(ts->apply(dpr, dpi, dor, doi), "toeplitz apply");
        if (hr && (s = copy_out(ctx, q_out_r, dor, N))) return s;
        if (hi && (s = copy_out(ctx, q_out_i, doi, N))) return s;
        s = imp::finish(ctx);
        ctx->launches = ts->launches();
        return s;
    });
}

}  // extern "C"
