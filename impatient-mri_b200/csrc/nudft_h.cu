// NUDFT tile engine on the tensor cores, FP16 head / tail operands.
//
// Same operator, inputs and partial-sum layout as k_nudft (nudft.cu), which
// replaces ftGpuKernel / iftGpuKernel (kernels/ftGpu.cu:306-604, 756-1013) and
// the coil loop of parallelFtGpu / parallelIftGpu (kernels/parImagingGpu.cu:92-152).
//
// For every (ours, theirs) pair the CUDA cores compute the exact fixed-point
// phase and e = (cos, sin) once and split it into an FP16 head and tail
// (v = h + l, 11 significant bits each, |v| <= 1); the per-coil complex
// multiply-add is an FP16 x FP16 -> FP32 tcgen05.mma.  The "theirs" data d_c
// is scaled per (64-element tile, coil) by a power of two that puts its largest
// component into [2^14, 2^15) and split the same way beforehand (k_h_image):
// a scaled component keeps 22 bits or an absolute error of 2^-25, 2^-40 of the
// tile's largest.  With the accumulator columns
//     n = 2c, 2c + 1          (re, im, head):  (dh_x,  dh_y), (dh_y, -dh_x)
//     n = H + 2c, H + 2c + 1  (re, im, tail):  the same of dl    (H = N / 2)
// the head MMA multiplies the e heads by all N columns (h h + h l), the tail
// MMA the e tails by the head columns (l h); l l is below 2^-23 of a term.
// Every 64 "theirs" elements the accumulator moves into FP32 registers,
// multiplied by the tile's inverse scale (exact).
//
// Against the TF32 form of the same split (nudft_tc.cu) a pair takes two
// 32-bit A columns instead of four and an MMA covers eight pairs per row
// instead of two, the conversion packs two values per instruction, and the B
// operand is expanded once per apply instead of once per row tile.
//
// Per CTA (one per SM): PT accumulator tiles of 128 "ours" rows, PT = 2 up to
// 16 coils and 1 for 32.  Warp roles:
//   warps 0 .. 15   A producers, four groups of four: group g writes elements
//                   8 g .. 8 g + 7 of every 32 (one K = 16 block), warp quadrant
//                   by quadrant of the 128 rows, for all PT row tiles, into A
//                   buffers of its own, so that the groups (the four warps of a
//                   scheduler are of different groups) need not wait in step;
//                   they also drain the accumulators
//   warp 16         bulk loads of the tiles (geometry, B image, scales), three slots
//   warp 17         MMA issue
// Every wait is bounded; after one expiry a thread stops waiting, so a broken
// pipeline ends the launch after one timeout per thread.  The block then waits
// once more (bounded) for its copies and MMAs in flight before it frees its
// tensor memory and ends.
//
// What bounds it: 30 issued instructions per 32 pairs and scheduler (3 or 4 DFMA,
// 2 MUFU, the packs, unpacks and subtraction of the split, the drain's share) at
// 0.62 of the issue slots, 49 cycles (TF32 form: 118); two MUFU alone are 16, the
// MMAs about 20 (75 cycles each whatever N: their issue, so one thread's operands
// must sit in uniform registers, see elect_one).  Adjoint of 192x192 voxels x
// 32768 samples x 32 coils: 1.84 ms; batched apply of 4 slices 160x160, 59392
// samples, 32 coils: 4.1 -> 2.2 ms.
#include "common.cuh"
#include "nudft.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>

namespace imp {

namespace {

constexpr double kMagicH = 1572864.0 + 0.5 + 5.9604644775390625e-08;
constexpr float kTwoPiH = 6.28318530717958647692f;
constexpr float kThreePiH = 9.42477796076937971538f;

// Bounded wait: at most 2^16 tries, each of which the hardware may suspend for
// up to 4 us (a thread that polls without suspending takes issue slots from the
// producers).
__device__ __forceinline__ void h_wait(uint64_t *bar, unsigned parity, bool &ok) {
    if (!ok) return;
    const unsigned addr = smem_u32(bar);
    for (unsigned it = 0; it < (1u << 16); ++it) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity), "r"(4000u)
            : "memory");
        if (done) return;
    }
    ok = false;
}

__device__ __forceinline__ void h_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void h_commit(uint64_t *bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}

// K-major, 128-byte swizzle, version 1; sbo = one 8-row group (1024 B).
__device__ __forceinline__ uint64_t h_bdesc(unsigned saddr) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// FP16 x FP16 -> FP32, A (tensor memory) and B K-major, M = 128.
__host__ __device__ constexpr uint32_t h_idesc(int N) {
    return (1u << 4) | ((uint32_t)(N >> 3) << 17) | (8u << 24);
}

__device__ __forceinline__ void h_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc,
                                      uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void h_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(
                     taddr),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
                 "r"(v[7])
                 : "memory");
}

__device__ __forceinline__ void h_ld8(uint32_t taddr, uint32_t *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),
                   "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
}

__device__ __forceinline__ void h_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void h_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

template <int CG>
struct HShape {
    static constexpr int PT = CG >= 32 ? 1 : 2;
    static constexpr int NN = CG <= 4 ? 16 : 4 * CG;  // accumulator columns
    static constexpr int NH = NN / 2;                 // tail columns start here
    static constexpr int NT = NH % 16 == 0 ? NH : NN; // columns of the tail MMA (M = 128: 16 k)
    static constexpr int SLOTS = NN / 4;              // coil slots (4 when CG < 4)
    static constexpr int GROUPS = 4, PROD = 16;       // producer groups (of 4 warps), warps
    static constexpr int JPW = 8;                     // "theirs" of a group's chunk: one K = 16
    static constexpr int KC = GROUPS * JPW;           // "theirs" per round of the groups
    static constexpr int ROUNDS = kTile / KC;
    static constexpr int ACOLS = 2 * JPW;             // A columns of a chunk and row tile
    static constexpr int NB = 2;                      // A chunk buffers per group
    static constexpr int DCOLS = 2 * PT * NN;         // two accumulator sets
    static constexpr int USED = DCOLS + GROUPS * NB * PT * ACOLS;
    static constexpr int TMEM = USED <= 256 ? 256 : 512;
    static constexpr int BCHUNK = NN * 128;           // B of one round: NN rows of 64 FP16
    static constexpr int BTILE = ROUNDS * BCHUNK;
    static constexpr int SBYTES = SLOTS * 4;          // inverse scales of a tile
    static constexpr int ITILE = BTILE + 128;         // image bytes per tile (scales after B)
    static constexpr int THREADS = 32 * (PROD + 2);
    static constexpr int NSLOT = 3;                   // tile slots
    // Accumulator drain: the GROUPS / PT groups of a row tile share its coils
    // (from 8 coils up; below, one of them takes all).
    static constexpr int SHARE = CG >= 8 ? GROUPS / PT : 1;
    static constexpr int NC = SLOTS / SHARE;          // coil slots per draining thread
    static_assert(USED <= 512 && SBYTES <= 128 && KC == 32, "shape");
    static_assert(ROUNDS == NB, "a round's buffer index is its place in the tile");
    static_assert((2 * NC) % 8 == 0, "8-column drains");
    // dynamic shared memory: B slots (1024-aligned) | geo | scales | red
    static constexpr size_t SMEM = 1024 + NSLOT * ((size_t)BTILE + kTile * sizeof(double4) + 128) +
                                   3 * 128 * sizeof(float2);
};

// B image of every tile of `tdata` [tiles][64][CG]: FP16 heads and tails in the
// MMA's swizzled layout, then the inverse scales.  One block per tile.
template <int CG>
__global__ void __launch_bounds__(256) k_h_image(unsigned char *__restrict__ img,
                                                 const float2 *__restrict__ tdata) {
    using S = HShape<CG>;
    __shared__ float2 sd[kTile * (CG + 1)];
    const float2 *src = tdata + (size_t)blockIdx.x * kTile * CG;
    for (int i = threadIdx.x; i < kTile * CG; i += 256) sd[(i / CG) * (CG + 1) + i % CG] = src[i];
    __syncthreads();
    unsigned char *dst = img + (size_t)blockIdx.x * S::ITILE;
    const int lane = threadIdx.x & 31;
    for (int c = threadIdx.x >> 5; c < S::SLOTS; c += 8) {
        float2 d[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        float m = 0.f;
        if (c < CG) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                d[h] = sd[(lane + 32 * h) * (CG + 1) + c];
                m = fmaxf(m, fmaxf(fabsf(d[h].x), fabsf(d[h].y)));
            }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(~0u, m, o));
        int k = 0;  // scale 2^k: an all-zero or non-finite tile is left as it is
        if (m > 0.f && m <= 3.402823466e38f) k = max(-112, min(14 - ilogbf(m), 126));
        const float up = __int_as_float((k + 127) << 23);
        if (lane == 0)
            reinterpret_cast<float *>(dst + S::BTILE)[c] = __int_as_float((127 - k) << 23);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float x = d[h].x * up, y = d[h].y * up;
            const __half xh = __float2half_rn(x), yh = __float2half_rn(y);
            const __half xl = __float2half_rn(x - __half2float(xh));
            const __half yl = __float2half_rn(y - __half2float(yh));
            const __half2 rows[4] = {__halves2half2(xh, yh), __halves2half2(yh, __hneg(xh)),
                                     __halves2half2(xl, yl), __halves2half2(yl, __hneg(xl))};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int n = (r >> 1) * S::NH + 2 * c + (r & 1);
                *reinterpret_cast<__half2 *>(dst + h * S::BCHUNK + n * 128 +
                                             (((lane >> 2) ^ (n & 7)) << 4) + (lane & 3) * 4) =
                    rows[r];
            }
        }
    }
}

template <int CG, bool USEZ, bool ADJ, bool BATCH>
__global__ void __launch_bounds__(HShape<CG>::THREADS, 1)
    k_nudft_h(const double4 *__restrict__ ours, const double4 *__restrict__ theirs,
              const unsigned char *__restrict__ img, const float2 *__restrict__ sens,
              float2 *__restrict__ out, int n_ours_pad, int n_theirs_pad, int per_split,
              unsigned *err, const NuSlice *__restrict__ sl, int n_groups) {
    using S = HShape<CG>;
    constexpr int PT = S::PT;
    extern __shared__ unsigned char smraw[];
    __shared__ __align__(8) uint64_t full[S::NSLOT], tempty[S::NSLOT];
    __shared__ __align__(8) uint64_t afull[S::GROUPS][S::NB], aempty[S::GROUPS][S::NB];
    __shared__ __align__(8) uint64_t dfull[2], ddone[2], last;
    __shared__ uint32_t tmem_sh;

    const int warp = (int)warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    int g = blockIdx.z;
    size_t tile0 = 0;  // first tile of this slice in the image
    if constexpr (BATCH) {
        const int s = blockIdx.z / n_groups;
        g = blockIdx.z - s * n_groups;
        const NuSlice d = sl[s];
        if (blockIdx.x * (128 * PT) >= d.n_ours) return;  // whole block: before any barrier
        ours += d.ours;
        theirs += d.theirs;
        tile0 = (size_t)d.tdata / (kTile * CG);
        out += d.out;
        n_ours_pad = d.n_ours;
        n_theirs_pad = d.n_theirs;
        per_split = d.per_split;
    }
    const int split = blockIdx.y;
    const int t0 = split * per_split;
    const int ntiles = per_split / kTile;
    const double4 *gsrc = theirs + t0;
    const unsigned char *isrc =
        img + (tile0 + ((size_t)g * n_theirs_pad + t0) / kTile) * S::ITILE;
    constexpr unsigned kGeoBytes = kTile * sizeof(double4);

    unsigned char *s_b = smraw + ((1024u - (smem_u32(smraw) & 1023u)) & 1023u);  // [NSLOT][BTILE]
    double4 *s_geo = reinterpret_cast<double4 *>(s_b + S::NSLOT * S::BTILE);     // [NSLOT][kTile]
    float *s_scl = reinterpret_cast<float *>(s_geo + S::NSLOT * kTile);          // [NSLOT][32]
    float2 *s_red = reinterpret_cast<float2 *>(s_scl + S::NSLOT * 32);           // [3][128]

    if (warp == S::PROD + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmem_sh)),
                     "r"(S::TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < S::NSLOT; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&tempty[i], S::PROD);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&dfull[i], 1);
            mbar_init(&ddone[i], S::PROD);
        }
        for (int i = 0; i < S::GROUPS * S::NB; ++i) {
            mbar_init(&afull[0][0] + i, S::PROD / S::GROUPS);
            mbar_init(&aempty[0][0] + i, 1);
        }
        mbar_init(&last, 1);
        fence_mbar_init();
    }
    h_fence_before();
    __syncthreads();
    h_fence_after();
    const uint32_t tmem = warp_uniform(tmem_sh);
    bool ok = true;
    int issued = 0;  // tiles whose copies were started (bulk-load thread)

    if (warp < S::PROD) {
        // ------------------------------ A producers ------------------------------
        const int quad = warp & 3, grp = warp >> 2;
        const int row = quad * 32 + lane;
        const int e0 = blockIdx.x * (128 * PT) + row;
        double ox[PT], oy[PT], oz[PT], ow[PT];
#pragma unroll
        for (int p = 0; p < PT; ++p) {
            const double4 q = ours[e0 + p * 128];
            ox[p] = q.x;
            oy[p] = q.y;
            oz[p] = q.z;
            ow[p] = q.w;
        }
        // this thread's part of the drain: row tile and coil slots
        const int dtile = S::SHARE == 1 ? grp : grp / S::SHARE;
        const int dpart = S::SHARE == 1 ? 0 : grp % S::SHARE;
        const bool drains = dtile < PT;
        float acc[2 * S::NC];
#pragma unroll
        for (int n = 0; n < 2 * S::NC; ++n) acc[n] = 0.f;
        const uint32_t tlane = tmem + ((uint32_t)(quad * 32) << 16);
        auto drain = [&](int t) {  // acc += inverse scale x accumulators of tile t
            const int b = t & 1, slot = t % S::NSLOT;
            h_wait(&dfull[b], (unsigned)(t >> 1) & 1, ok);
            h_fence_after();
            if (drains) {
                const uint32_t dcol =
                    tlane + (uint32_t)((b * PT + dtile) * S::NN + dpart * 2 * S::NC);
                const float *scl = s_scl + slot * 32 + dpart * S::NC;
                uint32_t h[2 * S::NC], l[2 * S::NC];
#pragma unroll
                for (int n0 = 0; n0 < 2 * S::NC; n0 += 8) {
                    h_ld8(dcol + (uint32_t)n0, h + n0);
                    h_ld8(dcol + (uint32_t)(S::NH + n0), l + n0);
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int n = 0; n < 2 * S::NC; ++n)
                    acc[n] = fmaf(__uint_as_float(h[n]) + __uint_as_float(l[n]), scl[n >> 1], acc[n]);
            }
            h_fence_before();
            __syncwarp();
            if (lane == 0) {
                h_arrive(&ddone[b]);
                h_arrive(&tempty[slot]);
            }
        };
        int ci = 0;  // chunk counter
        for (int t = 0; t < ntiles; ++t) {
            const int slot = t % S::NSLOT;
            if (t >= 2) drain(t - 2);
            h_wait(&full[slot], (unsigned)(t / S::NSLOT) & 1, ok);
            const double4 *geo = s_geo + slot * kTile + grp * S::JPW;
#pragma unroll 1
            for (int c = 0; c < S::ROUNDS; ++c, ++ci) {
                const int ab = ci % S::NB;
                uint32_t vh[PT][S::JPW], vl[PT][S::JPW];
#pragma unroll
                for (int jj = 0; jj < S::JPW; ++jj) {
                    const double4 q = geo[c * S::KC + jj];
#pragma unroll
                    for (int p = 0; p < PT; ++p) {
                        double a = fma(ox[p], q.x, kMagicH);
                        a = fma(oy[p], q.y, a);
                        if (USEZ) a = fma(oz[p], q.z, a);
                        a = fma(ow[p], q.w, a);
                        const unsigned P = (unsigned)__double2loint(a);
                        const float f1 = __uint_as_float(__funnelshift_r(P, 0x7Fu, 9));
                        const float ang = ADJ ? fmaf(f1, -kTwoPiH, kThreePiH)
                                              : fmaf(f1, kTwoPiH, -kThreePiH);
                        float sn, cs;
                        __sincosf(ang, &sn, &cs);
                        const __half2 h = __floats2half2_rn(cs, sn);  // cos in the low half
                        const float2 hf = __half22float2(h);
                        const float2 t2 = __ffma2_rn(hf, make_float2(-1.f, -1.f),
                                                     make_float2(cs, sn));  // exact
                        const __half2 l = __floats2half2_rn(t2.x, t2.y);
                        vh[p][jj] = *reinterpret_cast<const uint32_t *>(&h);
                        vl[p][jj] = *reinterpret_cast<const uint32_t *>(&l);
                    }
                }
                // A buffer ab is free once chunk ci - NB's MMAs are done
                if (ci >= S::NB) h_wait(&aempty[grp][ab], (unsigned)(ci / S::NB - 1) & 1, ok);
                h_fence_after();
#pragma unroll
                for (int p = 0; p < PT; ++p) {
                    const uint32_t ta =
                        tlane +
                        (uint32_t)(S::DCOLS + ((grp * S::NB + ab) * PT + p) * S::ACOLS);
                    h_st8(ta, vh[p]);
                    h_st8(ta + S::JPW, vl[p]);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                h_fence_before();
                __syncwarp();
                if (lane == 0) h_arrive(&afull[grp][ab]);
            }
        }
        for (int t = ntiles >= 2 ? ntiles - 2 : 0; t < ntiles; ++t) drain(t);

        // ------------------------------ partial sums -----------------------------
        const int G = BATCH ? n_groups : (int)gridDim.z;
        const int e = blockIdx.x * (128 * PT) + (drains ? dtile : 0) * 128 + row;
        const int c0 = dpart * S::NC;
        if (!ADJ) {
            if (drains) {
                float2 *o = out + ((size_t)(split * G + g) * n_ours_pad + e) * CG + c0;
#pragma unroll
                for (int c = 0; c < S::NC; ++c)
                    if (c < CG) o[c] = make_float2(acc[2 * c], acc[2 * c + 1]);
            }
        } else {
            float zr = 0.f, zi = 0.f;
            if (drains) {
                const float2 *sv = sens + ((size_t)g * n_ours_pad + e) * CG + c0;
#pragma unroll
                for (int c = 0; c < S::NC; ++c)
                    if (c < CG) {
                        const float2 w = sv[c];
                        zr += w.x * acc[2 * c] + w.y * acc[2 * c + 1];
                        zi += w.x * acc[2 * c + 1] - w.y * acc[2 * c];
                    }
            }
            if constexpr (S::SHARE > 1) {
                // coil sum across the groups of a row tile (producer warps only)
                float2 *red = s_red + (dtile * (S::SHARE - 1)) * 128 + row;
                if (dpart > 0) red[(dpart - 1) * 128] = make_float2(zr, zi);
                asm volatile("bar.sync 1, %0;" ::"n"(S::PROD * 32) : "memory");
                if (dpart == 0) {
#pragma unroll
                    for (int k = 0; k < S::SHARE - 1; ++k) {
                        zr += red[k * 128].x;
                        zi += red[k * 128].y;
                    }
                    out[(size_t)(split * G + g) * n_ours_pad + e] = make_float2(zr, zi);
                }
            } else if (drains) {
                out[(size_t)(split * G + g) * n_ours_pad + e] = make_float2(zr, zi);
            }
        }
    } else if (warp == S::PROD) {
        // ------------------------------ bulk loads ------------------------------
        if (lane == 0)
            for (int t = 0; t < ntiles; ++t) {
                const int s = t % S::NSLOT;
                // the slot is free once tile t - NSLOT has been drained (its MMAs are then
                // done and its geometry and scales read)
                if (t >= S::NSLOT) h_wait(&tempty[s], (unsigned)(t / S::NSLOT - 1) & 1, ok);
                if (!ok) break;
                issued = t + 1;
                fence_proxy_async_smem();
                mbar_arrive_expect_tx(&full[s], kGeoBytes + S::BTILE + S::SBYTES);
                bulk_g2s(s_geo + s * kTile, gsrc + (size_t)t * kTile, kGeoBytes, &full[s]);
                const unsigned char *it = isrc + (size_t)t * S::ITILE;
                bulk_g2s(s_b + s * S::BTILE, it, S::BTILE, &full[s]);
                bulk_g2s(s_scl + s * 32, it + S::BTILE, S::SBYTES, &full[s]);
            }
        __syncwarp();
    } else {
        // ------------------------------- MMA issue -------------------------------
        // The whole warp runs the loop (uniform registers), one lane issues.
        constexpr uint32_t IDH = h_idesc(S::NN), IDT = h_idesc(S::NT);
        const uint64_t bd0 = h_bdesc(smem_u32(s_b));
        int ci = 0;
        for (int t = 0; t < ntiles; ++t) {
            const int s = t & 1, slot = t % S::NSLOT;
            if (t >= 2) h_wait(&ddone[s], (unsigned)((t - 2) >> 1) & 1, ok);
            h_wait(&full[slot], (unsigned)(t / S::NSLOT) & 1, ok);
            const uint32_t dbase = tmem + (uint32_t)(s * PT * S::NN);
            const uint64_t bt = bd0 + (uint64_t)(slot * (S::BTILE >> 4));
#pragma unroll
            for (int c = 0; c < S::ROUNDS; ++c, ++ci) {
                const int ab = c;  // ci % NB
                // group kb's chunk is the round's K block kb (always in this order)
#pragma unroll
                for (int kb = 0; kb < S::GROUPS; ++kb) {
                    h_wait(&afull[kb][ab], (unsigned)(ci / S::NB) & 1, ok);
                    h_fence_after();
                    const uint64_t b = bt + (uint64_t)((c * S::BCHUNK + kb * 32) >> 4);
                    if (elect_one()) {
#pragma unroll
                        for (int p = 0; p < PT; ++p) {
                            const uint32_t d = dbase + (uint32_t)(p * S::NN);
                            const uint32_t a =
                                tmem +
                                (uint32_t)(S::DCOLS + ((kb * S::NB + ab) * PT + p) * S::ACOLS);
                            h_mma(d, a, b, IDH, (c > 0 || kb > 0) ? 1u : 0u);
                            h_mma(d, a + S::JPW, b, IDT, 1u);
                        }
                        h_commit(&aempty[kb][ab]);
                        if (c == S::ROUNDS - 1 && kb == S::GROUPS - 1) h_commit(&dfull[s]);
                    }
                    __syncwarp();
                }
            }
        }
    }
    if (!ok && err) atomicOr(err, DEV_ERR_TIMEOUT);
    h_fence_before();
    if (__syncthreads_or(!ok)) {  // a wait ran out: what is in flight ends before the block
        bool again = true;
        if (warp == S::PROD && lane == 0)
            for (int t = max(issued - S::NSLOT, 0); t < issued; ++t)
                h_wait(&full[t % S::NSLOT], (unsigned)(t / S::NSLOT) & 1, again);
        if (warp == S::PROD + 1) {
            if (elect_one()) h_commit(&last);
            __syncwarp();
            h_wait(&last, 0, again);
        }
    }
    if (warp == S::PROD + 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(S::TMEM)
                     : "memory");
}

struct HArgs {
    dim3 grid;
    const double4 *ours, *theirs;
    const float2 *tdata, *sens;
    float2 *out;
    unsigned char *img;
    unsigned tiles;  // tiles of tdata
    int n_ours, n_theirs, per_split;
    unsigned *err;
    const NuSlice *sl;
    int G;
    cudaStream_t st;
};

template <int CG, bool USEZ, bool ADJ, bool BATCH>
cudaError_t launch_h(const HArgs &a) {
    using S = HShape<CG>;
    auto k = k_nudft_h<CG, USEZ, ADJ, BATCH>;
    // the shared-memory limit is set once per instantiation and device (-mgpu
    // workers drive several devices from several threads)
    static std::atomic<unsigned long long> attr_set{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (!bit || !(attr_set.load(std::memory_order_acquire) & bit)) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
        if (e != cudaSuccess) return e;
        attr_set.fetch_or(bit, std::memory_order_acq_rel);
    }
    k_h_image<CG><<<a.tiles, 256, 0, a.st>>>(a.img, a.tdata);
    k<<<a.grid, S::THREADS, S::SMEM, a.st>>>(a.ours, a.theirs, a.img, a.sens, a.out, a.n_ours,
                                             a.n_theirs, a.per_split, a.err, a.sl, a.G);
    return cudaGetLastError();
}

template <int CG>
cudaError_t launch_h_cg(const HArgs &a, bool use_z, bool adj) {
    if (a.sl) {
        if (adj) return use_z ? launch_h<CG, true, true, true>(a) : launch_h<CG, false, true, true>(a);
        return use_z ? launch_h<CG, true, false, true>(a) : launch_h<CG, false, false, true>(a);
    }
    if (adj) return use_z ? launch_h<CG, true, true, false>(a) : launch_h<CG, false, true, false>(a);
    return use_z ? launch_h<CG, true, false, false>(a) : launch_h<CG, false, false, false>(a);
}

cudaError_t launch_any(const HArgs &a, int CG, bool use_z, bool adj) {
    switch (CG) {
        case 1: return launch_h_cg<1>(a, use_z, adj);
        case 2: return launch_h_cg<2>(a, use_z, adj);
        case 4: return launch_h_cg<4>(a, use_z, adj);
        case 8: return launch_h_cg<8>(a, use_z, adj);
        case 16: return launch_h_cg<16>(a, use_z, adj);
        case 32: return launch_h_cg<32>(a, use_z, adj);
        default: return cudaErrorInvalidConfiguration;
    }
}

size_t image_tile_bytes(int CG) {
    switch (CG) {
        case 1: return HShape<1>::ITILE;
        case 2: return HShape<2>::ITILE;
        case 4: return HShape<4>::ITILE;
        case 8: return HShape<8>::ITILE;
        case 16: return HShape<16>::ITILE;
        default: return HShape<32>::ITILE;
    }
}

}  // namespace

size_t nu_image_bytes(int CG, size_t elems) { return elems / kTile * image_tile_bytes(CG); }

cudaError_t nu_partials_h(const NuPlan &p, const NuLaunch &l, bool adj, const float2 *tdata,
                          float2 *out, unsigned *err, cudaStream_t st) {
    const int n_ours = adj ? p.Npad : p.Mpad;
    const int n_theirs = adj ? p.Mpad : p.Npad;
    const int rows = nu_tc_rows(p.CG);
    const size_t elems = (size_t)p.G * n_theirs;
    if (!nu_split_ok(n_theirs, l.split) || n_ours % rows || !p.img ||
        nu_image_bytes(p.CG, elems) > p.img_bytes)
        return cudaErrorInvalidConfiguration;
    HArgs a{dim3(n_ours / rows, l.split, p.G), adj ? p.vgeo : p.kgeo, adj ? p.kgeo : p.vgeo,
            tdata, p.sens, out, p.img, (unsigned)(elems / kTile), n_ours, n_theirs,
            n_theirs / l.split, err, nullptr, p.G, st};
    return launch_any(a, p.CG, p.use_z, adj);
}

cudaError_t nu_partials_h_batch(const NuPlan &p, const NuLaunch &l, bool adj, int S, int max_ours,
                                size_t elems, const NuSlice *d_slices, const double4 *ours,
                                const double4 *theirs, const float2 *tdata, float2 *out,
                                unsigned *err, cudaStream_t st) {
    const int rows = nu_tc_rows(p.CG);
    if ((long long)S * p.G > 65535 || max_ours % rows || !p.img ||
        nu_image_bytes(p.CG, elems) > p.img_bytes || elems % kTile)
        return cudaErrorInvalidConfiguration;
    HArgs a{dim3(max_ours / rows, l.split, S * p.G), ours, theirs, tdata, p.sens, out, p.img,
            (unsigned)(elems / kTile), 0, 0, 0, err, d_slices, p.G, st};
    return launch_any(a, p.CG, p.use_z, adj);
}

}  // namespace imp
