// Row transforms in three register stages, M = R1 R2 R3 fixed at compile time.
//
// What bounds it, and why this form: a row is read and written once (8 bytes
// a real pair each way), which the shared-memory transforms of fft.cuh missed
// by three times: five stages of radix 4 to 8 with run-time strides spend
// their time on index arithmetic and barriers.  With radices 4 to 20 three
// stages cover every length, all strides are constants, and two exchanges
// through shared memory join the stages.  The thread that holds output
// columns j + r M / R3 also takes M / R3 - j, so the real packing (forward)
// and unpacking (inverse, at the first stage) pair bins k and M - k in
// registers, one twiddle for both.  Blocks are persistent over the rows; the
// next row is copied (cp.async) into shared memory while the current one is
// transformed.  Stage twiddles are compact tables read through L1.
//
// 10560 rows, shared-memory stages -> this, in us (floor: one read and one
// write at the copy rate): M = 1600 forward 125 -> 68, inverse 170 -> 79,
// complex 143 -> 54 (42); M = 3584 266 -> 147, 438 -> 162, 352 -> 128 (94);
// M = 400 63 -> 23, 80 -> 29, 88 -> 20 (11).  960 rows, M = 1600: 27 -> 14.
// 10560 rows are 50 to 100 % above the floor: latency of the row's own chain
// at 30 to 50 % occupancy, set by the registers of the paired stage.
//
// Exchange layouts (float2 index): the first stage's v[r] of butterfly j at
// r S1 + j with S1 odd, the second's at (j / R1) S2 + r R1 + j mod R1 with
// S2 = R1 mod 16: both are written and read without bank conflicts beyond
// the one or two where a radix below 16 wraps inside a half warp.
#pragma once

#include <atomic>

#include "fft.cuh"
#include "kernels.cuh"

namespace wctb200 {

// The plans: radices of the forward order (the inverse runs them reversed).
// The smallest is last, where the forward pairs two butterflies a thread.
// Lengths: from 256 to 6000, the halves of the time-FFT lengths that the
// reference's window lengths lead to (gpu_fft_length) as far as three of the
// radices make them (not 2058, 2430, 4116, 4704 and 5376), and the halves of
// round record lengths, which the noise and the 2-D transforms run at (1000,
// 1120, 1200, 1500, 1536, 1920, 2000, 2400, 3072, 4000). Other lengths take the
// transforms of fft.cuh.
#define WCT_FFT3_PLANS(X)                                                                              \
    X(8, 8, 4) X(8, 7, 5) X(8, 8, 5) X(10, 7, 5) X(8, 8, 6) X(10, 8, 5) X(12, 6, 6) X(8, 8, 7) X(8, 8, 8) \
    X(10, 8, 7) X(10, 8, 8) X(12, 8, 7) X(14, 7, 7) X(10, 10, 7) X(12, 8, 8) X(10, 10, 8) X(14, 8, 8)   \
    X(10, 10, 10) X(16, 8, 8) X(14, 10, 8) X(12, 10, 10) X(16, 10, 8) X(14, 12, 8) X(14, 14, 7)         \
    X(15, 10, 10) X(16, 12, 8) X(16, 10, 10) X(16, 14, 8) X(16, 15, 8) X(20, 10, 10) X(16, 16, 8)       \
    X(16, 14, 10) X(16, 15, 10) X(16, 16, 10) X(16, 14, 12) X(20, 14, 10) X(16, 15, 12) X(20, 15, 10)   \
    X(16, 14, 14) X(15, 15, 14) X(16, 16, 12) X(16, 15, 14) X(16, 16, 14) X(20, 14, 14) X(20, 20, 10)   \
    X(16, 16, 16) X(20, 16, 14) X(20, 16, 16) X(20, 20, 15)

template <int R1_, int R2_, int R3_>
struct Fft3 {
    static constexpr int R1 = R1_, R2 = R2_, R3 = R3_;
    static constexpr int M = R1 * R2 * R3;
    static constexpr int N1 = M / R1, N2 = M / R2, NS = R1 * R2;
    static constexpr int S1 = N1 | 1;
    static constexpr int S2 = NS + ((R1 - NS) % 16 + 16) % 16;
    static constexpr int E1 = R1 * S1, E2 = R3 * S2;
    static constexpr int T2 = (R2 - 1) * R1;  // stage-2 twiddles, then (R3 - 1) NS of stage 3
    // one exchange buffer for both stages where two would leave an SM under three blocks
    static constexpr bool kShare = M > 2048;
    static constexpr int kEx = kShare ? (E1 > E2 ? E1 : E2) : E1 + E2;
    static constexpr size_t kSmem = sizeof(float2) * (size_t)(M + kEx);
    static constexpr int cmax(int a, int b) { return a > b ? a : b; }
    static constexpr int threads(int a, int b, int c) { return (cmax(cmax(a, b), c) + 31) / 32 * 32; }
};

namespace fft3 {

// Second stage of every transform: butterfly j of M / R2 reads the first
// stage's outputs, multiplies the twiddles and writes for the third.
template <class P, int SIGN>
__device__ __forceinline__ void stage2(const float2* __restrict__ e1, float2* __restrict__ e2,
                                       const float2* __restrict__ t2, int j)
{
    const int k = j % P::R1, m = j / P::R1;
    float2 v[P::R2];
    if (j < P::N2) {
#pragma unroll
        for (int r = 0; r < P::R2; ++r) v[r] = e1[k * P::S1 + m + r * P::R3];
#pragma unroll
        for (int r = 1; r < P::R2; ++r) {
            const float2 w = __ldg(t2 + (r - 1) * P::R1 + k);
            v[r] = SIGN < 0 ? cmul(v[r], w) : cmulc(v[r], w);
        }
        fftk::bfly<P::R2, SIGN>(v);
    }
    if (P::kShare) __syncthreads();  // the first stage's outputs have been read
    if (j < P::N2) {
#pragma unroll
        for (int r = 0; r < P::R2; ++r) e2[m * P::S2 + r * P::R1 + k] = v[r];
    }
}

// Third-stage butterfly of column j: v[r] is output j + r NS.
template <class P, int SIGN>
__device__ __forceinline__ void stage3(const float2* __restrict__ e2, const float2* __restrict__ t3, int j, float2* v)
{
#pragma unroll
    for (int r = 0; r < P::R3; ++r) v[r] = e2[j + r * P::S2];
#pragma unroll
    for (int r = 1; r < P::R3; ++r) {
        const float2 w = __ldg(t3 + (r - 1) * P::NS + j);
        v[r] = SIGN < 0 ? cmul(v[r], w) : cmulc(v[r], w);
    }
    fftk::bfly<P::R3, SIGN>(v);
}

// Asynchronous copy of a row of len floats (16-byte aligned) into shared
// memory, zeros up to 2 M; one commit group.
template <int M>
__device__ __forceinline__ void copy_row(float2* s, const float* __restrict__ x, int len, int tid, int nth)
{
    for (int p = tid; p < M / 2; p += nth) {
        const int left = len - 4 * p;
        cp_async16(s + 2 * p, left > 0 ? x + 4 * p : x, left >= 4 ? 16 : (left > 0 ? 4 * left : 0));
    }
    cp_async_commit();
}

// The same for a row of 2 M values of a charge grid: tiles without visits
// (s_cnt, per tile of the row) were not written and count as zero. A piece
// that two tiles share is read if one of them has visits; the raster zeroes
// the other's part of it.
template <int M>
__device__ __forceinline__ void copy_tiles(float2* s, const float* __restrict__ x, const int* s_cnt, int off, int tid,
                                           int nth)
{
    for (int p = tid; p < M / 2; p += nth) {
        const int q = 4 * p + off;  // tick past the first tile's first
        const bool live = s_cnt[q / kTile] | s_cnt[(q + 3) / kTile];
        cp_async16(s + 2 * p, x + 4 * p, live ? 16 : 0);
    }
    cp_async_commit();
}

// Asks for the visit counts of a row's tiles (wire w; outside the plane or
// the readout: as if visited, the raster writes those); the caller commits.
__device__ __forceinline__ void ask_counts(int* s_cnt, const TileMap& t, int w, int tid)
{
    if (tid >= t.ntile) return;
    const int k = t.ktile0 + tid;
    if (w >= 0 && w < t.nwires && k >= 0 && k < t.ntiles_abs) cp_async4(s_cnt + tid, t.cnt + w * t.ntiles_abs + k);
    else s_cnt[tid] = 1;
}

}  // namespace fft3

// ---------------------------------------------------------------------------
// Real rows (in_len values, zeros beyond) -> M packed bins, in place allowed:
// one row, staged in sm_row; ask() copies the next one there once it is taken.
// ---------------------------------------------------------------------------
template <class P>
struct RfftShape {
    static constexpr int kThreads = P::threads(P::N1, P::N2, P::NS / 2 + 1);
    // resident blocks an SM asked for, from the registers that two butterflies of R3 take
    static constexpr int kRegs = P::R3 <= 8 ? 64 : P::R3 <= 10 ? 72 : P::R3 <= 12 ? 80 : 104;
    static constexpr int kBlocks = P::cmax(1, 65536 / (kThreads * kRegs));
};

template <class P, class Ask>
__device__ __forceinline__ void rfft3_row(const float2* sm_row, float2* ex, float2* __restrict__ o,
                                          const float2* __restrict__ t3, const float2* __restrict__ twh, int tid,
                                          Ask ask)
{
    float2* e1 = ex;
    float2* e2 = P::kShare ? ex : ex + P::E1;
    if (tid < P::N1) {
        float2 v[P::R1];
#pragma unroll
        for (int r = 0; r < P::R1; ++r) v[r] = sm_row[tid + r * P::N1];
        fftk::bfly<P::R1, -1>(v);
#pragma unroll
        for (int r = 0; r < P::R1; ++r) e1[r * P::S1 + tid] = v[r];
    }
    __syncthreads();  // the staged row has been taken too
    ask();
    fft3::stage2<P, -1>(e1, e2, t3, tid);
    __syncthreads();
    const int a = tid;
    if (a <= P::NS / 2) {
        const int b = a ? P::NS - a : 0;
        float2 va[P::R3], vb[P::R3];
        fft3::stage3<P, -1>(e2, t3 + P::T2, a, va);
        fft3::stage3<P, -1>(e2, t3 + P::T2, b, vb);
        if (a == 0) {  // column 0 pairs with itself, one row of outputs further
#pragma unroll
            for (int r = 0; r < P::R3; ++r) vb[r] = va[(r + 1) % P::R3];
        }
        // bins k and M - k: E = (Z_k + conj Z_{M-k}) / 2, O = -i (Z_k - conj Z_{M-k}) / 2,
        // X_k = E + w_k O, X_{M-k} = conj(E - w_k O)
#pragma unroll
        for (int r = 0; r < P::R3; ++r) {
            const int k = a + r * P::NS;
            const float2 zk = va[r], zm = cconj(vb[P::R3 - 1 - r]);
            if (k == 0) o[0] = make_float2(zk.x + zk.y, zk.x - zk.y);
            else {
                const float2 E = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y + zm.y));
                const float2 O = make_float2(0.5f * (zk.y - zm.y), -0.5f * (zk.x - zm.x));
                const float2 t = cmul(__ldg(twh + k), O);
                o[k] = cadd(E, t);
                o[P::M - k] = cconj(csub(E, t));
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Packed bins -> real values of ticks tick0 + c, c < ncols, inside [0, nticks)
// of a frame row: one row.
// ---------------------------------------------------------------------------
template <class P>
struct IrfftShape {
    static constexpr int kThreads = P::threads(P::N1 / 2 + 1, P::N2, P::NS);
    static constexpr int kRegs = P::R1 <= 7 ? 96 : P::R1 <= 10 ? 112 : P::R1 <= 14 ? 128 : 168;
    static constexpr int kBlocks = P::cmax(1, 65536 / (kThreads * kRegs));
};

// ADD: onto the frame's values (tick0 0, ncols = nticks), which `next` then
// points to where they are 16-byte aligned (more): they arrive while the row is
// transformed.
template <class P, bool ADD = false>
__device__ __forceinline__ void irfft3_row(const float2* sm_row, float2* ex, float* __restrict__ f, int tick0,
                                           int ncols, int nticks, bool vec, const float2* __restrict__ t3,
                                           const float2* __restrict__ twh, int tid, bool more, const float2* next)
{
    float2* e1 = ex;
    float2* e2 = P::kShare ? ex : ex + P::E1;
    const int a = tid;
    if (a <= P::N1 / 2) {
        const int b = a ? P::N1 - a : 0;
        float2 xa[P::R1], xb[P::R1];
#pragma unroll
        for (int r = 0; r < P::R1; ++r) {
            xa[r] = sm_row[a + r * P::N1];
            xb[r] = sm_row[b + r * P::N1];
        }
        if (a == 0) {
#pragma unroll
            for (int r = 0; r < P::R1; ++r) xb[r] = xa[(r + 1) % P::R1];
        }
        // E = (X_k + conj X_{M-k}) / 2, O = conj(w_k) (X_k - conj X_{M-k}) / 2,
        // Z_k = E + i O, Z_{M-k} = conj(E - i O)
        float2 za[P::R1], zb[P::R1];
#pragma unroll
        for (int r = 0; r < P::R1; ++r) {
            const float2 xk = xa[r], xm = cconj(xb[P::R1 - 1 - r]);
            const float2 E = make_float2(0.5f * (xk.x + xm.x), 0.5f * (xk.y + xm.y));
            const float2 D = make_float2(0.5f * (xk.x - xm.x), 0.5f * (xk.y - xm.y));
            const float2 O = cmulc(D, __ldg(twh + a + r * P::N1));
            za[r] = make_float2(E.x - O.y, E.y + O.x);
            zb[P::R1 - 1 - r] = make_float2(E.x + O.y, O.x - E.y);
        }
        if (a == 0) za[0] = make_float2(0.5f * (xa[0].x + xa[0].y), 0.5f * (xa[0].x - xa[0].y));
        fftk::bfly<P::R1, +1>(za);
#pragma unroll
        for (int r = 0; r < P::R1; ++r) e1[r * P::S1 + a] = za[r];
        if (b != a) {
            fftk::bfly<P::R1, +1>(zb);
#pragma unroll
            for (int r = 0; r < P::R1; ++r) e1[r * P::S1 + b] = zb[r];
        }
    }
    __syncthreads();
    if (more) fft3::copy_row<P::M>(const_cast<float2*>(sm_row), reinterpret_cast<const float*>(next),
                                   ADD ? ncols : 2 * P::M, tid, IrfftShape<P>::kThreads);
    fft3::stage2<P, +1>(e1, e2, t3, tid);
    if (ADD) cp_async_wait<0>();
    __syncthreads();
    if (tid < P::NS) {
        float2 v[P::R3];
        fft3::stage3<P, +1>(e2, t3 + P::T2, tid, v);
        const float sc = 1.0f / (float)P::M;
#pragma unroll
        for (int r = 0; r < P::R3; ++r) {
            const int c0 = 2 * (tid + r * P::NS), t0 = tick0 + c0;
            float2 z = make_float2(v[r].x * sc, v[r].y * sc);
            if (ADD) {
                const float* was = more ? reinterpret_cast<const float*>(sm_row) : f;
                if (c0 < ncols) z.x += was[c0];
                if (c0 + 1 < ncols) z.y += was[c0 + 1];
            }
            if (vec && c0 + 1 < ncols && t0 >= 0 && t0 + 1 < nticks) *reinterpret_cast<float2*>(f + t0) = z;
            else {
                if (c0 < ncols && t0 >= 0 && t0 < nticks) f[t0] = z.x;
                if (c0 + 1 < ncols && t0 + 1 >= 0 && t0 + 1 < nticks) f[t0 + 1] = z.y;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Launch helpers
// ---------------------------------------------------------------------------
// Persistent blocks of a kernel on the current device (looked up once per
// kernel and device), its shared memory allowed.
constexpr int kFft3Devices = 64;
inline int persistent_blocks(const void* f, int threads, size_t smem, std::atomic<int>* cache)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return 0;
    if (dev < kFft3Devices) {
        const int n = cache[dev].load(std::memory_order_acquire);
        if (n > 0) return n;
    }
    int nsm = 0, per = 0;
    if (smem > 40 * 1024 &&  // (a kernel's own static arrays count towards the 48 KB too)
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return 0;
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, threads, smem) != cudaSuccess) return 0;
    if (dev < kFft3Devices) cache[dev].store(per * nsm, std::memory_order_release);
    return per * nsm;
}

#define WCT_CASE(A, B, C, ...)                                                                         \
    case A * B * C: {                                                                                 \
        using P = Fft3<A, B, C>;                                                                      \
        using I = Fft3<C, B, A>;                                                                      \
        (void)sizeof(P);                                                                              \
        (void)sizeof(I);                                                                              \
        __VA_ARGS__;                                                                                       \
    }

}  // namespace wctb200
