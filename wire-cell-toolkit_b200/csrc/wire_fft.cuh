// Wire-direction convolution in the (wire, frequency) domain by overlap-save:
// blocks of kWL wires are transformed along the wire axis, multiplied with
// the responses' wire spectra and transformed back.
//
//   V[o] = sum_g sum_jj R_g[jj] Q_g[o - jj],  jj = 0 .. 2P   (forward)
//   dQ_g[i] = sum_jj conj(R_g[jj]) G[i + jj]                  (adjoint)
//
// What bounds it, and why this split: the direct form does G (2P + 1) complex
// multiply-adds per output (473 for 11 groups of 43 taps) and ran at the FP32
// pipe.  A transform of 256 wires in two radix-16 stages costs about 25
// operations a point, and there are G + 1 of them per 256 - 2P outputs, so
// the arithmetic falls to under a third.  What is left is shared by the issue
// slots, shared memory and the reads of the grid (x 256 / (256 - 2P)) and of
// the wire spectra, a value for each of the grid's.  A thread block takes 16
// frequencies (128 bytes of every row) x 16 sub-transforms; a thread holds 16
// points, and one shared-memory exchange joins the stages.  Group spectra
// accumulate in registers, so there is one inverse per block however many
// groups.  128 wires (8 x 16) would redo a third of the rows.
// 960 wires, 11 groups of 43 taps, M = 1600: 148 -> 71 us (direct, cp.async
// double buffered -> this); the adjoint 195 -> 113 us.
//
// Bin 0 of a packed row holds two real spectra (DC and Nyquist).  The DC
// value is column 0 here and the Nyquist value column M, each real with
// its own (real-tap) wire spectrum, so no bin needs a special product.
#pragma once

#include "fft.cuh"

namespace wctb200 {

constexpr int kWL = 256;          // wires per transform (16 x 16)
constexpr int kWF = 16;           // frequencies per block
constexpr int kWThreads = 256;    // kWF x 16
constexpr int kWEx = kWL * kWF;   // complex values of one exchange buffer
// shared memory: the exchange buffer (and the tile of grid rows), the twiddles
constexpr size_t kWConvSmem = sizeof(float2) * (2 * kWEx + kWL);
constexpr size_t kWAdjSmem = sizeof(float2) * (kWEx + kWL);
constexpr int kWMaxPad = 64;      // at least half of every block's rows are outputs
constexpr size_t kWMaxSpec = (size_t)1 << 24;  // wire-spectrum values of a plane (128 MB)

__host__ __device__ __forceinline__ int wire_fblocks(int M) { return (M + 1 + kWF - 1) / kWF; }
// Outputs (forward) or inputs (adjoint) of one block.
__host__ __device__ __forceinline__ int wire_valid(int pad) { return kWL - 2 * pad; }
__host__ __device__ __forceinline__ int wire_blocks(int n, int pad)
{
    return (n + wire_valid(pad) - 1) / wire_valid(pad);
}

namespace wfft {

// Twiddles exp(-2 pi i m / 256) into shared memory, once per block (the
// caller synchronises before the first use).
__device__ __forceinline__ void load_twiddles(float2* tw, int tid)
{
    float s, c;
    sincospif(-(float)tid / 128.0f, &s, &c);  // tid / 128 is exact
    tw[tid] = make_float2(c, s);
}

// Transform of 256 points in two halves around the exchange.  In: point
// n = ty + 16 r in v[r] (forward), or bin 16 k1 + ty in v[k1] (inverse).
// Out: bin 16 k1 + ty in v[k1] (forward), or point ty + 16 n2 in v[n2]
// (inverse, unscaled).
template <int SIGN>
__device__ __forceinline__ void fft256_a(float2* v, const float2* __restrict__ tw, int ty)
{
    fftk::bfly16<SIGN>(v);
#pragma unroll
    for (int k = 1; k < 16; ++k) v[k] = SIGN < 0 ? cmul(v[k], tw[ty * k]) : cmulc(v[k], tw[ty * k]);
}
template <int SIGN>
__device__ __forceinline__ void fft256_b(float2* v, float2* ex, int fl, int ty)
{
    __syncthreads();  // the previous exchange has been read
#pragma unroll
    for (int k = 0; k < 16; ++k) ex[(k * 16 + ty) * kWF + fl] = v[k];
    __syncthreads();
#pragma unroll
    for (int n = 0; n < 16; ++n) v[n] = ex[(ty * 16 + n) * kWF + fl];
    fftk::bfly16<SIGN>(v);
}

// Column F (0 .. M) of a packed row: its address, and the value of what is
// there (DC and Nyquist as reals).
__device__ __forceinline__ int col_of(int F, int M) { return F == M ? 0 : F; }
__device__ __forceinline__ float2 col_value(float2 x, int F, int M)
{
    if (F == 0) x.y = 0.f;
    if (F == M) x = make_float2(x.y, 0.f);
    return x;
}
__device__ __forceinline__ void store_col(float2* row, int F, int M, float2 x)
{
    if (F == 0) row[0].x = x.x;
    else if (F == M) row[0].y = x.x;
    else row[F] = x;
}

// Wire spectra are stored as the thread blocks use them: a tile of 16 columns
// of one group is [8][256 threads][2], thread (ty, fl)'s bins 16 k + ty of
// column fl for k = 2 j, 2 j + 1 at [j][thread]: eight 128-bit loads a thread.
__device__ __forceinline__ const float4* spec_at(const float2* Rw, int M, int g, int fblk)
{
    return reinterpret_cast<const float4*>(Rw) + ((size_t)g * wire_fblocks(M) + fblk) * (kWEx / 2) + threadIdx.x;
}

// One forward tile: columns fblk * 16 .. +15, outputs oblk * (256 - 2P) ...
// All kWThreads threads call it; sm holds kWConvSmem bytes, its twiddles
// loaded.  The rows of group g + 1 are copied into shared memory (16 bytes a
// copy) while group g is transformed; its wire spectra go straight to
// registers, asked for before the exchange.
__device__ __forceinline__ void conv_tile(const float2* __restrict__ Qh, const float2* __restrict__ Rw,
                                          float2* __restrict__ Vh, int G, int P, int nin, int nout, int M, int fblk,
                                          int oblk, float2* sm)
{
    const int tid = threadIdx.x;
    float2* ex = sm;
    float2* qs = sm + kWEx;  // [256 rows][16 columns]
    const float2* tw = sm + 2 * kWEx;
    const int fl = tid & (kWF - 1), ty = tid / kWF;
    const int F = fblk * kWF + fl;
    const bool edge = fblk == 0 || fblk * kWF + kWF > M;  // holds column 0 or M (or none): uniform
    const int ib = oblk * wire_valid(P) - 2 * P;          // input row of point 0
    const int crow = tid >> 3, ccol = fblk * kWF + 2 * (tid & 7);  // this thread's copies: rows crow + 32 j
    auto issue_q = [&](int g) {
        if (g < G) {
            const float2* src = Qh + ((size_t)g * nin + (ib + crow)) * M + ccol;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int i = ib + crow + 32 * j;
                const bool ok = i >= 0 && i < nin && ccol < M;
                cp_async16(qs + (crow + 32 * j) * kWF + 2 * (tid & 7), ok ? src + (size_t)(32 * j) * M : Qh,
                           ok ? 16 : 0);
            }
        }
        cp_async_commit();
    };
    float2 acc[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) acc[k] = make_float2(0.f, 0.f);
    __syncthreads();  // the previous tile of a persistent block is done with sm
    issue_q(0);
    for (int g = 0; g < G; ++g) {
        float2 v[16];
        cp_async_wait<0>();
        __syncthreads();  // every thread's rows of group g have landed, and the last exchange has been read
#pragma unroll
        for (int r = 0; r < 16; ++r) v[r] = qs[(ty + 16 * r) * kWF + fl];
        if (edge) {
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const int i = ib + ty + 16 * r;
                if (F == M && i >= 0 && i < nin) v[r] = __ldg(Qh + ((size_t)g * nin + i) * M);
                v[r] = col_value(v[r], F, M);
            }
        }
        fft256_a<-1>(v, tw, ty);
#pragma unroll
        for (int k = 0; k < 16; ++k) ex[(k * 16 + ty) * kWF + fl] = v[k];
        const float4* rp = spec_at(Rw, M, g, fblk);
        float4 rr[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) rr[j] = __ldg(rp + j * kWThreads);
        __syncthreads();
        issue_q(g + 1);  // every thread has taken group g's rows
#pragma unroll
        for (int n = 0; n < 16; ++n) v[n] = ex[(ty * 16 + n) * kWF + fl];
        fftk::bfly16<-1>(v);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            acc[2 * j].x = fmaf(rr[j].x, v[2 * j].x, fmaf(-rr[j].y, v[2 * j].y, acc[2 * j].x));
            acc[2 * j].y = fmaf(rr[j].x, v[2 * j].y, fmaf(rr[j].y, v[2 * j].x, acc[2 * j].y));
            acc[2 * j + 1].x = fmaf(rr[j].z, v[2 * j + 1].x, fmaf(-rr[j].w, v[2 * j + 1].y, acc[2 * j + 1].x));
            acc[2 * j + 1].y = fmaf(rr[j].z, v[2 * j + 1].y, fmaf(rr[j].w, v[2 * j + 1].x, acc[2 * j + 1].y));
        }
    }
    fft256_a<+1>(acc, tw, ty);
    fft256_b<+1>(acc, ex, fl, ty);
    if (F <= M) {
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            const int o = ib + ty + 16 * n;
            if (ty + 16 * n >= 2 * P && o < nout) store_col(Vh + (size_t)o * M, F, M, acc[n]);
        }
    }
}

// One adjoint tile: rows i = iblk * (256 - 2P) ... of dQ for every group, from
// nout rows of G: one transform forward, one back per group.  sm: kWAdjSmem.
__device__ __forceinline__ void adj_tile(const float2* __restrict__ Gh, const float2* __restrict__ Rw,
                                         float2* __restrict__ dQh, int G, int P, int nin, int nout, int M, int fblk,
                                         int iblk, float2* sm)
{
    const int tid = threadIdx.x;
    float2* ex = sm;
    const float2* tw = sm + kWEx;
    const int fl = tid & (kWF - 1), ty = tid / kWF;
    const int F = fblk * kWF + fl;
    const int i0 = iblk * wire_valid(P) + ty;
    float2 x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const int o = i0 + 16 * r;
        x[r] = F <= M && o < nout ? __ldg(Gh + (size_t)o * M + col_of(F, M)) : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int r = 0; r < 16; ++r) x[r] = col_value(x[r], F, M);
    fft256_a<-1>(x, tw, ty);
    fft256_b<-1>(x, ex, fl, ty);
    for (int g = 0; g < G; ++g) {
        const float4* rp = spec_at(Rw, M, g, fblk);
        float2 v[16];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float4 r = __ldg(rp + j * kWThreads);
            v[2 * j] = cmulc(x[2 * j], make_float2(r.x, r.y));
            v[2 * j + 1] = cmulc(x[2 * j + 1], make_float2(r.z, r.w));
        }
        fft256_a<+1>(v, tw, ty);
        fft256_b<+1>(v, ex, fl, ty);
        if (F <= M) {
            float2* dq = dQh + ((size_t)g * nin + i0) * M;
#pragma unroll
            for (int n = 0; n < 16; ++n) {
                if (ty + 16 * n < wire_valid(P) && i0 + 16 * n < nin)
                    store_col(dq + (size_t)(16 * n) * M, F, M, v[n]);
            }
        }
    }
}

// One table tile: the wire spectrum of group g's taps [2P + 1][M] (packed
// rows), scaled by the inverse transform's 1/256.  sm: kWAdjSmem.
__device__ __forceinline__ void spec_tile(const float2* __restrict__ taps, float2* __restrict__ Rw, int P, int M,
                                          int fblk, int g, float2* sm)
{
    const float2* tw = sm + kWEx;
    const int fl = threadIdx.x & (kWF - 1), ty = threadIdx.x / kWF;
    const int F = fblk * kWF + fl;
    const int nt = 2 * P + 1;
    float2 v[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const int j = ty + 16 * r;
        v[r] = F <= M && j < nt ? col_value(__ldg(taps + ((size_t)g * nt + j) * M + col_of(F, M)), F, M)
                                : make_float2(0.f, 0.f);
    }
    fft256_a<-1>(v, tw, ty);
    fft256_b<-1>(v, sm, fl, ty);
    float4* w = const_cast<float4*>(spec_at(Rw, M, g, fblk));
    const float sc = 1.0f / kWL;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        w[j * kWThreads] = make_float4(v[2 * j].x * sc, v[2 * j].y * sc, v[2 * j + 1].x * sc, v[2 * j + 1].y * sc);
}

}  // namespace wfft
}  // namespace wctb200
