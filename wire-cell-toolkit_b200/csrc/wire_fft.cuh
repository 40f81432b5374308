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
// Rounding: a transform spreads the rounding of a block's strong rows evenly over
// all 256, about 1e-7 of the block's rms a row, where the direct sum's stays with
// the wires within P.  So each tile also leaves the energy of its 256 rows, and
// rows with under a ninth of the block's mean energy (or where that is not
// finite) are convolved again directly (pick_tile below): wires beside a
// bright one keep their own precision, and a NaN stays within P wires.
//
// Bin 0 of a packed row holds two real spectra (DC and Nyquist).  The DC
// value is column 0 here and the Nyquist value column M, each real with
// its own (real-tap) wire spectrum, so no bin needs a special product.
#pragma once

#include <cmath>

#include "fft.cuh"
#include "kernels.cuh"

namespace wctb200 {

constexpr int kWL = 256;          // wires per transform (16 x 16)
constexpr int kWF = 16;           // frequencies per block
constexpr int kWThreads = 256;    // kWF x 16
constexpr int kWEx = kWL * kWF;   // complex values of one exchange buffer
// shared memory: the exchange buffer (and the tile of grid rows), the twiddles
constexpr size_t kWConvSmem = sizeof(float2) * (2 * kWEx + kWL);
constexpr size_t kWAdjSmem = sizeof(float2) * (kWEx + kWL);
constexpr int kPickThreads = 4 * kWL;
constexpr int kConvGroups = 16;  // groups of eight rows in a chunk's window: forward, adjoint
constexpr int kAdjGroups = 8;
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

// Energies of a tile's rows are kept as [thread]: thread ty * 16 + fl holds point ty + 16 fl.
__device__ __forceinline__ int energy_point(int t) { return t / kWF + 16 * (t & (kWF - 1)); }

// Sums over the 16 lanes of a half warp that hold a row's columns: lane fl
// returns the sum of e[fl] (the other half of the values goes to the lane across).
template <typename T>
__device__ __forceinline__ T row_sums(T* e, int fl)
{
#pragma unroll
    for (int h = 8; h; h >>= 1) {
        const bool up = fl & h;
#pragma unroll
        for (int j = 0; j < h; ++j) {
            const T keep = up ? e[j + h] : e[j], give = up ? e[j] : e[j + h];
            e[j] = keep + __shfl_xor_sync(0xffffffffu, give, h);
        }
    }
    return e[0];
}

// One forward tile: columns fblk * 16 .. +15, outputs oblk * (256 - 2P) ...
// All kWThreads threads call it; sm holds kWConvSmem bytes, its twiddles
// loaded.  The rows of group g + 1 are copied into shared memory (16 bytes a
// copy) while group g is transformed; its wire spectra go straight to
// registers, asked for before the exchange.  energy: of the tile's 256 rows.
__device__ __forceinline__ void conv_tile(const float2* __restrict__ Qh, const float2* __restrict__ Rw,
                                          float2* __restrict__ Vh, int G, int P, int nin, int nout, int M, int fblk,
                                          int oblk, double* __restrict__ energy, float2* sm)
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
    double e[16];  // (columns past M are zero)
#pragma unroll
    for (int n = 0; n < 16; ++n) e[n] = (double)acc[n].x * (double)acc[n].x + (double)acc[n].y * (double)acc[n].y;
    energy[tid] = row_sums(e, fl);
}

// One adjoint tile: rows i = iblk * (256 - 2P) ... of dQ for every group, from
// nout rows of G: one transform forward, one back per group.  energy: of the
// tile's 256 rows, over the groups.  sm: kWAdjSmem.
__device__ __forceinline__ void adj_tile(const float2* __restrict__ Gh, const float2* __restrict__ Rw,
                                         float2* __restrict__ dQh, int G, int P, int nin, int nout, int M, int fblk,
                                         int iblk, double* __restrict__ energy, float2* sm)
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
    // a power of two that brings the tile's gradients near 2^40, so that squares of their
    // products with the responses neither vanish nor overflow
    __shared__ unsigned s_top[kWThreads / 32];
    unsigned top = 0;
#pragma unroll
    for (int r = 0; r < 16; ++r) top = max(top, max(__float_as_uint(fabsf(x[r].x)), __float_as_uint(fabsf(x[r].y))));
    top = __reduce_max_sync(0xffffffffu, top);
    if ((tid & 31) == 0) s_top[tid >> 5] = top;
    fft256_a<-1>(x, tw, ty);
    fft256_b<-1>(x, ex, fl, ty);  // (its barriers stand between s_top's writes and reads)
#pragma unroll
    for (int k = 0; k < kWThreads / 32; ++k) top = max(top, s_top[k]);
    const int expo = min(max((int)(top >> 23), 42), 253);
    const float sc = __uint_as_float((unsigned)(254 + 40 - expo) << 23);  // 2^(40 + 127 - expo), at most 2^125
    float es = 0.f;
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
        float e[16];
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            const float a = v[n].x * sc, b = v[n].y * sc;
            e[n] = a * a + b * b;
        }
        es += row_sums(e, fl);
    }
    const double back = 1.0 / (double)sc;
    energy[tid] = (double)es * back * back;
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

// ---------------------------------------------------------------------------
// Rows whose energy is under a ninth of their block's mean: picked here, convolved
// directly by conv2_chunk (kernels.cu) and adj_ways (adjoint.cu).
//
// kFaintEnergy: a row's rms at a third of its block's. The rounding that reaches a
// row, in 1e-7 of the row itself against 64 bits (full APA, 20k track depos; by
// rms around the row / rms of the row): 1 to 2: 2.2, worst 3.0 in overlap-save
// blocks; 2 to 4: 2.9, worst 8.1; 4 to 8: 9; 8 to 16: 19; over 64: 4500.  The
// direct sum: 1.6 throughout, worst 2.6 (3.8 and 5.1 before the blocks).
//
// What it costs, and why this form: a launch that adds up the energies (9 us, a
// block per 256 wires) and one that takes the list.  Rows are few on tracks (3 %
// of a full APA's) and up to two thirds of a plane's around showers, where the
// direct kernel's time a row decides, so the list keeps the shape of its blocks:
// windows of sixteen groups of eight rows, staged once (one warp a group from L2:
// 348 us against 146 for the three planes of 200k shower depos).  Events without
// -> with this, us: plane 2k 267 -> 282, full APA on tracks 20k 487 -> 528, 520k
// 965 -> 1003, shower 200k 1624 -> 1715, fit step 20k 1409 -> 1496; 16 batched
// events 4.25 -> 5.33 ms a call, 64 of 500-5000 depos 9.2 -> 12.4.
// ---------------------------------------------------------------------------
constexpr double kFaintEnergy = 9.0;

// Block blk's rows that are faint and wanted into the list, as groups of eight,
// those of a window of neighbouring groups a chunk (the kernels that take them
// stage the window's input rows).  energy: [nfb][256] of the block, an eighth of
// the columns per 128 threads, added in a fixed order; null: every wanted row.
template <bool ADJ>
__device__ __forceinline__ void pick_tile(const double* __restrict__ energy, int nfb, int P, int blk, int n,
                                          const WantRows& want, int entry, const RowList& list)
{
    __shared__ double2 s_e[8][kWL / 2];
    __shared__ double s_w[kWL / 32];
    __shared__ unsigned char s_f[kWL], s_want[4][kWL + 2 * kWMaxPad];
    const int t = threadIdx.x & (kWL - 1), q = threadIdx.x / kWL;
    const int base = blk * wire_valid(P), p0 = ADJ ? 0 : 2 * P;  // first row, its point
    // forward: the flags of wires base .. of the block's rows and P on either side; adjoint: a
    // quarter of the tiles of each row's wire
    if (ADJ) {
        const int W = want.wire0 + base + t;
        int any = 0;
        if (W >= 0 && W < want.nwires)
            for (int k = q; k < want.ntiles; k += 4) any |= want.cnt[(size_t)W * want.ntiles + k];
        s_want[q][t] = any != 0;
    }
    else if (threadIdx.x < wire_valid(P) + 2 * P) {
        const int W = want.wire0 + base - P + (int)threadIdx.x;
        s_want[0][threadIdx.x] = W >= 0 && W < want.nwires ? want.flag[W] : 0;
    }
    const bool every = energy == nullptr;  // no blocks: all wanted rows
    double e = 0.0;
    if (!every) {
        const int h = threadIdx.x & (kWL / 2 - 1), part = threadIdx.x / (kWL / 2);
        const double2* at = reinterpret_cast<const double2*>(energy) + h;
        const int f1 = nfb * (part + 1) / 8;
        double2 v = make_double2(0.0, 0.0);
        for (int f = nfb * part / 8; f < f1; f += 8) {
            double2 x[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                x[k] = f + k < f1 ? at[(size_t)(f + k) * (kWL / 2)] : make_double2(0.0, 0.0);
#pragma unroll
            for (int k = 0; k < 8; ++k) v = make_double2(v.x + x[k].x, v.y + x[k].y);
        }
        s_e[part][h] = v;
    }
    __syncthreads();
    if (q == 0 && !every) {
        const double* s = reinterpret_cast<const double*>(s_e) + t;
#pragma unroll
        for (int k = 0; k < 8; ++k) e += s[k * kWL];
        double m = e;
#pragma unroll
        for (int o = 16; o; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
        if ((t & 31) == 0) s_w[t >> 5] = m;
    }
    __syncthreads();
    if (q == 0) {
        double mean = INFINITY;
        if (!every) {
            mean = 0.0;
#pragma unroll
            for (int k = 0; k < kWL / 32; ++k) mean += s_w[k];
            mean *= 1.0 / kWL;
        }
        const int p = energy_point(t), r = p - p0, W = want.wire0 + base + r;
        // (a NaN in either, or an infinite mean: faint)
        bool faint = r >= 0 && r < wire_valid(P) && base + r < n && W >= want.wlo && W < want.whi &&
                     !(kFaintEnergy * e >= mean && mean < INFINITY);
        if (faint) {
            int any = 0;
            if (ADJ) any = s_want[0][r] | s_want[1][r] | s_want[2][r] | s_want[3][r];
            else {
#pragma unroll 1
                for (int k = 0; k <= 2 * P; ++k) any |= s_want[0][r + k];
            }
            faint = any;
        }
        s_f[p] = faint;
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // at most 32 groups
        const int g = threadIdx.x;
        int mask = 0;
#pragma unroll 1
        for (int r = 0; r < 8 && 8 * g + r < wire_valid(P); ++r) mask |= s_f[p0 + 8 * g + r] << r;
        const unsigned on = __ballot_sync(0xffffffffu, mask != 0);
        int at = 0;
        if (g == 0 && on) at = atomicAdd(list.count, __popc(on));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (mask) list.item[at + __popc(on & ((1u << g) - 1))] = make_int2(base + 8 * g, mask);
        constexpr int kWindow = ADJ ? kAdjGroups : kConvGroups;
        const unsigned here = g * kWindow < 32 ? on >> (g * kWindow) & ((1u << kWindow) - 1) : 0u;
        if (here)
            list.chunk[atomicAdd(list.count + 1, 1)] =
                make_int4(at + __popc(on & ((1u << (g * kWindow)) - 1)), __popc(here), entry,
                          8 * (32 - __clz(here) - (__ffs(here) - 1)));
    }
}

}  // namespace wfft
}  // namespace wctb200
