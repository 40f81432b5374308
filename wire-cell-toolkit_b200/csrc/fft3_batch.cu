// Row transforms of batched events in three register stages (fft3.cuh): a launch
// per length class.
#include <algorithm>

#include "fft3.cuh"
#include "kernels.cuh"

namespace wctb200 {

// ---------------------------------------------------------------------------
// Batched events: the rows of every (event, plane) whose time-FFT length is
// class cls, dealt over persistent blocks.  s_pre: the entries' row prefixes
// (zero rows for entries of other classes), built once per block.
// ---------------------------------------------------------------------------
template <bool INV>
__device__ __forceinline__ int class_rows(const BatchPlan* __restrict__ plan, const BatchStatic& bs, int cls,
                                          int* s_pre)
{
    const int ne = plan->nev * plan->np;
    for (int k = threadIdx.x; k < ne; k += blockDim.x) {
        const EvPlane& E = plan->ep[k];
        s_pre[k] = E.cls != cls || !E.nin ? 0 : (INV ? E.nout : bs.pl[k % plan->np].G * E.nin);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        int carry = 0;
        for (int b = 0; b < ne; b += 32) {
            const int k = b + threadIdx.x;
            const int n = k < ne ? s_pre[k] : 0;
            int x = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if ((int)threadIdx.x >= o) x += y;
            }
            if (k < ne) s_pre[k] = carry + x - n;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
        if (threadIdx.x == 0) s_pre[ne] = carry;
    }
    __syncthreads();
    return s_pre[ne];
}

// The last entry k in [0, n) with pre[k] <= item.
__device__ __forceinline__ int entry_of(const int* pre, int n, int item)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pre[mid] <= item) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

template <class P>
__global__ void __launch_bounds__(RfftShape<P>::kThreads, RfftShape<P>::kBlocks)
    k_rfft3_batch(const BatchPlan* __restrict__ plan, BatchStatic bs, int cls, float* Q,
                  const int* __restrict__ wire_cnt, const float2* __restrict__ t3, const float2* __restrict__ twh)
{
    extern __shared__ __align__(16) float2 f3sm[];
    __shared__ int s_pre[kMaxBatch * kMaxPlanes + 1];
    if (plan->status & kBatchSkip) return;
    const int tid = threadIdx.x;
    const int ne = plan->nev * plan->np, total = class_rows<false>(plan, bs, cls, s_pre);
    __shared__ int s_cnt[2][kMaxRowTiles];
    int row = blockIdx.x;
    if (row >= total) return;
    // visit counts of row r's tiles; its address and the offset of its first column in its first tile
    auto ask = [&](int buf, int r, float*& x, int& off) {
        if (r >= total) return;
        const int k = entry_of(s_pre, ne, r), e = k / plan->np, ip = k - e * plan->np;
        const EvPlane& E = plan->ep[k];
        const int rel = r - s_pre[k];
        const TileMap t{wire_cnt + (size_t)e * bs.nkeys + (size_t)bs.pl[ip].wire_base * bs.ntiles, bs.pl[ip].nwires,
                        bs.ntiles, E.start_ch, E.nin, E.start_tick, E.ktile0, E.ntile};
        fft3::ask_counts(s_cnt[buf], t, E.start_ch + rel % E.nin, tid);
        x = Q + E.qoff + (size_t)rel * (2 * P::M);
        off = E.start_tick - E.ktile0 * kTile;
    };
    float *x = nullptr, *xn = nullptr;
    int off = 0, offn = 0;
    ask(0, row, x, off);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    ask(1, row + gridDim.x, xn, offn);
    fft3::copy_tiles<P::M>(f3sm, x, s_cnt[0], off, tid, RfftShape<P>::kThreads);
    for (int buf = 0; row < total; row += gridDim.x, buf ^= 1) {
        cp_async_wait<0>();
        __syncthreads();
        const int next = row + gridDim.x;
        float* xnn = nullptr;
        rfft3_row<P>(f3sm, f3sm + P::M, reinterpret_cast<float2*>(x), t3, twh, tid, [&] {
            if (next >= total) return;
            const int o = offn;
            ask(buf, next + gridDim.x, xnn, offn);
            fft3::copy_tiles<P::M>(f3sm, xn, s_cnt[buf ^ 1], o, tid, RfftShape<P>::kThreads);
        });
        x = xn;
        xn = xnn;
    }
}

template <class P>
__global__ void __launch_bounds__(IrfftShape<P>::kThreads, IrfftShape<P>::kBlocks)
    k_irfft3_batch(const BatchPlan* __restrict__ plan, BatchStatic bs, int cls, const float2* __restrict__ V,
                   float* __restrict__ frames, long long fstride, const unsigned char* __restrict__ row_flag,
                   const float2* __restrict__ t3, const float2* __restrict__ twh)
{
    extern __shared__ __align__(16) float2 f3sm[];
    __shared__ int s_pre[kMaxBatch * kMaxPlanes + 1];
    if (plan->status & kBatchSkip) return;
    const int tid = threadIdx.x;
    const int np = plan->np, ne = plan->nev * np, total = class_rows<true>(plan, bs, cls, s_pre);
    // the next row from `row` on that is a frame wire within reach of charge (total: none); its entry in k
    auto seek = [&](int row, int& k) {
        for (; row < total; row += gridDim.x) {
            k = entry_of(s_pre, ne, row);
            const EvPlane& E = plan->ep[k];
            const int e = k / np;
            const BatchPlaneStatic& pl = bs.pl[k - e * np];
            const int W = E.start_ch - pl.npad + (row - s_pre[k]);
            if (W < max(0, E.m_start_ch) || W >= min(pl.nwires, E.m_end_ch)) continue;
            if (row_reached(row_flag + (size_t)e * bs.nwires_total + pl.wire_base, pl.nwires, W, pl.npad)) break;
        }
        return row;
    };
    auto src = [&](int row, int k) { return V + plan->ep[k].voff + (size_t)(row - s_pre[k]) * P::M; };
    int k = 0, row = seek(blockIdx.x, k);
    if (row < total)
        fft3::copy_row<P::M>(f3sm, reinterpret_cast<const float*>(src(row, k)), 2 * P::M, tid,
                             IrfftShape<P>::kThreads);
    while (row < total) {
        int kn = k;
        const int next = seek(row + gridDim.x, kn);
        const EvPlane& E = plan->ep[k];
        const int e = k / np;
        const BatchPlaneStatic& pl = bs.pl[k - e * np];
        const int W = E.start_ch - pl.npad + (row - s_pre[k]), tick0 = E.start_tick;
        float* f = frames + (size_t)e * fstride + (size_t)(pl.row0 + W) * bs.nticks;
        const bool vec = ((tick0 | bs.nticks) & 1) == 0 && (reinterpret_cast<uintptr_t>(f) & 7) == 0;
        cp_async_wait<0>();
        __syncthreads();
        irfft3_row<P>(f3sm, f3sm + P::M, f, tick0, min(E.N, E.nt_ref), bs.nticks, vec, t3, twh, tid, next < total,
                      next < total ? src(next, kn) : V);
        row = next;
        k = kn;
    }
}

template <class P, class I>
static bool go_batch_ready(int* blocks)
{
    static std::atomic<int> cf[kFft3Devices], ci[kFft3Devices];
    blocks[0] = persistent_blocks((const void*)k_rfft3_batch<P>, RfftShape<P>::kThreads, P::kSmem, cf);
    blocks[1] = persistent_blocks((const void*)k_irfft3_batch<I>, IrfftShape<I>::kThreads, I::kSmem, ci);
    return blocks[0] > 0 && blocks[1] > 0;
}

bool fft3_batch_blocks(int M, int* blocks)
{
    switch (M) {
#define X(A, B, C) WCT_CASE(A, B, C, return go_batch_ready<P, I>(blocks))
        WCT_FFT3_PLANS(X)
#undef X
        default: return false;
    }
}

void launch_rfft3_batch(const BatchPlan* plan, const BatchStatic& bs, int cls, const FftDesc& d, int nblocks,
                        float* Q, const int* wire_cnt, cudaStream_t s)
{
    switch (d.M) {
#define X(A, B, C)                                                                                     \
    WCT_CASE(A, B, C,                                                                                  \
             k_rfft3_batch<P><<<nblocks, RfftShape<P>::kThreads, P::kSmem, s>>>(plan, bs, cls, Q, wire_cnt, d.t3f, d.twh); \
             return)
        WCT_FFT3_PLANS(X)
#undef X
    }
}

void launch_irfft3_batch(const BatchPlan* plan, const BatchStatic& bs, int cls, const FftDesc& d, int nblocks,
                         const float2* V, float* frames, long long fstride, const unsigned char* row_flag,
                         cudaStream_t s)
{
    switch (d.M) {
#define X(A, B, C)                                                                                     \
    WCT_CASE(A, B, C,                                                                                  \
             k_irfft3_batch<I><<<nblocks, IrfftShape<I>::kThreads, I::kSmem, s>>>(plan, bs, cls, V, frames, fstride, \
                                                                                 row_flag, d.t3i, d.twh);      \
             return)
        WCT_FFT3_PLANS(X)
#undef X
    }
}

}  // namespace wctb200
