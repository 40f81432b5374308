// Real row transforms in three register stages (fft3.cuh): kernels and launchers.
#include <algorithm>

#include "fft3.cuh"
#include "kernels.cuh"

namespace wctb200 {

template <class P>
__global__ void __launch_bounds__(RfftShape<P>::kThreads, RfftShape<P>::kBlocks) k_rfft3(const float* in, long in_ld, int in_len,
                                                                  float2* out, long out_ld, int nrows, TileMap tiles,
                                                                  const float2* __restrict__ t3,
                                                                  const float2* __restrict__ twh)
{
    extern __shared__ __align__(16) float2 f3sm[];
    __shared__ int s_cnt[2][kMaxRowTiles];  // a sparse grid's counts, a row ahead of its copy
    const int tid = threadIdx.x;
    const bool sparse = tiles.cnt != nullptr;
    const int off = tiles.col0 - tiles.ktile0 * kTile;
    int row = blockIdx.x;
    if (row >= nrows) return;
    auto counts = [&](int buf, int r) {
        if (sparse && r < nrows) fft3::ask_counts(s_cnt[buf], tiles, tiles.start_ch + r % tiles.nin, tid);
    };
    auto copy = [&](int buf, int r) {
        const float* x = in + (size_t)r * in_ld;
        if (sparse) fft3::copy_tiles<P::M>(f3sm, x, s_cnt[buf], off, tid, RfftShape<P>::kThreads);
        else fft3::copy_row<P::M>(f3sm, x, in_len, tid, RfftShape<P>::kThreads);
    };
    if (sparse) {
        counts(0, row);
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
    }
    counts(1, row + gridDim.x);
    copy(0, row);
    for (int buf = 0; row < nrows; row += gridDim.x, buf ^= 1) {
        cp_async_wait<0>();
        __syncthreads();
        const int next = row + gridDim.x;
        rfft3_row<P>(f3sm, f3sm + P::M, out + (size_t)row * out_ld, t3, twh, tid, [&] {
            if (next >= nrows) return;
            counts(buf, next + gridDim.x);
            copy(buf ^ 1, next);
        });
    }
}

template <class P>
__global__ void __launch_bounds__(IrfftShape<P>::kThreads, IrfftShape<P>::kBlocks) k_irfft3(const float2* Vh, int r0, int r1, int wire0,
                                                                    int tick0, int ncols, int nticks, float* frame,
                                                                    const float2* __restrict__ t3,
                                                                    const float2* __restrict__ twh,
                                                                    const unsigned char* __restrict__ row_flag,
                                                                    int nwires, int npad)
{
    extern __shared__ __align__(16) float2 f3sm[];
    const int tid = threadIdx.x;
    // 8-byte stores: even first tick and row length on an aligned frame (uniform)
    const bool vec = ((tick0 | nticks) & 1) == 0 && (reinterpret_cast<uintptr_t>(frame) & 7) == 0;
    auto live = [&](int row) { return !row_flag || row_reached(row_flag, nwires, wire0 + row, npad); };
    int row = r0 + blockIdx.x;
    while (row < r1 && !live(row)) row += gridDim.x;
    if (row < r1)
        fft3::copy_row<P::M>(f3sm, reinterpret_cast<const float*>(Vh + (size_t)row * P::M), 2 * P::M, tid,
                             IrfftShape<P>::kThreads);
    while (row < r1) {
        int next = row + gridDim.x;
        while (next < r1 && !live(next)) next += gridDim.x;
        cp_async_wait<0>();
        __syncthreads();
        irfft3_row<P>(f3sm, f3sm + P::M, frame + (size_t)(wire0 + row) * nticks, tick0, ncols, nticks, vec, t3, twh,
                      tid, next < r1, Vh + (size_t)next * P::M);
        row = next;
    }
}

template <class P>
static bool go_rfft3(const float* in, long in_ld, int in_len, float2* out, long out_ld, int nrows, const FftDesc& d,
                     const TileMap& tiles, cudaStream_t s)
{
    static std::atomic<int> cache[kFft3Devices];
    const int nb = persistent_blocks((const void*)k_rfft3<P>, RfftShape<P>::kThreads, P::kSmem, cache);
    if (nb <= 0) return false;
    if (nrows > 0)
        k_rfft3<P><<<std::min(nrows, nb), RfftShape<P>::kThreads, P::kSmem, s>>>(in, in_ld, in_len, out, out_ld, nrows,
                                                                                tiles, d.t3f, d.twh);
    return true;
}

template <class P>
static bool go_irfft3(const float2* Vh, int r0, int r1, const FftDesc& d, int wire0, int tick0, int ncols, int nticks,
                      float* frame, const unsigned char* row_flag, int nwires, int npad, cudaStream_t s)
{
    static std::atomic<int> cache[kFft3Devices];
    const int nb = persistent_blocks((const void*)k_irfft3<P>, IrfftShape<P>::kThreads, P::kSmem, cache);
    if (nb <= 0) return false;
    k_irfft3<P><<<std::min(r1 - r0, nb), IrfftShape<P>::kThreads, P::kSmem, s>>>(
        Vh, r0, r1, wire0, tick0, ncols, nticks, frame, d.t3i, d.twh, row_flag, nwires, npad);
    return true;
}

bool fft3_radices(int M, int* r)
{
    switch (M) {
#define X(A, B, C) case A * B * C: r[0] = A, r[1] = B, r[2] = C; return true;
        WCT_FFT3_PLANS(X)
#undef X
        default: return false;
    }
}

int fft3_next(int M)
{
    int best = 0;
#define X(A, B, C) \
    if (A * B * C >= M && (!best || A * B * C < best)) best = A * B * C;
    WCT_FFT3_PLANS(X)
#undef X
    return best;
}

bool launch_rfft3(const float* in, long in_ld, int in_len, float2* out, long out_ld, int nrows, const FftDesc& d,
                  const TileMap& tiles, cudaStream_t s)
{
    // whole 16-byte pieces of every row
    if (!d.t3f || (reinterpret_cast<uintptr_t>(in) & 15) || in_ld % 4) return false;
    switch (d.M) {
#define X(A, B, C) WCT_CASE(A, B, C, return go_rfft3<P>(in, in_ld, in_len, out, out_ld, nrows, d, tiles, s))
        WCT_FFT3_PLANS(X)
#undef X
        default: return false;
    }
}

bool rfft3_takes(const float* in, long in_ld, const FftDesc& d)
{
    return launch_rfft3(in, in_ld, 0, nullptr, 0, 0, d, TileMap{}, nullptr);
}

bool launch_irfft3(const float2* Vh, int r0, int r1, const FftDesc& d, int wire0, int tick0, int ncols, int nticks,
                   float* frame, const unsigned char* row_flag, int nwires, int npad, cudaStream_t s)
{
    if (!d.t3i || (reinterpret_cast<uintptr_t>(Vh) & 15) || d.M % 2) return false;
    switch (d.M) {
#define X(A, B, C) \
    WCT_CASE(A, B, C, return go_irfft3<I>(Vh, r0, r1, d, wire0, tick0, ncols, nticks, frame, row_flag, nwires, npad, s))
        WCT_FFT3_PLANS(X)
#undef X
        default: return false;
    }
}

}  // namespace wctb200
