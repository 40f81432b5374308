// Complex row transforms in three register stages (fft3.cuh).
#include <algorithm>

#include "fft3.cuh"
#include "kernels.cuh"

namespace wctb200 {

// ---------------------------------------------------------------------------
// Complex rows, out = scale * DFT_SIGN(in), in place allowed.
// ---------------------------------------------------------------------------
template <class P>
struct CfftShape {
    static constexpr int kThreads = P::threads(P::N1, P::N2, P::NS);
};

template <class P, int SIGN>
__global__ void __launch_bounds__(CfftShape<P>::kThreads) k_cfft3(const float2* in, long ld_in, float2* out,
                                                                  long ld_out, int nrows, float scale,
                                                                  const float2* __restrict__ t3)
{
    extern __shared__ __align__(16) float2 f3sm[];
    const int tid = threadIdx.x, nth = CfftShape<P>::kThreads;
    float2* e1 = f3sm + P::M;
    float2* e2 = P::kShare ? e1 : e1 + P::E1;
    int row = blockIdx.x;
    auto fetch = [&](int r) {
        fft3::copy_row<P::M>(f3sm, reinterpret_cast<const float*>(in + (size_t)r * ld_in), 2 * P::M, tid, nth);
    };
    if (row < nrows) fetch(row);
    for (; row < nrows; row += gridDim.x) {
        cp_async_wait<0>();
        __syncthreads();
        if (tid < P::N1) {
            float2 v[P::R1];
#pragma unroll
            for (int r = 0; r < P::R1; ++r) v[r] = f3sm[tid + r * P::N1];
            fftk::bfly<P::R1, SIGN>(v);
#pragma unroll
            for (int r = 0; r < P::R1; ++r) e1[r * P::S1 + tid] = v[r];
        }
        __syncthreads();
        if (row + (int)gridDim.x < nrows) fetch(row + gridDim.x);
        fft3::stage2<P, SIGN>(e1, e2, t3, tid);
        __syncthreads();
        if (tid < P::NS) {
            float2 v[P::R3];
            fft3::stage3<P, SIGN>(e2, t3 + P::T2, tid, v);
            float2* o = out + (size_t)row * ld_out;
#pragma unroll
            for (int r = 0; r < P::R3; ++r) o[tid + r * P::NS] = cscale(v[r], scale);
        }
    }
}

template <class P, int SIGN>
static bool go_cfft3(const float2* in, long ld_in, float2* out, long ld_out, int nrows, float scale, const float2* t3,
                     cudaStream_t s)
{
    static std::atomic<int> cache[kFft3Devices];
    const int nb = persistent_blocks((const void*)k_cfft3<P, SIGN>, CfftShape<P>::kThreads, P::kSmem, cache);
    if (nb <= 0) return false;
    k_cfft3<P, SIGN><<<std::min(nrows, nb), CfftShape<P>::kThreads, P::kSmem, s>>>(in, ld_in, out, ld_out, nrows,
                                                                                  scale, t3);
    return true;
}

bool launch_cfft3(const float2* in, long ld_in, float2* out, long ld_out, int nrows, const FftDesc& d, int sign,
                  float scale, cudaStream_t s)
{
    if (!d.t3f || (reinterpret_cast<uintptr_t>(in) & 15) || ld_in % 2) return false;
    switch (d.M) {
#define X(A, B, C)                                                                                     \
    WCT_CASE(A, B, C,                                                                                  \
             return sign < 0 ? go_cfft3<P, -1>(in, ld_in, out, ld_out, nrows, scale, d.t3f, s)         \
                             : go_cfft3<P, +1>(in, ld_in, out, ld_out, nrows, scale, d.t3f, s))
        WCT_FFT3_PLANS(X)
#undef X
        default: return false;
    }
}

}  // namespace wctb200
