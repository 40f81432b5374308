// Kernels and launchers of the overlap-save wire convolution (wire_fft.cuh).
#include "kernels.cuh"
#include "wire_fft.cuh"

namespace wctb200 {

__global__ void __launch_bounds__(kWThreads, 2) k_wire_conv_fft(const float2* __restrict__ Qh,
                                                                const float2* __restrict__ Rw,
                                                                float2* __restrict__ Vh, int G, int P, int nin,
                                                                int nout, int M, double* __restrict__ energy)
{
    extern __shared__ float2 wsm[];
    wfft::load_twiddles(wsm + 2 * kWEx, threadIdx.x);
    __syncthreads();
    wfft::conv_tile(Qh, Rw, Vh, G, P, nin, nout, M, blockIdx.x, blockIdx.y,
                    energy + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * kWL, wsm);
}

__global__ void __launch_bounds__(kWThreads, 2) k_wire_adj_fft(const float2* __restrict__ Gh,
                                                               const float2* __restrict__ Rw,
                                                               float2* __restrict__ dQh, int G, int P, int nin,
                                                               int nout, int M, double* __restrict__ energy)
{
    extern __shared__ float2 wsm[];
    wfft::load_twiddles(wsm + kWEx, threadIdx.x);
    __syncthreads();
    wfft::adj_tile(Gh, Rw, dQh, G, P, nin, nout, M, blockIdx.x, blockIdx.y,
                   energy + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * kWL, wsm);
}

template <bool ADJ>
__global__ void __launch_bounds__(kPickThreads) k_wire_pick(const double* __restrict__ energy, int nfb, int P, int n,
                                                            WantRows want, RowList list)
{
    wfft::pick_tile<ADJ>(energy ? energy + (size_t)blockIdx.x * nfb * kWL : nullptr, nfb, P, blockIdx.x, n, want, 0, list);
}

__global__ void __launch_bounds__(kWThreads) k_wire_spec(const float2* __restrict__ taps, float2* __restrict__ Rw,
                                                         int P, int M)
{
    extern __shared__ float2 wsm[];
    wfft::load_twiddles(wsm + kWEx, threadIdx.x);
    __syncthreads();
    wfft::spec_tile(taps, Rw, P, M, blockIdx.x, blockIdx.y, wsm);
}

size_t wire_spec_count(int G, int M) { return (size_t)G * wire_fblocks(M) * kWEx; }

bool wire_fft_fits(int G, int npad, int M)
{
    return npad <= kWMaxPad && M % 2 == 0 && wire_spec_count(G, M) <= kWMaxSpec;
}

// The forms of an event's wire convolution.  The blocks' time goes by 256 - 2P rows,
// that of the direct kernels and of the listed rows by G (2P + 1) a row.  Kernels
// alone, direct / blocks with a few faint rows, us (11 groups, M = 1600, inputs not
// in L2):
//   P = 21: one tile of 128 rows 31 / 39, 170 charge wires 54 / 56, 240 78 / 61,
//           960 150 / 99 (M = 3200: 54 / 52, 80 / 75, 125 / 104, 269 / 172);
//   P = 10: 23 / 40, 47 / 54 (240), 86 / 91 (960; M = 3200: 150 / 158);
//   P = 1 39 / 39, 43 / 46, 64 / 86; P = 0 31 / 39, 45 / 85; other pads have no
//           direct kernel of their own: P = 16 269 / 40, 539 / 102.
bool wire_lists(int npad) { return npad >= 2 && npad != 10 && npad <= kWMaxPad; }
bool wire_blocks_pay(int npad) { return wire_lists(npad) && npad > 5; }
// Where few rows or little charge make the blocks, they leave most rows faint and
// both forms are paid: events in us, rows listed at once / blocks (5000 point depos
// on W wires unless given; M = 950 at 2000 ticks, 1792 at 6000):
//   few visits a row, 960 wires: 0.3 366 / 426, 0.8 382 / 376, 2 386 / 323 (P = 16);
//   few rows (the blocks pad them to 256): P = 16 W = 100 151 / 165 and 178 / 180, 230
//     179 / 187 and 210 / 207, 500 223 / 209 and 277 / 267; P = 64 W = 40 246 / 299,
//     230 307 / 295;
//   few taps: P = 5 W = 100 150 / 172, 500 224 / 254, 940 305 / 313; P = 2 W = 300
//     179 / 204, 940 283 / 315.
// P = 21 has a direct kernel, 16 columns x 128 rows a block, which is the faster one
// while all its blocks are resident at once: direct / blocks W = 190 169 / 182 and 188 /
// 201, 300 181 / 193 and (two waves) 227 / 225, 400 211 / 199 and 263 / 257; full APA,
// 1500 depos in showers on 200 wires a plane 279 / 324; visits a row 0.3 346 / 441, 0.8
// 364 / 382, 2 370 / 315.
WireForm wire_form(int npad, int nout, int M, long long visits, long long rows, bool have_spectra)
{
    if (!wire_lists(npad)) return WireForm::Direct;
    const bool few = !have_spectra || visits < rows;
    if (npad == 21) return few || ((M + 15) / 16) * ((nout + 127) / 128) <= 2 * 148 ? WireForm::Direct : WireForm::Blocks;
    return few || nout <= kWL ? WireForm::Listed : WireForm::Blocks;
}
// The adjoint, a transform back per group: P = 21: two tiles of 64 46 / 48, 170
// wires 74 / 52, 960 197 / 101; P = 16: 37 / 48, 60 / 52, 160 / 103; P = 10: 46 /
// 52 (170), 78 / 86 (600), 113 / 102 (960); P = 30, 40 wires: 54 / 46.
bool wire_adj_fft_pays(int npad, int nin) { return npad > 21 || (npad >= 16 && nin > 128); }

void launch_wire_spec(const float2* taps, float2* Rw, int G, int npad, int M, cudaStream_t s)
{
    cudaFuncSetAttribute((const void*)k_wire_spec, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWAdjSmem);
    k_wire_spec<<<dim3(wire_fblocks(M), G), kWThreads, kWAdjSmem, s>>>(taps, Rw, npad, M);
}

size_t wire_energy_count(int n, int npad, int M) { return (size_t)wire_blocks(n, npad) * wire_fblocks(M) * kWL; }
size_t wire_list_count(int n, int npad) { return (size_t)wire_blocks(n, npad) * ((wire_valid(npad) + 7) / 8); }
size_t wire_chunk_count(int n, int npad) { return (size_t)wire_blocks(n, npad) * 4; }
int wire_row_blocks(int n, int npad) { return wire_blocks(n, npad); }

void launch_wire_conv_fft(const float2* Qh, const float2* Rw, const float2* taps, float2* Vh, int G, int npad, int nin,
                          int nout, int M, bool pair, double* energy, const WantRows& want, const RowList& list,
                          cudaStream_t s)
{
    if (nout <= 0) return;
    if (energy) {
        cudaFuncSetAttribute((const void*)k_wire_conv_fft, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kWConvSmem);
        k_wire_conv_fft<<<dim3(wire_fblocks(M), wire_blocks(nout, npad)), kWThreads, kWConvSmem, s>>>(
            Qh, Rw, Vh, G, npad, nin, nout, M, energy);
    }
    k_wire_pick<false><<<wire_blocks(nout, npad), kPickThreads, 0, s>>>(energy, wire_fblocks(M), npad, nout, want, list);
    launch_wire_rows(Qh, taps, Vh, G, npad, nin, nout, M, pair, list, s);
}

void launch_wire_adj_fft(const float2* Gh, const float2* Rw, const float2* taps, float2* dQh, int G, int npad, int nin,
                         int nout, int M, double* energy, const WantRows& want, const RowList& list, cudaStream_t s)
{
    if (nin <= 0) return;
    cudaFuncSetAttribute((const void*)k_wire_adj_fft, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWAdjSmem);
    k_wire_adj_fft<<<dim3(wire_fblocks(M), wire_blocks(nin, npad)), kWThreads, kWAdjSmem, s>>>(
        Gh, Rw, dQh, G, npad, nin, nout, M, energy);
    k_wire_pick<true><<<wire_blocks(nin, npad), kPickThreads, 0, s>>>(energy, wire_fblocks(M), npad, nin, want, list);
    launch_wire_rows_adj(Gh, taps, dQh, G, npad, nin, nout, M, list, s);
}

}  // namespace wctb200
