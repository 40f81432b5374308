// Adjoint (reverse-mode derivative) of the DepoTransform forward path.
//
// Forward (kernels.cu), per plane:
//   Q_g[w][t]  = sum over depo patches of qn * t_tau * (a_k or b_k)      (raster)
//   F[o][t]    = sum_g sum_j (R_g[j] (x) Q_g[o - npad - j])[t]          (FFT convolution)
// with, per patch bin k of a depo (pitch) and tau (time),
//   p_k = Phi(u_{k+1}) - Phi(u_k),  u = (edge - c_p) / sigma_p
//   a_k = p_k * w_k = [sigma_p (phi(u_{k+1}) - phi(u_k)) + (e_{k+1} - c_p) p_k] / bs
//   b_k = p_k - a_k,   t_tau likewise in time,   qn = q' / (sum p * sum t)
// (GaussianDiffusion.cxx:30-92,116-182; BinnedDiffusion_transform.cxx:296-367).
//
// Backward, per plane, given G = dL/dF on the frame window:
//   dQ_g[i] = sum_j conj(R_g[j]) * G[i + npad + j]   (per frequency; transposed convolution)
//   then per depo: gather the patch cells of dQ and apply the closed-form
//   derivatives of p, a, t and qn, chained through the drift
//   (Drifter.cxx:164-192) to (t, q, x, y, z, extent_long, extent_tran) and to
//   the global DL, DT and lifetime.  Patch windows are recomputed (k_prep_all),
//   never stored, and treated as fixed (the window edges are the only
//   non-differentiable points of the model).

#include "gauss.cuh"
#include "kernels.cuh"
#include "wire_fft.cuh"

namespace wctb200 {

// ---------------------------------------------------------------------------
// dL/dF of one plane as real grid rows: row o is wire wire0 + o, column c is
// tick tick0 + c; zero outside the reference window and the readout.
// ---------------------------------------------------------------------------
__global__ void k_grad_rows(const float* __restrict__ gframe, int nticks, int wire0, int wlo, int whi, int tick0,
                            int ncols, int nrows, int N, float* __restrict__ out)
{
    const int o = blockIdx.y;
    const int W = wire0 + o;
    const bool wok = W >= wlo && W < whi;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) {
        const int t = tick0 + c;
        float v = 0.f;
        if (wok && c < ncols && t >= 0 && t < nticks) v = gframe[(size_t)W * nticks + t];
        out[(size_t)o * N + c] = v;
    }
}

void launch_grad_rows(const float* gframe, int nticks, int wire0, int wlo, int whi, int tick0, int ncols, int nrows,
                      int N, float* out, cudaStream_t s)
{
    if (nrows <= 0) return;
    dim3 grid((N + 255) / 256, nrows);
    k_grad_rows<<<grid, 256, 0, s>>>(gframe, nticks, wire0, wlo, whi, tick0, ncols, nrows, N, out);
}

// ---------------------------------------------------------------------------
// Transposed wire convolution in the (wire, frequency) domain:
//   dQ_g[i][f] = sum_{j=-P}^{P} conj(R_g[j][f]) * G[i + P + j][f],  i in [0, nin)
// Block: 32 frequencies x 8 row groups, 8 consecutive rows per thread with a
// register window over the G rows staged in shared memory once for all
// groups; the taps of group g + 1 are copied by cp.async into the second of
// two tap buffers while group g is multiplied out of the first.
// ---------------------------------------------------------------------------
constexpr int kAdjRB = 8;
constexpr int kAdjRG = 8;
constexpr int kAdjRows = kAdjRB * kAdjRG;

// Rows at 32 frequencies: a warp's RB rows from i0 + rb0 on (rb0 < 0: none) of
// every group, of which mask are written; the block's rows lie within span (at
// most kAdjRows) of i0.  Called by all threads of a (32, kAdjRG) block.
template <int RB>
__device__ __forceinline__ void adj_unit(const float2* __restrict__ Gh, const float2* __restrict__ Rh,
                                         float2* __restrict__ dQh, int G, int PAD, int nin, int nout, int M, int f0,
                                         int i0, int span, int rb0, unsigned mask, float2* adj_smem)
{
    const int SROWS = span + 2 * PAD;
    const int NT = 2 * PAD + 1;
    float2(*Gs)[32] = reinterpret_cast<float2(*)[32]>(adj_smem);
    float2* Rbuf = adj_smem + (size_t)(kAdjRows + 2 * PAD) * 32;  // two tap buffers of NT x 32
    const int lane = threadIdx.x, rg = threadIdx.y;
    const int tid = rg * 32 + lane;
    const int f = f0 + lane;
    const bool fok = f < M;
    const bool dc = f == 0;
    // taps of group g into buffer st: 16 pieces of 16 bytes per 32-frequency row (M even)
    auto issue = [&](int g, int st) {
        float2* Rs = Rbuf + (size_t)st * NT * 32;
        const int fp = f0 + 2 * (tid & 15);
        const int nb = fp < M ? 16 : 0;
        for (int e = tid; e < NT * 16; e += 32 * kAdjRG) {
            const int jj = e >> 4;
            cp_async16(Rs + jj * 32 + 2 * (e & 15), nb ? Rh + ((size_t)g * NT + jj) * M + fp : Rh, nb);
        }
        cp_async_commit();
    };
    issue(0, 0);
    // rows i0 + s of G, s in [0, SROWS): input row i uses G rows i .. i + 2P
    for (int s = rg; s < SROWS; s += kAdjRG) {
        const int o = i0 + s;
        Gs[s][lane] = (fok && o < nout) ? Gh[(size_t)o * M + f] : make_float2(0.f, 0.f);
    }
    for (int g = 0; g < G; ++g) {
        if (g + 1 < G) {
            issue(g + 1, (g + 1) & 1);
            cp_async_wait<1>();
        }
        else
            cp_async_wait<0>();
        __syncthreads();  // group g's taps (and, at g = 0, the G rows) visible to every thread
        const float2* Rs = Rbuf + (size_t)(g & 1) * NT * 32;
        if (fok && rb0 >= 0) {
            float2 acc[RB], win[RB];
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                acc[r] = make_float2(0.f, 0.f);
                win[r] = Gs[rb0 + r][lane];
            }
            for (int jj = 0; jj < NT; ++jj) {
                const float2 rr = Rs[jj * 32 + lane];
                // conj(R) * G, component-wise in bin 0
                const float rc = dc ? 0.f : rr.y;
                const float ry = dc ? rr.y : rr.x;
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    const float2 q = win[r];  // G row rb0 + r + jj
                    acc[r].x = fmaf(rr.x, q.x, fmaf(rc, q.y, acc[r].x));
                    acc[r].y = fmaf(ry, q.y, fmaf(-rc, q.x, acc[r].y));
                }
#pragma unroll
                for (int r = 0; r < RB - 1; ++r) win[r] = win[r + 1];
                win[RB - 1] = Gs[min(rb0 + RB + jj, SROWS - 1)][lane];
            }
#pragma unroll
            for (int r = 0; r < RB; ++r)
                if (mask >> r & 1) dQh[((size_t)g * nin + i0 + rb0 + r) * M + f] = acc[r];
        }
        __syncthreads();  // buffer g & 1 is refilled with group g + 2 next
    }
}

__global__ void __launch_bounds__(32 * kAdjRG) k_wire_conv_adj(const float2* __restrict__ Gh,
                                                                const float2* __restrict__ Rh,
                                                                float2* __restrict__ dQh, int G, int PAD, int nin,
                                                                int nout, int M)
{
    extern __shared__ __align__(16) float2 adj_smem[];
    const int i0 = blockIdx.y * kAdjRows, rb0 = threadIdx.y * kAdjRB, left = nin - (i0 + rb0);
    adj_unit<kAdjRB>(Gh, Rh, dQh, G, PAD, nin, nout, M, blockIdx.x * 32, i0, kAdjRows, rb0,
             left >= kAdjRB ? 0xffu : (1u << max(left, 0)) - 1u, adj_smem);
}

// The chunks of a list (wire_fft.cuh), WAYS warps a group of rows.
static_assert(kAdjGroups == kAdjRG, "a chunk is a block's rows");
template <int WAYS>
__device__ __forceinline__ void adj_ways(const float2* __restrict__ Gh, const float2* __restrict__ Rh,
                                         float2* __restrict__ dQh, int G, int PAD, int nin, int nout, int M, int f0,
                                         const RowList& list, const int4& c, float2* adj_smem)
{
    constexpr int RB = kAdjRB / WAYS;
    const int mine = threadIdx.y / WAYS, first = RB * (threadIdx.y & (WAYS - 1));
    const int i0 = list.item[c.x].x;
    const int2 it = mine < c.y ? list.item[c.x + mine] : make_int2(0, 0);
    adj_unit<RB>(Gh, Rh, dQh, G, PAD, nin, nout, M, f0, i0, c.w, mine < c.y ? it.x - i0 + first : -1,
                 (unsigned)it.y >> first & ((1u << RB) - 1u), adj_smem);
}
__global__ void __launch_bounds__(32 * kAdjRG) k_wire_rows_adj(const float2* __restrict__ Gh,
                                                               const float2* __restrict__ Rh,
                                                               float2* __restrict__ dQh, int G, int PAD, int nin,
                                                               int nout, int M, RowList list)
{
    extern __shared__ __align__(16) float2 adj_smem[];
    const int nf = (M + 31) / 32, total = list.count[1] * nf;
    for (int u = blockIdx.x; u < total; u += gridDim.x) {
        const int4 c = list.chunk[u / nf];
        const int f0 = u % nf * 32;
        if (c.y <= kAdjRG / 4) adj_ways<4>(Gh, Rh, dQh, G, PAD, nin, nout, M, f0, list, c, adj_smem);
        else if (c.y <= kAdjRG / 2) adj_ways<2>(Gh, Rh, dQh, G, PAD, nin, nout, M, f0, list, c, adj_smem);
        else adj_ways<1>(Gh, Rh, dQh, G, PAD, nin, nout, M, f0, list, c, adj_smem);
    }
}

static size_t adj_smem_bytes(int npad)
{
    return sizeof(float2) * 32 * ((size_t)(kAdjRows + 2 * npad) + 2 * (size_t)(2 * npad + 1));
}

void launch_wire_rows_adj(const float2* Gh, const float2* taps, float2* dQh, int G, int npad, int nin, int nout, int M,
                          const RowList& list, cudaStream_t s)
{
    const size_t smem = adj_smem_bytes(npad);
    cudaFuncSetAttribute((const void*)k_wire_rows_adj, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_wire_rows_adj<<<148 * 4, dim3(32, kAdjRG), smem, s>>>(Gh, taps, dQh, G, npad, nin, nout, M, list);
}

void launch_wire_conv_adj(const float2* Gh, const float2* Rh, float2* dQh, int G, int npad, int nin, int nout, int M,
                          cudaStream_t s)
{
    if (nin <= 0) return;
    dim3 grid((M + 31) / 32, (nin + kAdjRows - 1) / kAdjRows);
    dim3 block(32, kAdjRG);
    const size_t smem = adj_smem_bytes(npad);
    cudaFuncSetAttribute((const void*)k_wire_conv_adj, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_wire_conv_adj<<<grid, block, smem, s>>>(Gh, Rh, dQh, G, npad, nin, nout, M);
}

// ---------------------------------------------------------------------------
// Per depo: gather the patch cells of dL/dQ on every plane and form the
// gradients.  One warp per depo; the patch's rows are tabulated in shared
// memory in chunks of impact bins, then each lane takes a tick (8 or 16 ticks
// and several rows side by side for short patches) and walks down the rows.
//
// What bounds it: the reads of dL/dQ, one value a cell, mostly from L2.  Two
// bins of a wire share the impact group between them, so the bins' factors
// are summed per group row first (as the raster does): a cell costs one load
// and three multiply-adds, and the tick factors enter once a lane at the end.
// Cells spread over the lanes, with both groups loaded and five sums a cell,
// took 5.1 ms for 500k depos (half in showers of 100 ticks x 30 impacts, three
// planes); this takes 3.7 ms, at half the issue slots and 20 warps an SM (96
// registers; 72 spill and take 4.8 ms).
//
// With x_k = edge_k - c (c the pitch centre, k = 0..np), u_k = x_k / s,
// phi the unit normal density and bs the impact bin size:
//   p_k      = Phi(u_{k+1}) - Phi(u_k)
//   a_k      = [s (phi(u_{k+1}) - phi(u_k)) + x_{k+1} p_k] / bs   (p_k * weight_k)
//   dp/dc    = -(phi_{k+1} - phi_k) / s
//   dp/ds    = -(u_{k+1} phi_{k+1} - u_k phi_k) / s
//   da/dc    = [(u phi)_{k+1} - (u phi)_k - p_k + x_{k+1} dp/dc] / bs
//   da/ds    = [phi_{k+1} - phi_k + (u^2 phi)_{k+1} - (u^2 phi)_k + x_{k+1} dp/ds] / bs
// and the same bin integrals and derivatives in time.  The patch adds
// qn t_tau a_k to group l and qn t_tau (p_k - a_k) to group l + 1 of its wire,
// qn = q / (sum_k p_k * sum_tau t_tau) (sums over the clipped patch).  Every
// accumulated quantity is a sum over rows and ticks of a row factor times a
// tick factor times dL/dQ, e.g. dL/dqn = sum_tau tv_tau sum_rows A_row D, with
// A_row = a_k + (p_{k-1} - a_{k-1}) for the row that bins k - 1 and k share.
// ---------------------------------------------------------------------------
constexpr int kGatherWarps = 4;
constexpr int kChunkP = 128;  // impact bins per table chunk
constexpr int kChunkT = 128;  // ticks per table chunk
constexpr int kChunkRows = kChunkP + kChunkP / 2 + 2;  // + one row a wire (at least two impacts each)

// One impact-group row of a patch chunk: the sums of the bin factors of
// dL/dqn, dL/dc and dL/dsigma, and where the row's first tick lies in the
// plane's grid.
struct __align__(16) RowTab {
    float a, dc, ds;
    int base;
};

__device__ __forceinline__ double warp_sum_d(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// s += v, the rounding error added to e (D. E. Knuth's two-sum).
__device__ __forceinline__ void add_carried(float& s, float& e, float v)
{
    const float t = __fadd_rn(s, v), b = __fsub_rn(t, s);
    e += __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(v, b));
    s = t;
}

// Quantities of one bin edge at distance x from the centre (sigma s > 0,
// is = 1/s, inv = 1/(sqrt(2) s)): the signed erfc of the forward's bin
// integrals, the density phi(u), u phi(u) and u^2 phi(u) with u = x/s.
__device__ __forceinline__ void edge_terms(float x, float is, float inv, float& E, float& f, float& uf, float& uuf)
{
    const float u = x * is;
    E = copysignf(erfc_nr(fabsf(x * inv)), x);
    f = norm_pdf(u);
    uf = u * f;
    uuf = u * uf;
}

__device__ __forceinline__ float warp_sum_f(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__global__ void __launch_bounds__(kGatherWarps * 32, 5) k_adj_gather(int n, PlaneSet ps, AdjSet as, double inv_vd,
                                                                     const PatchRec* __restrict__ rec,
                                                                     const float* __restrict__ dQ,
                                                                     double* __restrict__ grad,
                                                                     const double* __restrict__ qscale)
{
    __shared__ RowTab s_r[kGatherWarps][kChunkRows];
    __shared__ float4 s_t[kGatherWarps][kChunkT];
    const unsigned full = 0xffffffffu;
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * kGatherWarps + wib;
    if (i >= n) return;  // whole warps only: no block-level barrier follows
    // per-depo sums over planes: dL/dt', dL/dq', dL/dsL, dL/dsT, dL/d(x', y, z) through the pitch
    double s_ct = 0.0, s_qf = 0.0, s_sL = 0.0, s_sT = 0.0, s_px = 0.0, s_py = 0.0, s_pz = 0.0;
    bool any = false;
    // the tick table and its sums are the same on every plane unless the patch is cut differently
    int t_nt = -1;
    float t_cr = 0.f, t_st = 0.f, tS = 0.f, tSc = 0.f, tSs = 0.f;
    for (int ip = 0; ip < ps.nplanes; ++ip) {
        const PatchRec r = rec[(size_t)ip * n + i];
        const AdjPlane& A = as.p[ip];
        const int np = r.np, nt = r.nt;
        if (np == 0 || nt == 0 || A.nin == 0) continue;
        any = true;
        const float pbs = A.pbs, tbs = A.tbs, ipbs = 1.0f / pbs;
        const float sp = r.sp, st = r.st;
        const float isp = sp > 0.f ? 1.0f / sp : 0.f, invp = 0.70710678118654752f * isp;
        const float ist = st > 0.f ? 1.0f / st : 0.f, invt = 0.70710678118654752f * ist;
        // lane partial sums of the bin integrals and their derivatives (normalisation)
        float pS = 0.f, pSc = 0.f, pSs = 0.f;
        double acc_qn = 0.0, acc_cp = 0.0, acc_sp = 0.0, acc_ct = 0.0, acc_st = 0.0;
        const float* dQp = dQ + A.qoff;
        const int col = r.toff - A.col0;
        const bool have_t = nt <= kChunkT && t_nt == nt && t_cr == r.tcr && t_st == st;
        if (!have_t) {
            tS = tSc = tSs = 0.f;
            t_nt = nt;
            t_cr = r.tcr;
            t_st = st;
        }
        for (int t0 = 0; t0 < nt; t0 += kChunkT) {
            const int ntc = min(kChunkT, nt - t0);
            __syncwarp();
            if (have_t) {
            }
            else if (st > 0.f) {
                // one edge per lane, bins from neighbouring lanes (31 bins per round)
                for (int tb = t0; tb < t0 + ntc; tb += 31) {
                    const int e = tb + lane;
                    const float x = (float)e * tbs - r.tcr;
                    float E = 0.f, f = 0.f, uf = 0.f, uuf = 0.f;
                    if (e <= nt) edge_terms(x, ist, invt, E, f, uf, uuf);
                    const float E2 = __shfl_down_sync(full, E, 1), f2 = __shfl_down_sync(full, f, 1);
                    const float uf2 = __shfl_down_sync(full, uf, 1);
                    if (lane < 31 && e < t0 + ntc) {
                        const float tv = bin_from_edges(E, E2);
                        const float dtc = -(f2 - f) * ist, dts = -(uf2 - uf) * ist;
                        s_t[wib][e - t0] = make_float4(tv, dtc, dts, 0.f);
                        tS += tv;
                        tSc += dtc;
                        tSs += dts;
                    }
                    (void)uuf;
                }
            }
            else if (lane == 0) {  // point in time: one tick
                s_t[wib][0] = make_float4(1.f, 0.f, 0.f, 0.f);
                tS = 1.f;
            }
            for (int k0 = 0; k0 < np; k0 += kChunkP) {
                const int nk = min(kChunkP, np - k0);
                const int wire0 = (r.poff + k0) / A.nimp;
                int nrows = 0;
                __syncwarp();
                // 30 bins a round: lane 0 holds the bin before (its upper share goes to this round's first row)
                for (int kb = k0 - 1; kb < k0 + nk - 1; kb += 30) {
                    const int e = kb + lane;  // lanes 0 .. 30: bins kb .. kb + 30; lane 31: the last one's upper edge
                    float E = 0.f, f = 0.f, uf = 0.f, uuf = 0.f;
                    if (sp > 0.f && e >= 0 && e <= np) edge_terms((float)e * pbs - r.pcr, isp, invp, E, f, uf, uuf);
                    const float E2 = __shfl_down_sync(full, E, 1), f2 = __shfl_down_sync(full, f, 1);
                    const float uf2 = __shfl_down_sync(full, uf, 1), uuf2 = __shfl_down_sync(full, uuf, 1);
                    float bp = 0.f, ba = 0.f, dpdc = 0.f, dpds = 0.f, dadc = 0.f, dads = 0.f;
                    const bool real = lane < 31 && e >= k0 && e < k0 + nk;
                    if (real) {
                        if (sp > 0.f) {
                            const float x2 = (float)(e + 1) * pbs - r.pcr;
                            bp = bin_from_edges(E, E2);
                            dpdc = -(f2 - f) * isp;
                            dpds = -(uf2 - uf) * isp;
                            ba = fmaf(sp, f2 - f, x2 * bp) * ipbs;
                            dadc = (((uf2 - uf) - bp) + x2 * dpdc) * ipbs;
                            dads = (((f2 - f) + (uuf2 - uuf)) + x2 * dpds) * ipbs;
                        }
                        else {  // point in pitch: one bin, weight (edge_{k+1} - c) / bs
                            bp = 1.f;
                            ba = (pbs - r.pcr) * ipbs;
                            dadc = -ipbs;
                        }
                    }
                    // what the bin below leaves for this bin's lower row
                    const float ub = bp - ba, ubc = dpdc - dadc, ubs = dpds - dads;
                    const float lb = __shfl_up_sync(full, ub, 1), lbc = __shfl_up_sync(full, ubc, 1);
                    const float lbs = __shfl_up_sync(full, ubs, 1);
                    if (real && lane > 0) {
                        const int kabs = r.poff + e;
                        const int wire = kabs / A.nimp;
                        const int l = kabs - wire * A.nimp;
                        const bool below = l > 0 && e > k0;  // bin e - 1 shares the row
                        const int row = e - k0 + (wire - wire0);
                        const int base = (l * A.nin + (wire - A.start_ch)) * A.N + col + t0;
                        s_r[wib][row] = RowTab{below ? ba + lb : ba, below ? dadc + lbc : dadc,
                                               below ? dads + lbs : dads, base};
                        if (l == A.nimp - 1 || e == k0 + nk - 1)  // the wire's (or the chunk's) last row
                            s_r[wib][row + 1] = RowTab{ub, ubc, ubs, base + A.nin * A.N};
                        if (t0 == 0) {
                            pS += bp;
                            pSc += dpdc;
                            pSs += dpds;
                        }
                    }
                }
                nrows = nk + (r.poff + k0 + nk - 1) / A.nimp - wire0 + 1;
                __syncwarp();
                const int lg = ntc <= 8 ? 3 : (ntc <= 16 ? 4 : 5);  // ticks side by side: 8, 16 or 32
                const int sub = lane >> lg, tl = lane & ((1 << lg) - 1), nsub = 32 >> lg;
                for (int tc = 0; tc < ntc; tc += 32) {
                    const int tau = tc + tl;
                    if (tau >= ntc) continue;
                    const float* q = dQp + tau;
                    // eight rows a step, their loads in flight together; the steps' sums are
                    // added with their rounding errors carried along
                    float U = 0.f, Vc = 0.f, Vs = 0.f, Ue = 0.f, Vce = 0.f, Vse = 0.f;
                    for (int row = sub; row < nrows; row += 8 * nsub) {
                        float u[2] = {0.f, 0.f}, vc[2] = {0.f, 0.f}, vs[2] = {0.f, 0.f}, D[8];
#pragma unroll
                        for (int m = 0; m < 8; ++m) {
                            const int rm = row + m * nsub;
                            D[m] = rm < nrows ? __ldg(q + s_r[wib][rm].base) : 0.f;
                        }
#pragma unroll
                        for (int m = 0; m < 8; ++m) {
                            const RowTab R = s_r[wib][min(row + m * nsub, nrows - 1)];
                            u[m & 1] = fmaf(R.a, D[m], u[m & 1]);
                            vc[m & 1] = fmaf(R.dc, D[m], vc[m & 1]);
                            vs[m & 1] = fmaf(R.ds, D[m], vs[m & 1]);
                        }
                        add_carried(U, Ue, u[0] + u[1]);
                        add_carried(Vc, Vce, vc[0] + vc[1]);
                        add_carried(Vs, Vse, vs[0] + vs[1]);
                    }
                    const double dU = (double)U + (double)Ue;
                    const float4 tq = s_t[wib][tau];
                    acc_qn = fma((double)tq.x, dU, acc_qn);
                    acc_cp = fma((double)tq.x, (double)Vc + (double)Vce, acc_cp);
                    acc_sp = fma((double)tq.x, (double)Vs + (double)Vse, acc_sp);
                    acc_ct = fma((double)tq.y, dU, acc_ct);
                    acc_st = fma((double)tq.z, dU, acc_st);
                }
            }
        }
        // normalisation sums (whole warp), then this lane's share of the gradients:
        // every term is linear in the lane's partial sums, so the warp reduction
        // waits until all planes are done
        const float Sp = warp_sum_f(pS), dSp_c = warp_sum_f(pSc), dSp_s = warp_sum_f(pSs);
        const float St = warp_sum_f(tS), dSt_c = warp_sum_f(tSc), dSt_s = warp_sum_f(tSs);
        const float iSp = 1.0f / Sp, iSt = 1.0f / St;
        const double qn = r.qn;
        // centres and widths, through qn = q / (Sp * St) as well
        const double gcp = qn * acc_cp - acc_qn * (double)(r.qn * iSp * dSp_c);
        s_sT += qn * acc_sp - acc_qn * (double)(r.qn * iSp * dSp_s);                  // sigma_pitch = extent_tran
        s_ct += qn * acc_ct - acc_qn * (double)(r.qn * iSt * dSt_c);
        s_sL += (qn * acc_st - acc_qn * (double)(r.qn * iSt * dSt_s)) * inv_vd;      // sigma_time = extent_long / v
        // the plane's charge is qscale * q' (modify_depo): its share of dL/dq' carries the scale
        s_qf += acc_qn * (double)(iSp * iSt) * (qscale ? qscale[(size_t)i * ps.nplanes + ip] : 1.0);
        s_px += gcp * A.ax;
        s_py += gcp * A.ay;
        s_pz += gcp * A.az;
    }
    if (!any) return;
    s_ct = warp_sum_d(s_ct);
    s_qf = warp_sum_d(s_qf);
    s_px = warp_sum_d(s_px);
    s_py = warp_sum_d(s_py);
    s_pz = warp_sum_d(s_pz);
    s_sL = warp_sum_d(s_sL);
    s_sT = warp_sum_d(s_sT);
    if (lane == 0) {
        // sums over planes; k_adj_drift takes them back through the drift in place
        double* gd = grad + 7 * (size_t)i;
        gd[0] = s_ct;
        gd[1] = s_qf;
        gd[2] = s_px;
        gd[3] = s_py;
        gd[4] = s_pz;
        gd[5] = s_sL;
        gd[6] = s_sT;
    }
}

// Back through the drift (Drifter::insert, gen/src/Drifter.cxx:164-192), one
// thread per depo, in place on the per-depo sums of k_adj_gather
// (dL/dt', dL/dq', dL/d(x', y, z) through the pitch, dL/dsigma_L, dL/dsigma_T),
// plus the block sums of dL/d(DL, DT, lifetime).
__global__ void __launch_bounds__(256) k_adj_drift(const double* __restrict__ dep, int n, DriftDev dd,
                                                    double* __restrict__ grad, double* __restrict__ gglob)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double gDL = 0.0, gDT = 0.0, gTau = 0.0;
    if (i < n) {
        double* gd = grad + 7 * (size_t)i;
        const double s_ct = gd[0], s_qf = gd[1], s_sL = gd[5], s_sT = gd[6];
        const double* pd = dep + 7 * (size_t)i;
        const double q0 = pd[1], x0 = pd[2], el0 = pd[5], et0 = pd[6];
        int found = -1;
        double dir = 0.0;
        for (int k = 0; k < dd.nxr; ++k) {
            const double a = dd.xr[k][0], rp = dd.xr[k][1];
            if ((a < x0 && x0 < rp) || (rp < x0 && x0 < a)) { found = k; dir = -1.0; break; }
        }
        if (found < 0)
            for (int k = 0; k < dd.nxr; ++k) {
                const double rp = dd.xr[k][1], c = dd.xr[k][2];
                if ((rp < x0 && x0 < c) || (c < x0 && x0 < rp)) { found = k; dir = 1.0; break; }
            }
        double gx = 0.0;  // x' = x_response: x enters through the drift time only
        if (found >= 0) {
            const double respx = dd.xr[found][1];
            const double dtm = fabs((respx - x0) / dd.speed);
            const double dtdx = (x0 > respx ? 1.0 : -1.0) / dd.speed;  // d(dt)/dx
            if (dir > 0) {
                // t' = t + dt, q' = q exp(-dt/lifetime), sL^2 = 2 DL dt + el^2, sT^2 = 2 DT dt + et^2
                const double ex = exp(-dtm / dd.lifetime);
                const double qd = q0 * ex;
                const double sL = sqrt(2.0 * dd.DL * dtm + el0 * el0);
                const double sT = sqrt(2.0 * dd.DT * dtm + et0 * et0);
                const double hL = sL > 0.0 ? s_sL / sL : 0.0;
                const double hT = sT > 0.0 ? s_sT / sT : 0.0;
                const double gdt = s_ct - s_qf * qd / dd.lifetime + hL * dd.DL + hT * dd.DT;
                gx = gdt * dtdx;
                gd[1] = s_qf * ex;
                gd[5] = hL * el0;
                gd[6] = hT * et0;
                gDL = hL * dtm;
                gDT = hT * dtm;
                gTau = s_qf * qd * dtm / (dd.lifetime * dd.lifetime);
            }
            else {
                gx = -s_ct * dtdx;  // t' = t - dt in the response region
            }
        }
        gd[2] = gx;
    }
    __shared__ double s_glob[8][3];
    gDL = warp_sum_d(gDL);
    gDT = warp_sum_d(gDT);
    gTau = warp_sum_d(gTau);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) {
        s_glob[w][0] = gDL;
        s_glob[w][1] = gDT;
        s_glob[w][2] = gTau;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double v = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) v += s_glob[k][threadIdx.x];
        if (v != 0.0) atomicAdd(gglob + threadIdx.x, v);
    }
}

void launch_adj_gather(const double* depos, int n, const DriftDev& dd, int do_drift, const PlaneSet& ps,
                       const AdjSet& as, double drift_speed, const PatchRec* rec, const float* dQ, double* grad,
                       double* gglob, cudaStream_t s, const double* qscale)
{
    if (n <= 0) return;
    const int blocks = (n + kGatherWarps - 1) / kGatherWarps;
    k_adj_gather<<<blocks, kGatherWarps * 32, 0, s>>>(n, ps, as, 1.0 / drift_speed, rec, dQ, grad, qscale);
    if (do_drift) k_adj_drift<<<(n + 255) / 256, 256, 0, s>>>(depos, n, dd, grad, gglob);
}

}  // namespace wctb200
