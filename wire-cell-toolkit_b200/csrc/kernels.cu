// DepoTransform forward kernels for sm_100a.
//
// Pipeline for one event (all on one stream):
//   k_prep_all     drift + sensitive cut + BinnedDiffusion_transform::add +
//                  patch sample ranges + event window reduction + per-wire
//                  visit counts, all planes, one thread per depo
//   k_scan/k_fill  per-wire visit lists (CSR)
//   k_raster_*     erf-integrated patches with linear impact weights,
//                  accumulated per (wire, 256 ticks) in shared memory, written
//                  as the impact-group x tick charge grids: light, middling and
//                  heavy tiles                            gen/src/BinnedDiffusion_transform.cxx:227-391
//   k_rfft3        real FFT along time of each group row (fft3.cu; lengths
//                  without a plan: k_rfft_rows)            gen/src/ImpactTransform.cxx:149-151,237
//   k_wire_conv_fft  wire-direction convolution with the per-group response
//                  spectra, overlap-save (wire_fft.cu; short pads and rows:
//                  direct taps, k_wire_conv*)              gen/src/ImpactTransform.cxx:153-212,242-300
//   k_irfft3       inverse FFT along time, frame write     gen/src/ImpactTransform.cxx:303-347
//
// The 2-D FFT convolution of the reference is replaced by an equivalent (no
// wrap-around) real FFT along time plus a convolution along wires in the
// frequency domain.
//
// Index arithmetic that decides bins (drift, pitch distance, rejection,
// sample_bin_range, window min/max) is written with explicit _rn intrinsics
// so that no multiply-add is contracted and results are bit-identical to the
// reference's IEEE double arithmetic.

#include "kernels.cuh"
#include "gauss.cuh"
#include "rng.cuh"
#include "wire_fft.cuh"

#include <algorithm>
#include <cfloat>
#include <climits>
#include <type_traits>

namespace wctb200 {

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------
// Binning::bin (Binning.h:75), the truncated quotient. The product with the
// width's reciprocal is within 3 parts in 2^53 of the quotient, so away from a
// whole number both truncate to the same bin; next to one (and for NaN and
// out-of-range values) the division decides.
__device__ __forceinline__ int bin_of(double v, double lo, double bs, double rbs)
{
    const double d = __dsub_rn(v, lo);
    const double a = __dmul_rn(d, rbs);
    if (fabs(a) < 1e8 && fabs(a - rint(a)) > 1e-6) return __double2int_rz(a);
    return __double2int_rz(__ddiv_rn(d, bs));
}
__device__ __forceinline__ double edge_of(int i, double lo, double bs)
{
    return __dadd_rn(lo, __dmul_rn((double)i, bs));  // Binning::edge, Binning.h:88
}
__device__ __forceinline__ double gdistance(double x, double c, double s)
{
    return s != 0.0 ? __ddiv_rn(__dsub_rn(x, c), s) : __dsub_rn(x, c);  // GaussianDiffusion.h:34-44
}

// gdistance(x, c, s) > eff or, with below, < -eff. The product eff * s is far
// closer to the border than 1e-12 of the two sides, so away from it the sign
// of the difference decides; next to it the division does.
__device__ __forceinline__ bool beyond(double x, double c, double s, double eff, bool below)
{
    const double d = below ? __dsub_rn(c, x) : __dsub_rn(x, c);
    const double m = eff * s;
    const double diff = d - m;
    if (s > 1e-200 && fabs(diff) > 1e-12 * (fabs(d) + fabs(m))) return diff > 0.0;
    return below ? gdistance(x, c, s) < -eff : gdistance(x, c, s) > eff;
}

__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v)
{
    const unsigned hi = (unsigned)(v >> 32), mh = __reduce_min_sync(0xffffffffu, hi);
    return ((unsigned long long)mh << 32) | __reduce_min_sync(0xffffffffu, hi == mh ? (unsigned)v : 0xffffffffu);
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) { return ~warp_min_u64(~v); }

template <typename T, typename Op>
__device__ __forceinline__ T warp_reduce(T v, Op op)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// ---------------------------------------------------------------------------
// Drift, sensitive volume, rejection, patch window and visit counting for
// every plane, one thread per depo.
//
//   Drifter::insert without fluctuation          gen/src/Drifter.cxx:127-196
//   sensitive-volume cut                          aux/src/DepoTools.cxx:110-123,
//                                                 util/src/BoundingBox.cxx:37-56
//   BinnedDiffusion_transform::add rejection      gen/src/BinnedDiffusion_transform.cxx:37-92
//   GaussianDiffusion sample ranges               gen/src/GaussianDiffusion.cxx:116-149
//   window reduction (impact/time_bin_range)      gen/src/BinnedDiffusion_transform.cxx:416-464
//
// Bin integrals of the unit Gaussian are differences of erfc on the side of
// the centre the bin lies on, so tail bins keep full FP32 relative accuracy
// (0.5*(erf(b) - erf(a)) of GaussianDiffusion.cxx:30-56 loses ~4 digits there).
// ---------------------------------------------------------------------------
// Visit keys of one patch: (wire, tick tile) pairs for the wires
// [w0, w0 + wspan) and tiles [k0, k0 + kspan); key = wire * ntiles + tile.
// Warp-aggregated increment of the per-key visit counters; keys that hold a
// long patch are marked (their raster block spreads visits over warps).
__device__ __forceinline__ void count_visits(int* cnt, unsigned char* wide, bool lng, int wbase, int w0, int wspan,
                                             int k0, int kspan, int ntiles)
{
    const int span = wspan * kspan;
    const int maxspan = __reduce_max_sync(0xffffffffu, span);
    const int lane = threadIdx.x & 31;
    const unsigned longs = __ballot_sync(0xffffffffu, lng);
    int key = (wbase + w0) * ntiles + k0, left = kspan;
    for (int k = 0; k < maxspan; ++k) {
        const unsigned m = __match_any_sync(0xffffffffu, k < span ? key : -1);
        if (k < span && lane == __ffs(m) - 1) {
            atomicAdd(cnt + key, __popc(m));
            if (m & longs) wide[key] = 1;
        }
        ++key;
        if (--left == 0) {  // next wire
            left = kspan;
            key += ntiles - kspan;
        }
    }
}

// Bound of the fraction of a Gaussian of width s (0: a point) in one bin.
__device__ __forceinline__ float peak_fraction(float bs, float s)
{
    return s > 0.f ? fminf(1.0f, 0.39894228040143268f * bs / s) : 1.0f;  // 1/sqrt(2 pi)
}

// Magnitude bound of one visit's contribution to any cell: |q| * max bin
// fraction in pitch * max bin fraction in time * 2 (two bracketing groups).
__device__ __forceinline__ float visit_bound(float qn, float sp, float st, float pbs, float tbs)
{
    return 2.0f * fabsf(qn) * peak_fraction(pbs, sp) * peak_fraction(tbs, st) * 1.0001f;
}

// Unit bin integral of bin k of a patch (edges at k*bs - cr and (k+1)*bs - cr
// from the centre), with explicitly rounded operations and not inlined, so
// every kernel that calls it gets the same value bit for bit.
__device__ __noinline__ float unit_bin(int k, float bs, float cr, float sigma)
{
    if (!(sigma > 0.f)) return 1.0f;  // point: its single bin holds everything
    const float inv = __frcp_rn(__fmul_rn(1.41421356237309505f, sigma));
    const float x1 = __fmul_rn(__fsub_rn(__fmul_rn((float)k, bs), cr), inv);
    const float x2 = __fmul_rn(__fsub_rn(__fmul_rn((float)(k + 1), bs), cr), inv);
    return bin_from_edges(copysignf(erfc_nr(fabsf(x1)), x1), copysignf(erfc_nr(fabsf(x2)), x2));
}

// 1 / (sum of the patch's unit bin integrals in pitch * in time), edge to edge.
__device__ __noinline__ float patch_inv_norm(const PatchRec& r, float pbs, float tbs)
{
    float sp = 1.f, st = 1.f;
    if (r.sp > 0.f) {
        const float inv = __frcp_rn(__fmul_rn(1.41421356237309505f, r.sp));
        const float x1 = __fmul_rn(__fsub_rn(0.f, r.pcr), inv);
        const float x2 = __fmul_rn(__fsub_rn(__fmul_rn((float)r.np, pbs), r.pcr), inv);
        sp = bin_from_edges(copysignf(erfc_nr(fabsf(x1)), x1), copysignf(erfc_nr(fabsf(x2)), x2));
    }
    if (r.st > 0.f) {
        const float inv = __frcp_rn(__fmul_rn(1.41421356237309505f, r.st));
        const float x1 = __fmul_rn(__fsub_rn(0.f, r.tcr), inv);
        const float x2 = __fmul_rn(__fsub_rn(__fmul_rn((float)r.nt, tbs), r.tcr), inv);
        st = bin_from_edges(copysignf(erfc_nr(fabsf(x1)), x1), copysignf(erfc_nr(fabsf(x2)), x2));
    }
    return __frcp_rn(__fmul_rn(sp, st));
}

// Event of a prep/fill block: blocks never straddle events.
__device__ __forceinline__ int event_of_block(const EventTable& et, int b)
{
    int lo = 0, hi = et.nev - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (et.blk0[mid] <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Frame ident of event ev of the launch: the key of its random streams.
__device__ __forceinline__ int fluc_ident(const FlucParams& fp, int ev)
{
    return (fp.ident_base ? *fp.ident_base : 0) + fp.ident0 + ev;
}

// The electrons a drifting depo loses (not inlined: the sampler's registers
// would be the prep kernel's).
__device__ __noinline__ int drift_draw(unsigned key0, unsigned key1, int i_ev, int nq, double absorb)
{
    Philox g;
    g.init(key0, key1, (unsigned)i_ev, kRngDriftTag, 0u);
    return binomial(nq, absorb, g);
}

// Depo counters of a plane in one word, six bits each: a warp's sum fits.
constexpr unsigned kAdded = 1u, kOutTime = 1u << 6, kOutPitch = 1u << 12, kOversize = 1u << 18, kBig = 1u << 24;

// One thread per (depo, plane) of every event of the table (plane =
// blockIdx.y; each plane's threads drift the depo again, which is cheaper
// than serialising the planes' FP64 chains in one thread); per-event window
// statistics, visit counters and bounds (nkeys keys per event); patch
// records [plane][depo]; plane 0's threads also write the drifted charge and
// the time profiles indexed by the depo's position in the concatenated depo
// array.
//
// Issue-bound at size (520k depos: 1460 instructions a warp, 70% of the issue
// slots), a chain of FP64 operations when small. Quotients that only place a
// patch or cut a depo are products away from the border (bin_of, beyond),
// warp sums are redux instructions with the counters packed in one word, the
// time window is found once, and profiles leave in 16-byte stores: 520k depos
// x 3 planes 113 -> 85 us, 20k x 3 12.0 -> 9.1, 2k 13.8 -> 8.6, 500k on tracks
// with long patches 484 -> 375 (there the bounds' atomics on shared wires; a
// warp's adding up per block first: no gain, and 9 -> 20 us at 20k).
// FLUC: charges fluctuate as they drift (kept apart: the sampler's call costs
// the other case 0.2 KB of spills).
template <bool FLUC>
__global__ void __launch_bounds__(256, 4) k_prep_all(const double* __restrict__ dep, EventTable evt, int nkeys,
                                                  DriftDev dd, int do_drift, PlaneSet ps, TimeDev tb,
                                                  double drift_speed, double nsigma, PatchRec* __restrict__ rec,
                                                  WindowDev* __restrict__ win_all, int* __restrict__ cnt_all,
                                                  float* __restrict__ tprof, unsigned long long* __restrict__ kb_all,
                                                  FlucParams fp, double* __restrict__ fq,
                                                  unsigned char* __restrict__ wide_all, int blk_offset,
                                                  const double* __restrict__ qscale)
{
    const int bid = blockIdx.x + blk_offset;  // a launch may cover a range of the table's blocks
    const int ev = event_of_block(evt, bid);
    const int i = evt.dep0[ev] + (bid - evt.blk0[ev]) * blockDim.x + threadIdx.x;
    const int n = evt.dep0[evt.nev];  // record stride: all depos of the table
    const bool in = i < evt.dep0[ev + 1];
    WindowDev* win = win_all + (size_t)ev * ps.nplanes;
    int* wire_cnt = cnt_all + (size_t)ev * nkeys;
    unsigned long long* key_bound = kb_all + (size_t)ev * nkeys * kTileBlocks;
    double t = 0, q = 0, x = 0, y = 0, z = 0, el = 0, et = 0;
    bool ok = false;
    if (in) {
        const double* p = dep + 7 * (size_t)i;
        t = p[0]; q = p[1]; x = p[2]; y = p[3]; z = p[4]; el = p[5]; et = p[6];
        // a depo with a NaN or infinite value is dropped: the reference's
        // bin-index arithmetic is undefined for it, and its extents would
        // otherwise reach the event window's min/max reduction
        ok = isfinite(t) && isfinite(q) && isfinite(x) && isfinite(y) && isfinite(z) && isfinite(el) && isfinite(et);
        if (ok && do_drift) {
            if (q == 0.0) ok = false;
            else {
                int found = -1;
                double dir = 0.0;
                for (int r = 0; r < dd.nxr; ++r) {
                    const double a = dd.xr[r][0], rp = dd.xr[r][1];
                    if ((a < x && x < rp) || (rp < x && x < a)) { found = r; dir = -1.0; break; }
                }
                if (found < 0)
                    for (int r = 0; r < dd.nxr; ++r) {
                        const double rp = dd.xr[r][1], c = dd.xr[r][2];
                        if ((rp < x && x < c) || (c < x && x < rp)) { found = r; dir = 1.0; break; }
                    }
                if (found < 0) ok = false;
                else {
                    const double respx = dd.xr[found][1];
                    const double dt = fabs(__ddiv_rn(__dsub_rn(respx, x), dd.speed));
                    if (dir > 0) {
                        const double absorb = __dsub_rn(1.0, exp(__ddiv_rn(-dt, dd.lifetime)));
                        if (FLUC) {
                            // Binomial(|Q|, absorb) electrons absorbed (Drifter.cxx:179-185)
                            const int nabs = drift_draw(
                                fp.key0, fp.key1 + 0x9E3779B9u * (unsigned)fluc_ident(fp, ev), i - evt.dep0[ev],
                                (int)fabs(q), absorb);
                            q = __dsub_rn(q, q < 0 ? -(double)nabs : (double)nabs);
                        }
                        else q = __dsub_rn(q, __dmul_rn(q, absorb));
                        el = __dsqrt_rn(__dadd_rn(__dmul_rn(__dmul_rn(2.0, dd.DL), dt), __dmul_rn(el, el)));
                        et = __dsqrt_rn(__dadd_rn(__dmul_rn(__dmul_rn(2.0, dd.DT), dt), __dmul_rn(et, et)));
                    }
                    t = __dadd_rn(__dadd_rn(t, __dmul_rn(dir, dt)), dd.toffset);
                    x = respx;
                }
            }
        }
    }
    const int ip = blockIdx.y;
    // DepoTransform::modify_depo (DepoTransform.h:33-35, applied before
    // BinnedDiffusion_transform::add at DepoTransform.cxx:182) as a per-plane
    // charge scale, [depo][plane]
    if (qscale && in) q = __dmul_rn(q, qscale[(size_t)i * ps.nplanes + ip]);
    if (fq && in) fq[(size_t)ip * n + i] = q;  // the plane's charge: trial count of its fluctuated patch
    // The time profile depends on the depo only (GaussianDiffusion.cxx:124-136):
    // compute it once here for every plane's raster.
    // its window is every plane's.
    unsigned mywide = 0;
    double st = 0, tlo = 0, thi = 0;
    int t0 = 0, t1 = 0;
    float tcr = 0.f;
    if (ok) {
        st = __ddiv_rn(el, drift_speed);  // DepoTransform.cxx:185
        tlo = __dsub_rn(t, __dmul_rn(st, nsigma));
        thi = __dadd_rn(t, __dmul_rn(st, nsigma));
        t0 = max(bin_of(tlo, tb.tmin, tb.bs, tb.rbs), 0);
        t1 = min(bin_of(thi, tb.tmin, tb.bs, tb.rbs) + 1, tb.nbins);
        tcr = (float)__dsub_rn(t, edge_of(t0, tb.tmin, tb.bs));
        const int nt = t1 - t0;
        if (ip == 0 && nt > kTprof) mywide = nt;
        if (ip == 0 && nt > 0 && nt <= kTprof) {
            float* tp = tprof + (size_t)i * kTprof;
            if (st > 0) {
                const float fst = (float)st;
                const float inv = 1.0f / (1.41421356237309505f * fst);
                const float tbs = (float)tb.bs;
                float e1 = edge_erfc(0.f, tbs, tcr, inv);
                for (int k = 0; k < nt; k += 4) {  // (a row is 64 bytes; past the patch: not read)
                    float v[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float e2 = edge_erfc((float)(k + j + 1), tbs, tcr, inv);
                        v[j] = bin_from_edges(e1, e2);
                        e1 = e2;
                    }
                    *reinterpret_cast<float4*>(tp + k) = make_float4(v[0], v[1], v[2], v[3]);
                }
            }
            else {
                tp[0] = 1.0f;
            }
        }
    }
    __shared__ unsigned long long s_k[4][8];
    __shared__ unsigned s_c[4][8];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    {
        const PlaneDev& pl = ps.p[ip];
        unsigned long long kpmin = ~0ull, kpmax = 0ull, ktmin = ~0ull, ktmax = 0ull;
        unsigned flags = 0;  // six bits for each of kAdd ...: a warp's sum stays apart
        PatchRec r;
        r.toff = r.poff = 0;
        r.nt = r.np = 0;
        r.tcr = r.pcr = r.st = r.sp = r.qn = 0.f;
        bool inbb = ok;
        if (ok && pl.have_bb) {
            const double pp[3] = {x, y, z};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double b1 = pl.bb_lo[k], b2 = pl.bb_hi[k];
                if (b1 < b2) { if (pp[k] < b1 || pp[k] > b2) inbb = false; }
                else if (b2 < b1) { if (pp[k] < b2 || pp[k] > b1) inbb = false; }
            }
        }
        if (inbb) {
            const double ct = t;
            const double rx = __dsub_rn(x, pl.ox), ry = __dsub_rn(y, pl.oy), rz = __dsub_rn(z, pl.oz);
            const double cp = __dadd_rn(__dadd_rn(__dmul_rn(pl.ax, rx), __dmul_rn(pl.ay, ry)),
                                        __dmul_rn(pl.az, rz));                  // Pimpos.cxx:58
            const double sp = et;
            const double eff_t = st > 0 ? nsigma : 0.0;
            const double eff_p = sp > 0 ? nsigma : 0.0;
            if (beyond(tb.tmin, ct, st, eff_t, false) || beyond(tb.tmax, ct, st, eff_t, true)) {
                flags = kOutTime;
            }
            else if (beyond(pl.imp_min, cp, sp, eff_p, false) || beyond(pl.imp_max, cp, sp, eff_p, true)) {
                flags = kOutPitch;
            }
            else {
                flags = kAdded;
                const double plo = __dsub_rn(cp, __dmul_rn(sp, nsigma));
                const double phi = __dadd_rn(cp, __dmul_rn(sp, nsigma));
                ktmin = dkey(tlo); ktmax = dkey(thi);
                kpmin = dkey(plo); kpmax = dkey(phi);
                const int p0 = max(bin_of(plo, pl.imp_min, pl.imp_bs, pl.imp_rbs), 0);
                const int p1 = min(bin_of(phi, pl.imp_min, pl.imp_bs, pl.imp_rbs) + 1, pl.imp_nbins);
                if (t1 > t0 && p1 > p0) {
                    const int nt = t1 - t0, np = p1 - p0;
                    if (nt > kMaxPatchT || np > kMaxPatchP || (st == 0.0 && nt != 1) || (sp == 0.0 && np != 1)) {
                        flags += kOversize;
                    }
                    else {
                        r.toff = t0;
                        r.poff = p0;
                        r.nt = (unsigned short)nt;
                        r.np = (unsigned short)np;
                        r.tcr = tcr;
                        r.pcr = (float)__dsub_rn(cp, edge_of(p0, pl.imp_min, pl.imp_bs));
                        r.st = (float)st;
                        r.sp = (float)sp;
                        // normalisation to the full charge (GaussianDiffusion.cxx:176-182) with the
                        // sums of the unit bin integrals taken edge to edge
                        float sum_t = 1.f, sum_p = 1.f;
                        if (st > 0) {
                            const float inv = 1.0f / (1.41421356237309505f * r.st);
                            sum_t = bin_from_edges(edge_erfc(0.f, (float)tb.bs, r.tcr, inv),
                                                   edge_erfc((float)nt, (float)tb.bs, r.tcr, inv));
                        }
                        if (sp > 0) {
                            const float inv = 1.0f / (1.41421356237309505f * r.sp);
                            sum_p = bin_from_edges(edge_erfc(0.f, (float)pl.imp_bs, r.pcr, inv),
                                                   edge_erfc((float)np, (float)pl.imp_bs, r.pcr, inv));
                        }
                        // the quotient by a Newton step on the float reciprocal (2^-46, far
                        // below the float that is kept)
                        const double sn = (double)sum_t * (double)sum_p;
                        if (sn > 1e-30) {
                            const double r0 = (double)__frcp_rn((float)sn);
                            r.qn = (float)(q * fma(r0, fma(-sn, r0, 1.0), r0));
                        }
                        else r.qn = (float)(q / sn);
                    }
                }
            }
        }
        if (in) rec[(size_t)ip * n + i] = r;
        const int w0 = r.np ? (int)((unsigned)r.poff / (unsigned)pl.nimp) : 0;
        const int span = r.np ? (int)((unsigned)(r.poff + r.np - 1) / (unsigned)pl.nimp) - w0 + 1 : 0;
        const int k0 = r.toff / kTile;
        const int kspan = r.np ? (r.toff + r.nt - 1) / kTile - k0 + 1 : 0;
        count_visits(wire_cnt, wide_all + (size_t)ev * nkeys, r.nt > kTprof, pl.wire_base, w0, span, k0, kspan, ps.ntiles);
        // fixed-point bounds of the raster: per (wire, tile, 64-tick block), summed
        // as integers in units of 2^-16 (each term rounded up), so the bound --
        // and with it the raster's scale -- does not depend on the order of the adds
        if (r.np) {
            const float b = visit_bound(r.qn, r.sp, r.st, (float)pl.imp_bs, (float)tb.bs);
            if (b > kMaxVisitBound) flags += kBig;
            const unsigned long long bu = __float2ull_ru(fminf(b, kMaxVisitBound) * 65536.0f);
            const int b0 = r.toff / kScaleBlock, b1 = (r.toff + r.nt - 1) / kScaleBlock;
            for (int ww = 0; ww < span; ++ww) {
                unsigned long long* kb = key_bound + (size_t)(pl.wire_base + w0 + ww) * ps.ntiles * kTileBlocks;
                for (int bb = b0; bb <= b1; ++bb) atomicAdd(kb + bb, bu);
            }
        }
        // block reduction, one atomic per block per quantity (the totals all go
        // to one address, where a thread's own atomics queue up: 500k depos,
        // half with long patches, 484 us with one per thread and long patch).
        // 32 bits hold a block's totals: a patch has at most 2^20 cells.
        kpmin = warp_min_u64(kpmin);
        ktmin = warp_min_u64(ktmin);
        kpmax = warp_max_u64(kpmax);
        ktmax = warp_max_u64(ktmax);
        flags = __reduce_add_sync(0xffffffffu, flags);
        const unsigned vis = __reduce_add_sync(0xffffffffu, (unsigned)(span * kspan));
        const unsigned cells = __reduce_add_sync(0xffffffffu, (unsigned)r.np * r.nt);
        if (ip == 0) mywide = __reduce_add_sync(0xffffffffu, mywide);
        if (l == 0) {
            s_k[0][w] = kpmin; s_k[1][w] = kpmax; s_k[2][w] = ktmin; s_k[3][w] = ktmax;
            s_c[0][w] = flags; s_c[1][w] = vis; s_c[2][w] = cells; s_c[3][w] = mywide;
        }
        __syncthreads();
        // a thread a quantity over the block's warps
        const int nw = blockDim.x >> 5;
        WindowDev* wd = win + ip;
        if (threadIdx.x < 4) {
            const int k = threadIdx.x;
            unsigned long long v = s_k[k][0];
            for (int j = 1; j < nw; ++j) v = k & 1 ? max(v, s_k[k][j]) : min(v, s_k[k][j]);
            if (v != (k & 1 ? 0ull : ~0ull)) {
                if (k == 0) atomicMin(&wd->pmin, v);
                else if (k == 1) atomicMax(&wd->pmax, v);
                else if (k == 2) atomicMin(&wd->tmin, v);
                else atomicMax(&wd->tmax, v);
            }
        }
        else if (threadIdx.x >= 32 && threadIdx.x < 32 + 5) {
            const int k = threadIdx.x - 32;
            unsigned v = 0;
            for (int j = 0; j < nw; ++j) v += (s_c[0][j] >> (6 * k)) & 63u;
            int* to = k == 0 ? &wd->nadded : k == 1 ? &wd->out_time : k == 2 ? &wd->out_pitch
                                                   : k == 3 ? &wd->oversize : &wd->bigcharge;
            if (v) atomicAdd(to, (int)v);
        }
        else if (threadIdx.x >= 64 && threadIdx.x < 64 + 3) {
            // 64-bit totals of the event (visits: the lists use int offsets)
            const int k = threadIdx.x - 64;
            unsigned long long v = 0;
            for (int j = 0; j < nw; ++j) v += s_c[1 + k][j];
            unsigned long long* to = k == 0 ? &win[0].nvisits : (k == 1 ? &win[0].ncells : &win[0].wide_ticks);
            if (v) atomicAdd(to, v);
        }
    }
}

void launch_prep_all(const double* depos, const EventTable& et, int nkeys, const DriftDev& dd, int do_drift,
                     const PlaneSet& ps, const TimeDev& tb, double drift_speed, double nsigma, PatchRec* rec,
                     WindowDev* win, int* wire_cnt, float* tprof, unsigned long long* key_bound,
                     const FlucParams& fp, double* fq, unsigned char* wide, cudaStream_t s, int blk_begin,
                     int blk_end, const double* qscale)
{
    const int nb = et.blk0[et.nev];
    const int b0 = std::max(0, blk_begin), b1 = blk_end < 0 ? nb : std::min(blk_end, nb);
    if (b1 <= b0) return;
    auto* k = fp.on_drift ? k_prep_all<true> : k_prep_all<false>;
    k<<<dim3(b1 - b0, ps.nplanes), 256, 0, s>>>(depos, et, nkeys, dd, do_drift, ps, tb, drift_speed, nsigma, rec, win,
                                                wire_cnt, tprof, key_bound, fp, fq, wide, b0, qscale);
}

// Exclusive scan of the per-key visit counts: block sums, a scan of the
// block sums, then per-block scans with their offsets.
constexpr int kScanBlock = 1024;

__device__ __forceinline__ int block_scan_excl(int v, int* s_warp, int& total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = lane < (int)(blockDim.x >> 5) ? s_warp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        s_warp[lane] = t;
    }
    __syncthreads();
    total = s_warp[(blockDim.x >> 5) - 1];
    const int before = w ? s_warp[w - 1] : 0;
    __syncthreads();
    return before + x - v;
}

__global__ void __launch_bounds__(kScanBlock) k_scan_sums(const int* __restrict__ cnt, int n, int* __restrict__ sums)
{
    __shared__ int s_warp[32];
    const int i = blockIdx.x * kScanBlock + threadIdx.x;
    int total = 0;
    block_scan_excl(i < n ? cnt[i] : 0, s_warp, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanBlock) k_scan_top(int* __restrict__ sums, int nb, int* __restrict__ total_out)
{
    __shared__ int s_warp[32];
    int carry = 0;
    for (int b0 = 0; b0 < nb; b0 += kScanBlock) {
        const int i = b0 + threadIdx.x;
        int total = 0;
        const int ex = block_scan_excl(i < nb ? sums[i] : 0, s_warp, total);
        if (i < nb) sums[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) *total_out = carry;
}

__global__ void __launch_bounds__(kScanBlock) k_scan_apply(const int* __restrict__ cnt, int n,
                                                           const int* __restrict__ sums, int* __restrict__ off,
                                                           int* __restrict__ cur)
{
    __shared__ int s_warp[32];
    const int i = blockIdx.x * kScanBlock + threadIdx.x;
    int total = 0;
    const int ex = block_scan_excl(i < n ? cnt[i] : 0, s_warp, total) + sums[blockIdx.x];
    if (i < n) {
        off[i] = ex;
        cur[i] = ex;
    }
}

void launch_scan(const int* wire_cnt, int nwires_total, int* wire_off, int* wire_cur, cudaStream_t s)
{
    // wire_cur[nwires_total + 1 ..] holds the block sums (the caller sizes it)
    const int n = nwires_total;
    const int nb = (n + kScanBlock - 1) / kScanBlock;
    int* sums = wire_cur + n + 1;
    k_scan_sums<<<nb, kScanBlock, 0, s>>>(wire_cnt, n, sums);
    k_scan_top<<<1, kScanBlock, 0, s>>>(sums, nb, wire_off + n);
    k_scan_apply<<<nb, kScanBlock, 0, s>>>(wire_cnt, n, sums, wire_off, wire_cur);
}

// Time profiles of the long patches, one warp per depo (its first plane with a
// patch: the time profile does not depend on the plane); room for a block's
// depos is taken in one go (one address: see k_prep_all).
__global__ void __launch_bounds__(256) k_tprof_pool(const PatchRec* __restrict__ rec, EventTable evt, int nplanes,
                                                   float tbs, TprofPool pool, int* status)
{
    __shared__ int s_nt[8];
    __shared__ long long s_off;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int n = evt.dep0[evt.nev];
    const int i = blockIdx.x * 8 + w;
    PatchRec r{};
    for (int ip = 0; ip < nplanes && i < n; ++ip) {
        r = rec[(size_t)ip * n + i];
        if (r.np) break;
    }
    const int nt = r.np && r.nt > kTprof ? r.nt : 0;
    if (lane == 0) s_nt[w] = nt;
    __syncthreads();
    if (threadIdx.x == 0) {
        int tot = 0;
        for (int k = 0; k < 8; ++k) tot += s_nt[k];
        s_off = tot ? (long long)atomicAdd(pool.used, (unsigned long long)tot) : 0;
    }
    __syncthreads();
    if (i >= n) return;
    int off = -1;
    if (nt) {
        long long off64 = s_off;
        for (int k = 0; k < w; ++k) off64 += s_nt[k];
        off = off64 + nt > pool.cap ? -1 : (int)off64;  // 64-bit counter: no wrap
        if (off < 0) {
            if (lane == 0 && status) atomicOr(status, kBatchPoolShort);
        }
        else
            for (int t = lane; t < nt; t += 32) pool.val[off + t] = unit_bin(t, tbs, r.tcr, r.st);
    }
    if (lane == 0) pool.off[i] = off;
}

void launch_tprof_pool(const PatchRec* rec, const EventTable& et, int nplanes, float tbs, const TprofPool& pool,
                       int* status, cudaStream_t s)
{
    const int n = et.dep0[et.nev];
    if (n <= 0) return;
    k_tprof_pool<<<(n + 7) / 8, 256, 0, s>>>(rec, et, nplanes, tbs, pool, status);
}

// Per-wire visit lists: wire_list[wire_off[w] ..] holds the depo indices whose
// patch covers wire w (any order).
__global__ void __launch_bounds__(256) k_fill(const PatchRec* __restrict__ rec, EventTable evt, int nkeys,
                                              PlaneSet ps, int* __restrict__ cur, Visit* __restrict__ list,
                                              long long cap)
{
    const int ev = event_of_block(evt, blockIdx.x);
    const int i = evt.dep0[ev] + (blockIdx.x - evt.blk0[ev]) * blockDim.x + threadIdx.x;
    const int n = evt.dep0[evt.nev];
    const bool in = i < evt.dep0[ev + 1];
    const int key0 = ev * nkeys;
    const int lane = threadIdx.x & 31;
    for (int ip = 0; ip < ps.nplanes; ++ip) {
        const PlaneDev& pl = ps.p[ip];
        int w0 = 0, span = 0, k0 = 0, kspan = 1;
        PatchRec r{};
        if (in) {
            r = rec[(size_t)ip * n + i];
            if (r.np) {
                w0 = r.poff / pl.nimp;
                k0 = r.toff / kTile;
                kspan = (r.toff + r.nt - 1) / kTile - k0 + 1;
                span = ((r.poff + r.np - 1) / pl.nimp - w0 + 1) * kspan;
            }
        }
        int maxspan = span;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) maxspan = max(maxspan, __shfl_xor_sync(0xffffffffu, maxspan, o));
        for (int k = 0; k < maxspan; ++k) {
            int key = -1;
            if (k < span) {
                const int dw = k / kspan, dk = k - dw * kspan;
                key = key0 + (pl.wire_base + w0 + dw) * ps.ntiles + k0 + dk;
            }
            const unsigned act = __ballot_sync(0xffffffffu, key >= 0);
            if (key >= 0) {
                const unsigned m = __match_any_sync(act, key);
                const int leader = __ffs(m) - 1;
                int base = 0;
                if (lane == leader) base = atomicAdd(cur + key, __popc(m));
                base = __shfl_sync(m, base, leader);
                const int rank = __popc(m & ((1u << lane) - 1u));
                const long long at = (long long)base + rank;
                if (at >= 0 && at < cap) list[at] = i;  // outside: the caller reports an overflow
            }
        }
    }
}

void launch_fill(const PatchRec* rec, const EventTable& et, int nkeys, const PlaneSet& ps, int* wire_cur,
                 Visit* visits, long long cap, cudaStream_t s)
{
    const int nblocks = et.blk0[et.nev];
    if (nblocks <= 0) return;
    k_fill<<<nblocks, 256, 0, s>>>(rec, et, nkeys, ps, wire_cur, visits, cap);
}

// ---------------------------------------------------------------------------
// Charge grids: one block per charge wire row of every plane.  The block
// accumulates the row's impact-group x tick grid in shared memory (one thread
// per depo visit of the wire), then writes the G rows of the plane grid with
// zero padding up to the FFT length.  Each patch bin adds weight*q to the
// group of its lower impact edge and (1-weight)*q to the next
// (BinnedDiffusion_transform.cxx:296-367, linear weights of
// GausDesc::weight, GaussianDiffusion.cxx:61-92).
//
// Accumulation is in 32-bit fixed point (native shared-memory integer
// atomics; FP32 shared atomics are compare-and-swap loops).  Every 64-tick
// block of the row has its own scale 2^30 / B, where B bounds the magnitude
// any cell of the block can reach: the sum over the visits touching the block
// of |q| * max bin fraction in pitch * max bin fraction in time * 2.  Cells
// cannot overflow and one add is resolved to ~2^-30 of that local bound.
// Integer sums are order independent (the bounds too are integer sums), so
// the grid is bit-reproducible.
// ---------------------------------------------------------------------------
constexpr int kRasterThreads = 256;
constexpr int kLightThreads = 64;  // of the launch over all tiles, most of them with few visits or none
constexpr int kLightBlocks = 11;
// staged per visit: 12 group coefficients and 16 scaled tick values (odd stride: no bank conflicts)
constexpr int kStageT = 12;
constexpr int kStageStride = 29;
constexpr int kTileLd = kTile + 8;  // fluctuated raster: row stride with an 8-word skew between groups
// Forward raster grid row stride: 4 words of skew, so eight visits scattering
// to eight consecutive group rows at the same four columns hit 32 distinct banks.
constexpr int kGridLd = kTile + 4;

static size_t raster_smem(int G, int threads)
{
    return sizeof(int) * (size_t)G * kGridLd + (sizeof(float) * kStageStride + sizeof(int4)) * (size_t)threads;
}
size_t raster_smem_bytes(int G) { return raster_smem(G, kRasterThreads); }
// Long visits of a heavy part, behind that: their integer coefficients by group
// (three int4) and one of (column | length, profile offset, scaled charge, depo).
constexpr int kLongQuads = 4;
static size_t raster_heavy_smem_bytes(int G)
{
    return raster_smem_bytes(G) + sizeof(int4) * (size_t)kRasterThreads * kLongQuads;
}

// The first launch rasterises the light tiles, a block each, lists middling ones
// for blocks of their own size and the heavy ones -- those with long patches (over kTprof ticks; a shower's run over
// a hundred) or with more visits than kHeavyVisits -- for the second, whose
// blocks take 256 visits of a tile each: the heaviest tile of an event (a
// shower's core, a track along a wire) holds thousands of visits and ran on
// long after the others.  The parts of a tile are added in the grid itself as
// integers, and the block that finishes a tile turns it into charges.
//
// Long patches are taken a column at a time there: a warp takes 32 tick columns
// of the tile, a lane each, and 32 of the staged visits, and adds those that
// cross its columns to the groups' sums in registers, one shared atomic a group
// at the end (warps that owned their columns waited for the fullest ones at the
// chunk's barrier).  Their cells are the high words of integer products, group coefficient times scaled tick
// value, so no float-to-int conversion a cell (a quarter of a warp a cycle).
// 500k depos, half with patches of 100 ticks x 30 impacts, three planes: 2.8 ->
// 2.1 ms (heavy parts 1.85, at 43 % of the issue slots and 24 warps an SM).
constexpr int kWideG = 12;         // impact groups (wct_dt_set_response_table takes no more)
constexpr int kWideAhead = 4;      // visits whose tick values are loaded together
// (full APA, 520k track depos, fullest tile 3300: 478 us whole; 549 us with tiles
// over 1024 in parts, 744 us over 512: a part pays for its grid again)
constexpr int kHeavyVisits = 4096;
// The other tiles: two blocks' warps of visits and no more stay with the first
// launch (its 64-thread blocks: 11 an SM, a tile's chain of loads, staging and
// barriers is what takes the time), the rest are listed for blocks of 256.
// Whole, in 256-thread blocks -> so, us: plane 2k depos 55 -> 38, full APA on
// tracks 20k 165 -> 114, 100k 216 -> 180, 200k 256 -> 254, shower 200k (without
// the heavy parts) 180 -> 170, 16 batched events 594 -> 380.  Lines at 128, 256,
// 512 visits: 20k 117, 107, 108; 100k 174, 191, 209; batch + 40, + 23, + 91.
constexpr int kLightVisits = kLightThreads;
// Mean visits a tile over which one launch of 256-thread blocks is the faster
// form (full APA on tracks, 520k depos, 147 a tile: 418 against 442 us; 200k,
// 56 a tile: 256 against 254).
constexpr long long kDenseVisits = 96;
static_assert(kRasterThreads == kHeavyPart, "a part is a block's chunk");

// A tile without work in this launch: its G rows are zero. Of one without
// visits in a sparse grid the transform reads only the 16-byte pieces that it
// shares with a neighbour. (Half to two thirds of the tiles: their zeros took
// the raster 24 of 81 us at 2k depos on a plane, 42 of 213 at 20k on a full APA,
// 198 of 792 for 16 batched events.)
__device__ __forceinline__ void zero_tile(const GridPlane& P, int row, int qc0, bool unread, float* __restrict__ Q)
{
    if (unread) {
        const int o = qc0 & 3;
        if (o == 0) return;
        for (int k = threadIdx.x; k < P.G * 4; k += blockDim.x) {
            const int g = k >> 2, j = k & 3;
            const int qc = j < 4 - o ? qc0 + j : qc0 + kTile - 4 + j;
            if (qc >= 0 && qc < P.N) Q[P.qoff + ((size_t)g * P.nin + row) * P.N + qc] = 0.f;
        }
        return;
    }
    for (int k = threadIdx.x; k < P.G * kTile; k += blockDim.x) {
        const int g = k / kTile, qc = qc0 + k - g * kTile;
        if (qc >= 0 && qc < P.N) Q[P.qoff + ((size_t)g * P.nin + row) * P.N + qc] = 0.f;
    }
}

// One raster work item: charge row `row` (wire start_ch + row) of plane P and
// absolute tick tile ktile.  Visit keys are key_base + wire * ntiles_abs +
// tile; at most vcap visits exist.  HEAVY: part `seg` of the nseg parts of a
// heavy tile (slot: its entry of heavy.done); otherwise the whole tile, or its
// listing under tile_id.  Called by all threads of the block; smem_i holds the
// dynamic shared memory of raster_smem_bytes(P.G).
template <bool HEAVY, int T, bool LIST>
__device__ __forceinline__ void raster_tile(const GridPlane& P, int row, int ktile, int key_base, int ntiles_abs,
                                            const PatchRec* __restrict__ rec, const float* __restrict__ tprof,
                                            const TprofPool& pool, const unsigned char* __restrict__ wide_key,
                                            const int* __restrict__ wire_cnt, const int* __restrict__ wire_off,
                                            const Visit* __restrict__ visits, long long vcap,
                                            const unsigned long long* __restrict__ key_bound,
                                            float* __restrict__ Q, unsigned char* __restrict__ row_flag,
                                            const HeavyList& heavy, int tile_id, int seg, int nseg, int slot,
                                            int* smem_i, float* scale, float* iscale)
{
    __syncthreads();  // the previous item of a persistent block is done with the shared arrays
    const int w = P.start_ch + row;
    const int G = P.G, nimp = P.nimp;
    const int tick_lo = ktile * kTile;                      // absolute first tick of the tile
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    int* grid = smem_i;                                       // [G][kGridLd], column = tick - tick_lo
    float* stage = reinterpret_cast<float*>(smem_i + (size_t)G * kGridLd);
    int4* stagei = reinterpret_cast<int4*>(stage + (size_t)T * kStageStride);
    int4* longq = stagei + T;  // heavy parts only
    int cnt = 0, held = 1;
    const Visit* list = nullptr;
    int key = -1;
    if (w >= 0 && w < P.nwires && ktile >= 0 && ktile < ntiles_abs) {
        key = key_base + (P.wire_base + w) * ntiles_abs + ktile;
        const int off = wire_off[key];
        held = wire_cnt[key];
        cnt = off < 0 ? 0 : (int)min((long long)held, max(0ll, vcap - off));  // no reads past the list
        list = visits + max(off, 0);
    }
    const bool spread = cnt > 0 && wide_key[key];
    const bool longs = HEAVY && spread;  // the tile holds long patches
    if (LIST && !spread && cnt > kLightVisits && cnt <= kHeavyVisits && heavy.mid) {
        if (tid == 0) heavy.mid[atomicAdd(heavy.count + 2, 1)] = tile_id;
        return;
    }
    const bool listed = LIST && (spread || cnt > kHeavyVisits);
    if (listed) {
        const int parts = (cnt + kHeavyPart - 1) / kHeavyPart;
        if (tid == 0) {
            const int sl = atomicAdd(heavy.count + 1, 1), at = atomicAdd(heavy.count, parts);
            heavy.done[sl] = 0;
            for (int k = 0; k < parts; ++k) heavy.item[at + k] = make_int4(tile_id, k, parts, sl);
        }
        if (parts == 1) return;  // written whole by its only part
    }
    if (cnt == 0 || listed) {
        zero_tile(P, row, tick_lo - P.col0, P.sparse && held == 0, Q);  // no visit (block-uniform), or parts to come
        return;
    }
    if (tid == 0) row_flag[P.wire_base + w] = 1;  // the wire holds charge (every block of the row writes the same)
    if (HEAVY) {
        list += (size_t)seg * kHeavyPart;
        cnt = min(cnt - seg * kHeavyPart, kHeavyPart);
    }
    __shared__ int s_unit[1];
    {
        if (HEAVY && tid == 0) *s_unit = 0;
        int4* g4 = reinterpret_cast<int4*>(grid);
        const int n4 = G * kGridLd / 4;
        for (int k = tid; k < n4; k += T) g4[k] = make_int4(0, 0, 0, 0);
        if (tid < kTileBlocks) {
            const float b = key >= 0 ? __ull2float_ru(key_bound[(size_t)key * kTileBlocks + tid]) * (1.0f / 65536.0f)
                                     : 0.f;
            scale[tid] = b > 0.f ? 1073741824.0f / b : 0.f;
            iscale[tid] = b > 0.f ? b / 1073741824.0f : 0.f;
        }
    }
    __syncthreads();
    const float pbs = P.pbs, tbs = P.tbs;
    const int wlo = w * nimp;
    // each lane stages the group coefficients and tick values of one visit, then
    // the warp scatters its 32 staged visits, eight at a time
    float* my = stage + (size_t)tid * kStageStride;
    const int wbase = wid * 32;
    const float inv_pbs = 1.0f / pbs;
    const int nchunks = (cnt + T - 1) / T;
    for (int ch = 0; ch < nchunks; ++ch) {
        // visit of this thread: in blocks with long patches, lanes 2k, 2k+1
        // hold consecutive visits (a pair) and consecutive pairs go to
        // different warps (the lists hold one depo kind in runs: long patches
        // would otherwise pile up on a few warps); elsewhere a warp's visits are
        // neighbours in the list (coalesced reads, alike along a track)
        const int e = ch * T +
                      (longs ? (lane >> 1) * (T / 16) + wid * 2 + (lane & 1) : tid);
        const bool valid = e < cnt;
        int4 si = make_int4(0, 0, 0, 0);  // d, l_lo, ng, (cb << 11) | nt  (cb = toff - tick_lo, ng = 0: none)
        if (valid) {
            const int d = list[e];
            const PatchRec r = rec[P.recoff + d];
            const int rnp = r.np, rnt = r.nt;
            const int l_lo = max(r.poff, wlo) - wlo;
            const int l_hi = min(r.poff + rnp, wlo + nimp) - wlo;
            if (l_hi > l_lo) {
                const int ng = l_hi - l_lo + 1;
                if (r.sp > 0.f) {
                    const float isg = __frcp_rn(r.sp);
                    const float inv = 0.70710678118654752f * isg;            // 1/(sqrt2 sigma)
                    const float c0 = r.sp * inv_pbs * 0.39894228040143268f;  // sigma / (step*sqrt(2 pi))
                    const int k0 = wlo + l_lo - r.poff;
                    float x1 = (float)k0 * pbs - r.pcr;
                    float e1 = copysignf(erfc_nr(fabsf(x1 * inv)), x1);
                    float u1 = x1 * isg;
                    float g1 = __expf(-0.5f * u1 * u1);
                    // group lb gets p_lb * w_lb + p_(lb-1) * (1 - w_(lb-1)): the
                    // second term is carried in a register to the next bin
                    float carry = 0.f;
                    for (int lb = 0; lb < ng - 1; ++lb) {
                        const float x2 = (float)(k0 + lb + 1) * pbs - r.pcr;
                        const float e2 = copysignf(erfc_nr(fabsf(x2 * inv)), x2);
                        const float u2 = x2 * isg;
                        const float g2 = __expf(-0.5f * u2 * u2);
                        const float p = bin_from_edges(e1, e2);
                        const float wt = p > 0.f ? fmaf(c0 * (g2 - g1), __fdividef(1.0f, p), x2 * inv_pbs) : 0.0f;
                        my[lb] = carry + p * wt;
                        carry = p * (1.0f - wt);
                        e1 = e2;
                        g1 = g2;
                    }
                    my[ng - 1] = carry;
                }
                else {
                    const float wt = (pbs - r.pcr) * inv_pbs;
                    my[0] = wt;
                    my[1] = 1.0f - wt;
                }
                const int cb = r.toff - tick_lo;  // may be negative for patches starting in the previous tile
                si = make_int4(d, l_lo, ng, ((cb + 1024) << 11) | rnt);
                if (longs && rnt > kTprof) {
                    // the coefficients by impact group as integers, in units of 2^-30 of the peak
                    // bin fraction (a group's is below twice that), four times the charge times
                    // that fraction (the scaled tick values stay below 2^31: the bound behind
                    // the scale holds twice this product), and where the profile is
                    const float pm = peak_fraction(pbs, r.sp);
                    const float unit = __fdividef(1073741824.0f, pm);
                    int ci[kWideG];
#pragma unroll
                    for (int g = 0; g < kWideG; ++g) {
                        const int lb = g - l_lo;
                        ci[g] = lb >= 0 && lb < ng ? __float2int_rn(my[max(lb, 0)] * unit) : 0;
                    }
                    int4* lq = longq + tid * kLongQuads;
                    lq[0] = make_int4(si.w, __ldg(pool.off + d), __float_as_int(4.0f * r.qn * pm), d);
                    lq[1] = make_int4(ci[0], ci[1], ci[2], ci[3]);
                    lq[2] = make_int4(ci[4], ci[5], ci[6], ci[7]);
                    lq[3] = make_int4(ci[8], ci[9], ci[10], ci[11]);
                }
                if (rnt <= 16) {
                    // tick values scaled to the fixed point of their 64-tick block (0 outside the tile);
                    // the whole 16-value profile row in four 128-bit loads (one L1 wavefront per
                    // lane each, against one per value with scalar loads)
                    static_assert(kTprof == 16, "profile rows are four float4");
                    const float4* tp4 = reinterpret_cast<const float4*>(tprof + (size_t)d * kTprof);
                    float tv[16];
#pragma unroll
                    for (int k4 = 0; k4 < 4; ++k4) {
                        const float4 x = __ldg(tp4 + k4);
                        tv[4 * k4] = x.x;
                        tv[4 * k4 + 1] = x.y;
                        tv[4 * k4 + 2] = x.z;
                        tv[4 * k4 + 3] = x.w;
                    }
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        const int c = cb + k;
                        float v = 0.f;
                        if (k < rnt && c >= 0 && c < kTile) v = tv[k] * r.qn * scale[c / kScaleBlock];
                        my[kStageT + k] = v;
                    }
                }
            }
        }
        stagei[tid] = si;
        if (longs) __syncthreads();
        else __syncwarp();
        // lanes 0 .. nv-1 of this warp hold visits (e grows with the lane)
        const int nv = __popc(__ballot_sync(0xffffffffu, valid));
        // eight visits at a time: four lanes per visit, each lane four ticks (hl + 4k)
        const int qv = lane >> 2, hl = lane & 3;
        for (int v0 = 0; v0 < nv; v0 += 8) {
            const int v = v0 + qv;
            int4 vi = make_int4(0, 0, 0, 0);
            if (v < nv) vi = stagei[wbase + v];
            int nt = vi.w & 2047;
            if (longs && nt > kTprof) nt = 0;  // below
            const int ng = vi.z;
            const int c0 = (vi.w >> 11) - 1024 + hl;  // tile column of this lane's first tick
            const float* vc = stage + (size_t)(wbase + min(v, 31)) * kStageStride;
            float tq[4];
            int gl[4];  // groups this lane adds at tick hl + 4k (0: tick outside the patch or tile)
            int mgl = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int c = c0 + 4 * k;
                const bool on = hl + 4 * k < nt && c >= 0 && c < kTile;
                tq[k] = on ? vc[kStageT + hl + 4 * k] : 0.f;
                gl[k] = on ? ng : 0;
                mgl = max(mgl, gl[k]);
            }
            const int mg = __reduce_max_sync(0xffffffffu, mgl);
            // the eight visits start at spread-out groups and wrap around
            // (visit slot qv at group qv*ng/8): visits of one track share
            // their columns and would otherwise hit the same words together
            int gg = (qv * ng) >> 3;
            int* dst = grid + (vi.y + gg) * kGridLd + c0;
            int* const wrap = grid + vi.y * kGridLd + c0;
            int* const last = wrap + (ng - 1) * kGridLd;
            float cf = vc[gg];
            for (int g = 0; g < mg; ++g) {
                const bool w = dst == last;
                const int gn = w ? 0 : gg + 1;
                const float cfn = vc[gn];  // next group's coefficient, loaded ahead
                int v4[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) v4[k] = __float2int_rn(cf * tq[k]);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (g < gl[k]) atomicAdd(dst + 4 * k, v4[k]);
                dst = w ? wrap : dst + kGridLd;
                gg = gn;
                cf = cfn;
            }
        }
        if (longs) {
            // units of 32 columns x 32 staged visits, taken in turn by whichever warp is free
            for (;;) {
                int unit = 0;
                if (lane == 0) unit = atomicAdd(s_unit, 1);
                unit = __shfl_sync(0xffffffffu, unit, 0);
                if (unit >= (kTile / 32) * (T / 32)) break;
                const int slab = unit & (kTile / 32 - 1), b0 = (unit / (kTile / 32)) * 32;
                const int c = slab * 32 + lane;  // this lane's column
                const float sc = scale[c / kScaleBlock];
                const int4 si0 = stagei[b0 + lane];
                const int cb0 = (si0.w >> 11) - 1024, nt0 = si0.w & 2047;
                unsigned m = __ballot_sync(0xffffffffu, si0.z > 0 && nt0 > kTprof && cb0 < slab * 32 + 32 &&
                                                            cb0 + nt0 > slab * 32);
                if (!m) continue;
                int acc[kWideG];
#pragma unroll
                for (int g = 0; g < kWideG; ++g) acc[g] = 0;
                // tick values of the next few visits, asked for while the last few are added
                int vn[kWideAhead];
                float tn[kWideAhead];
                auto ask = [&]() {
#pragma unroll
                    for (int a = 0; a < kWideAhead; ++a) {
                        vn[a] = m ? b0 + __ffs(m) - 1 : -1;
                        m &= m - 1;
                        tn[a] = 0.f;
                        if (vn[a] >= 0) {
                            const int4 lv = longq[vn[a] * kLongQuads];
                            const int it = c - ((lv.x >> 11) - 1024);
                            if (it >= 0 && it < (lv.x & 2047)) {
                                if (lv.y >= 0) tn[a] = __ldg(pool.val + lv.y + it);
                                else {
                                    const PatchRec r = rec[P.recoff + lv.w];
                                    tn[a] = unit_bin(it, tbs, r.tcr, r.st);
                                }
                            }
                        }
                    }
                };
                ask();
                while (vn[0] >= 0) {
                    int vs[kWideAhead];
                    float tv[kWideAhead];
#pragma unroll
                    for (int a = 0; a < kWideAhead; ++a) {
                        vs[a] = vn[a];
                        tv[a] = tn[a];
                    }
                    ask();
#pragma unroll
                    for (int a = 0; a < kWideAhead; ++a) {
                        if (vs[a] < 0) break;
                        const int4* lq = longq + vs[a] * kLongQuads;
                        const int tq = __float2int_rn(tv[a] * __int_as_float(lq[0].z) * sc);
#pragma unroll
                        for (int q = 0; q < kWideG / 4; ++q) {
                            const int4 ci = lq[1 + q];
                            // rounded high words of the products
                            acc[4 * q] += (int)(((long long)ci.x * tq + 0x80000000ll) >> 32);
                            acc[4 * q + 1] += (int)(((long long)ci.y * tq + 0x80000000ll) >> 32);
                            acc[4 * q + 2] += (int)(((long long)ci.z * tq + 0x80000000ll) >> 32);
                            acc[4 * q + 3] += (int)(((long long)ci.w * tq + 0x80000000ll) >> 32);
                        }
                    }
                }
#pragma unroll
                for (int g = 0; g < kWideG; ++g)
                    if (g < G) atomicAdd(grid + g * kGridLd + c, acc[g]);
            }
            __syncthreads();  // the stage is rewritten by the next chunk
        }
        else
            __syncwarp();
    }
    __syncthreads();
    if (HEAVY && nseg > 1) {
        // this part into the tile's rows, as integers; the last part to arrive makes them charges
        const int qc0 = tick_lo - P.col0;
        int* const Qi = reinterpret_cast<int*>(Q) + P.qoff + (size_t)row * P.N;
        for (int k = tid; k < G * kTile; k += T) {
            const int g = k / kTile, c = k - g * kTile, q = qc0 + c;
            const int v = grid[g * kGridLd + c];
            if (v && q >= 0 && q < min(P.N, P.ncols)) atomicAdd(Qi + (size_t)g * P.nin * P.N + q, v);
        }
        __threadfence();
        __syncthreads();
        __shared__ int s_last;
        if (tid == 0) s_last = atomicAdd(heavy.done + slot, 1) == nseg - 1;
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        for (int k = tid; k < G * kTile; k += T) {
            const int g = k / kTile, c = k - g * kTile, q = qc0 + c;
            if (q < 0 || q >= min(P.N, P.ncols)) continue;
            int* const at = Qi + (size_t)g * P.nin * P.N + q;
            *reinterpret_cast<float*>(at) = (float)__ldcg(at) * iscale[c / kScaleBlock];
        }
        return;
    }
    // write the tile's G rows, a column per thread (a warp's 128 bytes together: quads of
    // columns per thread left as 4-byte pieces of 16 sectors): grid column c is plane column
    // tick_lo + c - col0 (zero at or past the window's ncols)
    const size_t gs = (size_t)P.nin * P.N;
    for (int c = tid; c < kTile; c += T) {
        const int q = tick_lo - P.col0 + c;
        if (q < 0 || q >= P.N) continue;
        const float is = q < P.ncols ? iscale[c / kScaleBlock] : 0.f;
        float* dst = Q + P.qoff + (size_t)row * P.N + q;
#pragma unroll 4
        for (int g = 0; g < G; ++g, dst += gs) *dst = (float)grid[g * kGridLd + c] * is;
    }
}

// The plane and the (row, tile) of a block of the tile grid.
__device__ __forceinline__ int grid_tile(const GridSet& gs, int tile, int& row, int& ktile)
{
    int ip = 0;
    while (ip + 1 < gs.nplanes && tile >= gs.p[ip + 1].row_base) ++ip;
    const GridPlane& P = gs.p[ip];
    const int rel = tile - P.row_base;
    row = rel / P.ntile;
    ktile = P.ktile0 + (rel - row * P.ntile);  // absolute tick tile
    return ip;
}

template <int T>
__global__ void __launch_bounds__(T, T == kLightThreads ? kLightBlocks : kMidBlocks)
    k_raster_wires(const PatchRec* __restrict__ rec, const float* __restrict__ tprof,
                   const int* __restrict__ wire_cnt, const int* __restrict__ wire_off,
                   const Visit* __restrict__ visits, long long vcap, const unsigned long long* __restrict__ key_bound,
                   GridSet gs, float* __restrict__ Q, TprofPool pool, const unsigned char* __restrict__ wide_key,
                   unsigned char* __restrict__ row_flag, HeavyList heavy)
{
    extern __shared__ int smem_i[];
    __shared__ float scale[kTileBlocks], iscale[kTileBlocks];
    int row, ktile;
    const int ip = grid_tile(gs, blockIdx.x, row, ktile);
    raster_tile<false, T, true>(gs.p[ip], row, ktile, 0, gs.ntiles_abs, rec, tprof, pool, wide_key, wire_cnt, wire_off,
                                visits, vcap, key_bound, Q, row_flag, heavy, blockIdx.x, 0, 1, 0, smem_i, scale, iscale);
}

// The next of the listed middling tiles, -1 after the last (block-uniform).
__device__ __forceinline__ int next_mid(const HeavyList& heavy)
{
    __shared__ int s_next;
    __syncthreads();
    if (threadIdx.x == 0) s_next = atomicAdd(heavy.count + 3, 1);
    __syncthreads();
    return s_next < heavy.count[2] ? heavy.mid[s_next] : -1;
}

__global__ void __launch_bounds__(kRasterThreads, kMidBlocks)
    k_raster_mid(const PatchRec* __restrict__ rec, const float* __restrict__ tprof,
                 const int* __restrict__ wire_cnt, const int* __restrict__ wire_off,
                 const Visit* __restrict__ visits, long long vcap, const unsigned long long* __restrict__ key_bound,
                 GridSet gs, float* __restrict__ Q, TprofPool pool, const unsigned char* __restrict__ wide_key,
                 unsigned char* __restrict__ row_flag, HeavyList heavy)
{
    extern __shared__ int smem_i[];
    __shared__ float scale[kTileBlocks], iscale[kTileBlocks];
    for (int it = next_mid(heavy); it >= 0; it = next_mid(heavy)) {
        int row, ktile;
        const int ip = grid_tile(gs, it, row, ktile);
        raster_tile<false, kRasterThreads, false>(gs.p[ip], row, ktile, 0, gs.ntiles_abs, rec, tprof, pool, wide_key,
                                                  wire_cnt, wire_off, visits, vcap, key_bound, Q, row_flag, heavy, it,
                                                  0, 1, 0, smem_i, scale, iscale);
    }
}

__global__ void __launch_bounds__(kRasterThreads, kHeavyBlocks)
    k_raster_heavy(const PatchRec* __restrict__ rec, const float* __restrict__ tprof,
                   const int* __restrict__ wire_cnt, const int* __restrict__ wire_off,
                   const Visit* __restrict__ visits, long long vcap, const unsigned long long* __restrict__ key_bound,
                   GridSet gs, float* __restrict__ Q, TprofPool pool, const unsigned char* __restrict__ wide_key,
                   unsigned char* __restrict__ row_flag, HeavyList heavy)
{
    extern __shared__ int smem_i[];
    __shared__ float scale[kTileBlocks], iscale[kTileBlocks];
    const int total = heavy.count[0];
    for (int k = blockIdx.x; k < total; k += gridDim.x) {
        const int4 it = heavy.item[k];
        int row, ktile;
        const int ip = grid_tile(gs, it.x, row, ktile);
        raster_tile<true, kRasterThreads, false>(gs.p[ip], row, ktile, 0, gs.ntiles_abs, rec, tprof, pool, wide_key, wire_cnt, wire_off,
                          visits, vcap, key_bound, Q, row_flag, heavy, it.x, it.y, it.z, it.w, smem_i, scale, iscale);
    }
}

int launch_raster_wires(const PatchRec* rec, const float* tprof, const TprofPool& pool, const unsigned char* wide_key,
                         const int* wire_cnt,
                         const int* wire_off, const Visit* visits, long long vcap,
                         const unsigned long long* key_bound, const GridSet& gs, float* Q, unsigned char* row_flag,
                         const HeavyList& heavy, int nsm, cudaStream_t s)
{
    if (gs.nrows_total <= 0) return 0;
    int maxG = 0;
    for (int i = 0; i < gs.nplanes; ++i) maxG = std::max(maxG, gs.p[i].G);
    const bool dense = vcap > kDenseVisits * gs.nrows_total;
    const int T = dense ? kRasterThreads : kLightThreads;
    auto* light = dense ? k_raster_wires<kRasterThreads> : k_raster_wires<kLightThreads>;
    HeavyList lists = heavy;
    if (dense) lists.mid = nullptr;
    size_t smem = raster_smem(maxG, T);
    cudaFuncSetAttribute((const void*)light, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    light<<<gs.nrows_total, T, smem, s>>>(rec, tprof, wire_cnt, wire_off, visits, vcap, key_bound, gs, Q, pool,
                                          wide_key, row_flag, lists);
    if (nsm <= 0) return 1;  // no tile can be listed
    if (!dense) {
        smem = raster_smem_bytes(maxG);
        cudaFuncSetAttribute((const void*)k_raster_mid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        k_raster_mid<<<kMidBlocks * nsm, kRasterThreads, smem, s>>>(rec, tprof, wire_cnt, wire_off, visits, vcap,
                                                                    key_bound, gs, Q, pool, wide_key, row_flag, heavy);
    }
    smem = raster_heavy_smem_bytes(maxG);
    cudaFuncSetAttribute((const void*)k_raster_heavy, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_raster_heavy<<<kHeavyBlocks * nsm, kRasterThreads, smem, s>>>(rec, tprof, wire_cnt, wire_off, visits, vcap, key_bound,
                                                              gs, Q, pool, wide_key, row_flag, heavy);
    return dense ? 2 : 3;
}

// ---------------------------------------------------------------------------
// Fluctuated patches (GaussianDiffusion::set_sampling with an IRandom,
// gen/src/GaussianDiffusion.cxx:184-213): every cell (k, tau) of a patch is
// redrawn as N ~ Binomial((int)|Q|, p_k t_tau / (sum p * sum t)) and the
// patch is rescaled by Q / sum N; a patch whose draws are all zero adds
// nothing.  The draws are counter-based: k_fluc_sums draws every cell to get
// sum N and keeps the draws for the fluctuated raster; cells past the room for
// them are drawn again there.  The unit bin integrals that set each cell's
// probability come from one non-inlined function with explicitly rounded
// operations, so both see the same probabilities bit for bit and therefore the
// same draws.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int event_of_depo(const EventTable& et, int i)
{
    int lo = 0, hi = et.nev - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (et.dep0[mid] <= i) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The draw of cell (k, tau) of depo i_ev (index within its event) on plane ip.
__device__ __forceinline__ int cell_draw(const FlucParams& fp, int ident, int i_ev, int ip, int cell, int nq,
                                         float relval)
{
    Philox g;
    g.init(fp.key0, fp.key1 + 0x9E3779B9u * (unsigned)ident, (unsigned)i_ev, (unsigned)ip, (unsigned)cell);
    return binomial(nq, (double)relval, g);
}

// The draws of every patch's cells, stored for the raster, and their sums: one
// warp per (plane, four depos).
//
// What bounds it: the arithmetic of the draws.  Cells of a patch differ in the
// sampler they need (inversion below a mean of 10, BTRS above) and in how far
// it goes, so a warp that drew its cells in order had 9 of 32 lanes at work, in
// double precision, and the raster drew all of them a second time (3.3 + 5.1 ms
// for 100k depos on three planes, 40 M cells).  Here cells are sorted into
// small queues of the warp -- inversion, BTRS squeeze, BTRS full test -- and a
// queue is worked off when it holds a whole warp's worth; four patches share
// the queues, so that few are worked off part full, and the lanes of one pass
// over their bin integrals.  The transcendentals are in single precision where
// that decides the draw (rng.cuh).  Now 1.9 ms, and 1.1 ms of raster.
constexpr int kFlucWarps = 4;
constexpr int kFlucSlots = 4;      // depos of a warp
constexpr int kFlucTab = 2048;     // bin integrals of a warp (one patch: at most kMaxPatchP + kMaxPatchT)
constexpr int kFlucQueue = 64;     // a queue holds at most 31 cells when another 32 come
constexpr unsigned kNoCell = 0xffffffffu;
static_assert(kFlucTab >= kMaxPatchP + kMaxPatchT, "one patch fits the tables");

struct FlucSlot {
    float invS;
    int nq, nt, i_ev;
    unsigned key1;
    int pbase, tbase;  // its pitch and time integrals in the table
    int* store;        // its draws, or null
};

__global__ void __launch_bounds__(kFlucWarps * 32, 6) k_fluc_sums(const PatchRec* __restrict__ rec, EventTable evt,
                                                                  PlaneSet ps, float tbs, FlucParams fp,
                                                                  const double* __restrict__ fq,
                                                                  FlucRec* __restrict__ fluc, DrawPool draws,
                                                                  int* status)
{
    __shared__ float s_tab[kFlucWarps][kFlucTab];
    __shared__ unsigned s_q[kFlucWarps][3][kFlucQueue];
    __shared__ FlucSlot s_slot[kFlucWarps][kFlucSlots];
    const unsigned full = 0xffffffffu;
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = evt.dep0[evt.nev], groups = (n + kFlucSlots - 1) / kFlucSlots;
    const long long gw = (long long)blockIdx.x * kFlucWarps + wib;
    if (gw >= (long long)groups * ps.nplanes) return;  // whole warps only; no block barrier follows
    const int ip = (int)(gw / groups), i0 = (int)(gw - (long long)ip * groups) * kFlucSlots;
    const float pbs = (float)ps.p[ip].imp_bs;
    float* const tab = s_tab[wib];
    FlucSlot* const slot = s_slot[wib];
    // lanes 0 .. 3 own a depo each: its record, room for its draws, its normalisation
    const int mine = i0 + lane;
    const bool own = lane < kFlucSlots && mine < n;
    PatchRec r{};
    FlucRec out{0, 0.f, 0.f, -1};
    double Q = 0.0;
    int i_ev = 0;
    unsigned key1 = 0;
    if (own) {
        r = rec[(size_t)ip * n + mine];
        if (r.np > 0 && r.nt > 0) {
            out.invS = patch_inv_norm(r, pbs, tbs);
            Q = fq[(size_t)ip * n + mine];
            out.nq = (int)fabs(Q);
            const int ev = event_of_depo(evt, mine);
            i_ev = mine - evt.dep0[ev];
            key1 = fp.key1 + 0x9E3779B9u * (unsigned)fluc_ident(fp, ev);
        }
        else
            r.np = r.nt = 0;
    }
    {  // room for the warp's draws in one go (one address: see k_prep_all)
        const long long mycells = (long long)r.np * r.nt;
        long long before = 0, all = 0;
#pragma unroll
        for (int s = 0; s < kFlucSlots; ++s) {
            const long long c = __shfl_sync(full, mycells, s);
            if (s < lane) before += c;
            all += c;
        }
        long long off = 0;
        if (lane == 0 && all) off = (long long)atomicAdd(draws.used, (unsigned long long)all);
        off = __shfl_sync(full, off, 0) + before;
        if (mycells) {
            if (off + mycells <= draws.cap) out.off = (int)off;
            else if (status) atomicOr(status, kBatchDrawsShort);
        }
    }
    const int size = own ? r.np + r.nt : 0;
    const unsigned key0 = fp.key0;
    long long sum_mine = 0;
    for (int s0 = 0; s0 < kFlucSlots;) {
        // as many of the slots s0 .. s1-1 as the table holds (one always fits)
        int s1 = s0, used = 0, pre[kFlucSlots + 1], cells[kFlucSlots + 1], pbase = 0;
        pre[0] = cells[0] = 0;
#pragma unroll
        for (int s = 0; s < kFlucSlots; ++s) {
            const int sz = __shfl_sync(full, size, s), nc = __shfl_sync(full, (int)r.np * (int)r.nt, s);
            const bool take = s >= s0 && s == s1 && used + sz <= kFlucTab;
            if (take) {
                if (lane == s) pbase = used;
                used += sz;
                ++s1;
            }
            pre[s + 1] = used;
            cells[s + 1] = cells[s] + (take ? nc : 0);
        }
        __syncwarp();
        if (lane >= s0 && lane < s1 && own)
            slot[lane] = FlucSlot{out.invS, out.nq, r.nt, i_ev, key1, pbase, pbase + r.np,
                                  out.off >= 0 ? draws.val + out.off : nullptr};
        // unit bin integrals of all the taken patches, over the lanes
        for (int b0 = 0; b0 < used; b0 += 32) {
            const int b = b0 + lane;
            int s = s0;
#pragma unroll
            for (int q = 0; q + 1 < kFlucSlots; ++q)
                if (q >= s0 && q + 1 < s1 && b >= pre[q + 1]) s = q + 1;
            const int np = __shfl_sync(full, (int)r.np, s);
            const float pcr = __shfl_sync(full, r.pcr, s), sp = __shfl_sync(full, r.sp, s);
            const float tcr = __shfl_sync(full, r.tcr, s), st = __shfl_sync(full, r.st, s);
            int first = 0;
#pragma unroll
            for (int q = 0; q < kFlucSlots; ++q)
                if (q == s) first = pre[q];
            if (b < used) {
                const int k = b - first;
                tab[b] = k < np ? unit_bin(k, pbs, pcr, sp) : unit_bin(k - np, tbs, tcr, st);
            }
        }
        __syncwarp();
        // a cell: slot, bin and tick in one word
        long long sum[kFlucSlots] = {0, 0, 0, 0};
        int cnt[3] = {0, 0, 0};
        auto rel_of = [&](unsigned e) {
            const FlucSlot& S = slot[e >> 30];
            return __fmul_rn(__fmul_rn(tab[S.pbase + ((e >> 15) & 0x7fffu)], tab[S.tbase + (e & 0x7fffu)]), S.invS);
        };
        auto cell_of = [&](unsigned e) { return ((e >> 15) & 0x7fffu) * slot[e >> 30].nt + (e & 0x7fffu); };
        auto put = [&](unsigned e, int N) {
#pragma unroll
            for (int s = 0; s < kFlucSlots; ++s)
                if ((int)(e >> 30) == s) sum[s] += N;
            int* const st = slot[e >> 30].store;
            if (st) st[cell_of(e)] = N;
        };
        auto block_of = [&](unsigned e, unsigned at) {
            const FlucSlot& S = slot[e >> 30];
            return philox_block(key0, S.key1, (unsigned)S.i_ev, (unsigned)ip, cell_of(e), at);
        };
        auto again = [&](unsigned e) {  // the double-precision draw
            const FlucSlot& S = slot[e >> 30];
            Philox g;
            g.init(key0, S.key1, (unsigned)S.i_ev, (unsigned)ip, cell_of(e));
            return binomial_double(S.nq, (double)rel_of(e), g);
        };
        auto push = [&](int q, bool on, unsigned e) {
            const unsigned m = __ballot_sync(full, on);
            if (on) s_q[wib][q][cnt[q] + __popc(m & ((1u << lane) - 1u))] = e;
            cnt[q] += __popc(m);
            __syncwarp();
        };
        // the last m cells of queue q, one a lane
        auto pop = [&](int q, int m, unsigned& e) {
            cnt[q] -= m;
            const bool on = lane < m;
            e = on ? s_q[wib][q][cnt[q] + lane] : 0u;
            __syncwarp();
            return on;
        };
        const int ncell = cells[kFlucSlots];
        for (int c0 = 0; c0 < ncell; c0 += 32) {
            const int c = c0 + lane;
            int kind = -1;  // 0 inversion, 1 BTRS, 2 the full test's queue; -1 settled here
            unsigned e = 0;
            if (c < ncell) {
                int s = s0, first = 0;
#pragma unroll
                for (int q = 0; q < kFlucSlots; ++q)
                    if (q >= s0 && q < s1 && c >= cells[q]) s = q, first = cells[q];
                const int nt = slot[s].nt, nq = slot[s].nq;
                // bin = c / nt: (c - first + 1/2) / nt is 1/(2 nt) or more from an integer
                const int k = (int)(((float)(c - first) + 0.5f) * __fdividef(1.0f, (float)nt));
                e = ((unsigned)s << 30) | ((unsigned)k << 15) | (unsigned)(c - first - k * nt);
                const float rel = rel_of(e);
                if (nq <= 0 || !(rel > 0.f)) put(e, 0);
                else if (rel >= 1.f) put(e, nq);
                else if (rel > 0.5f) kind = 2;
                else kind = (double)nq * (double)rel < 10.0 ? 0 : 1;
            }
            __syncwarp();
            push(0, kind == 0, e);
            push(1, kind == 1, e);
            push(2, kind == 2, e);
            // work off the full queues, every queue after the last cells (each
            // sampler stands here once: its code is what fills the instruction cache)
            const int least = c0 + 32 >= ncell ? 1 : 32;
            for (;;) {
                unsigned x, doubt = kNoCell;  // doubt: a cell for the double-precision draw
                int N;
                if (cnt[1] >= least && cnt[2] < 32) {
                    const bool on = pop(1, min(32, cnt[1]), x);
                    N = 0;
                    if (on) {
                        const uint4 o = block_of(x, 0u);
                        N = draw_btrs<true>(slot[x >> 30].nq, (double)rel_of(x), uniform53(o.x, o.y) - 0.5,
                                            (float)uniform53(o.z, o.w));
                        if (N >= 0) put(x, N);
                    }
                    push(2, on && N < 0, x);  // open, out of range or in doubt
                }
                else if (cnt[2] >= least) {
                    if (pop(2, min(32, cnt[2]), x)) {
                        const double p = (double)rel_of(x);
                        N = p <= 0.5 && (double)slot[x >> 30].nq * p >= 10.0 ? kDrawReject : kDrawDoubt;
                        for (unsigned at = 0; at < 8 && N == kDrawReject; ++at) {
                            const uint4 o = block_of(x, at);
                            N = draw_btrs<false>(slot[x >> 30].nq, p, uniform53(o.x, o.y) - 0.5,
                                                 (float)uniform53(o.z, o.w));
                        }
                        if (N >= 0) put(x, N);
                        else doubt = x;
                    }
                }
                else if (cnt[0] >= least) {
                    if (pop(0, min(32, cnt[0]), x)) {
                        const uint4 o = block_of(x, 0u);
                        N = draw_inversion(slot[x >> 30].nq, rel_of(x), (float)uniform53(o.x, o.y));
                        if (N >= 0) put(x, N);
                        else doubt = x;
                    }
                }
                else
                    break;
                if (doubt != kNoCell) put(doubt, again(doubt));  // rare
                __syncwarp();
            }
        }
#pragma unroll
        for (int s = 0; s < kFlucSlots; ++s) {
            if (s < s0 || s >= s1) continue;
            long long t = sum[s];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(full, t, o);
            if (lane == s) sum_mine = t;
        }
        s0 = s1;
    }
    if (own) {
        out.scale = sum_mine > 0 ? (float)(Q / (double)sum_mine) : 0.f;
        fluc[(size_t)ip * n + mine] = out;
    }
}

void launch_fluc_sums(const PatchRec* rec, const EventTable& et, const PlaneSet& ps, float tbs, const FlucParams& fp,
                      const double* fq, FlucRec* fluc, const DrawPool& draws, int* status, cudaStream_t s)
{
    const long long warps = (long long)((et.dep0[et.nev] + kFlucSlots - 1) / kFlucSlots) * ps.nplanes;
    if (warps <= 0) return;
    const long long blocks = (warps + kFlucWarps - 1) / kFlucWarps;
    k_fluc_sums<<<(unsigned)blocks, kFlucWarps * 32, 0, s>>>(rec, et, ps, tbs, fp, fq, fluc, draws, status);
}

// Fluctuated raster of one (charge row, tick tile) item: one warp per visit,
// its stored draws spread over the lanes (8, 16 or 32 ticks of a bin side by
// side); cell charges N * Q / sum N split between the two impact groups of the
// bin by its linear weight (BinnedDiffusion_transform.cxx:296-367).
// Accumulation in 64-bit fixed point (2^-16 electron), so the grid does not
// depend on the order of the adds.
constexpr int kFlucRasterThreads = 256;
constexpr float kFlucFix = 65536.0f;

size_t raster_fluc_smem_bytes(int G) { return sizeof(long long) * (size_t)G * kTileLd; }

// A cell of a patch whose draws were not stored: the same draw again.
__device__ __noinline__ int redraw_cell(const FlucParams& fp, int ident, int i_ev, int ip, const PatchRec& r,
                                        const FlucRec& fr, int k, int t, float pbs, float tbs)
{
    const float relval = __fmul_rn(__fmul_rn(unit_bin(k, pbs, r.pcr, r.sp), unit_bin(t, tbs, r.tcr, r.st)), fr.invS);
    return cell_draw(fp, ident, i_ev, ip, k * r.nt + t, fr.nq, relval);
}

__device__ __forceinline__ void raster_tile_fluc(const GridPlane& P, int ip, int row, int ktile, int key_base,
                                                 int ntiles_abs, const EventTable& evt, const FlucParams& fp,
                                                 const PatchRec* __restrict__ rec, const FlucRec* __restrict__ fluc,
                                                 const int* __restrict__ draws, const int* __restrict__ wire_cnt,
                                                 const int* __restrict__ wire_off, const Visit* __restrict__ visits,
                                                 long long vcap, float* __restrict__ Q,
                                                 unsigned char* __restrict__ row_flag, long long* grid)
{
    __syncthreads();  // the previous item of a persistent block is done with the grid
    __shared__ float s_w[kFlucRasterThreads / 32][16];
    const int w = P.start_ch + row;
    const int G = P.G, nimp = P.nimp;
    const int tick_lo = ktile * kTile;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nwarps = blockDim.x >> 5;
    int cnt = 0, held = 1;
    const Visit* list = nullptr;
    if (w >= 0 && w < P.nwires && ktile >= 0 && ktile < ntiles_abs) {
        const int key = key_base + (P.wire_base + w) * ntiles_abs + ktile;
        const int off = wire_off[key];
        held = wire_cnt[key];
        cnt = off < 0 ? 0 : (int)min((long long)held, max(0ll, vcap - off));
        list = visits + max(off, 0);
    }
    const int qc0 = tick_lo - P.col0;
    if (cnt == 0) {  // no visit (block-uniform)
        zero_tile(P, row, qc0, P.sparse && held == 0, Q);
        return;
    }
    if (tid == 0) row_flag[P.wire_base + w] = 1;
    for (int k = tid; k < G * kTileLd; k += blockDim.x) grid[k] = 0;
    __syncthreads();
    const float pbs = P.pbs, tbs = P.tbs, inv_pbs = 1.0f / pbs;
    const int wlo = w * nimp;
    for (int e = wid; e < cnt; e += nwarps) {
        const int d = list[e];
        const FlucRec fr = fluc[P.recoff + d];
        const PatchRec r = rec[P.recoff + d];
        const int rnp = r.np, rnt = r.nt;
        const int l_lo = max(r.poff, wlo) - wlo, l_hi = min(r.poff + rnp, wlo + nimp) - wlo;
        if (fr.scale == 0.f || l_hi <= l_lo) continue;  // warp-uniform
        const int nb = l_hi - l_lo;
        const int k0 = wlo + l_lo - r.poff;  // first patch bin on this wire
        if (lane < nb) {
            const int k = k0 + lane;
            float wt;
            if (r.sp > 0.f) {
                const float p = unit_bin(k, pbs, r.pcr, r.sp);
                const float isg = __frcp_rn(r.sp);
                const float x1 = (float)k * pbs - r.pcr, x2 = (float)(k + 1) * pbs - r.pcr;
                const float g1 = __expf(-0.5f * (x1 * isg) * (x1 * isg)), g2 = __expf(-0.5f * (x2 * isg) * (x2 * isg));
                const float c0 = r.sp * inv_pbs * 0.39894228040143268f;
                wt = p > 0.f ? fmaf(c0 * (g2 - g1), __frcp_rn(p), x2 * inv_pbs) : 0.f;
            }
            else wt = (pbs - r.pcr) * inv_pbs;
            s_w[wid][lane] = wt;
        }
        __syncwarp();
        const int cb = r.toff - tick_lo;
        const int tstart = max(0, -cb), tend = min(rnt, kTile - cb);
        const int ntt = tend - tstart;
        if (ntt > 0) {  // warp-uniform
            int ident = 0, i_ev = 0;
            if (fr.off < 0) {
                const int ev = event_of_depo(evt, d);
                ident = fluc_ident(fp, ev);
                i_ev = d - evt.dep0[ev];
            }
            const int lg = ntt <= 8 ? 3 : (ntt <= 16 ? 4 : 5);  // ticks side by side: 8, 16 or 32
            const int sub = lane >> lg, tl = lane & ((1 << lg) - 1), nsub = 32 >> lg;
            for (int b = sub; b < nb; b += nsub) {
                const float wb = s_w[wid][b];
                for (int tt = tl; tt < ntt; tt += 32) {
                    const int t = tstart + tt, k = k0 + b;
                    const int N = fr.off >= 0 ? __ldg(draws + fr.off + k * rnt + t)
                                              : redraw_cell(fp, ident, i_ev, ip, r, fr, k, t, pbs, tbs);
                    if (N) {
                        const float c = (float)N * fr.scale;
                        const float a = c * wb;
                        long long* dst = grid + (size_t)(l_lo + b) * kTileLd + cb + t;
                        atomicAdd(reinterpret_cast<unsigned long long*>(dst),
                                  (unsigned long long)__float2ll_rn(a * kFlucFix));
                        atomicAdd(reinterpret_cast<unsigned long long*>(dst + kTileLd),
                                  (unsigned long long)__float2ll_rn((c - a) * kFlucFix));
                    }
                }
            }
        }
        __syncwarp();
    }
    __syncthreads();
    for (int k = tid; k < G * kTile; k += blockDim.x) {
        const int g = k / kTile, c = k - g * kTile;
        const int qc = qc0 + c;
        if (qc < 0 || qc >= P.N) continue;
        float val = 0.f;
        if (tick_lo + c - P.col0 < P.ncols) val = (float)((double)grid[g * kTileLd + c] * (1.0 / 65536.0));
        Q[P.qoff + ((size_t)g * P.nin + row) * P.N + qc] = val;
    }
}

__global__ void __launch_bounds__(kFlucRasterThreads, 4) k_raster_fluc(const PatchRec* __restrict__ rec,
                                                                    const FlucRec* __restrict__ fluc,
                                                                    const int* __restrict__ draws, FlucParams fp,
                                                                    EventTable evt,
                                                                    const int* __restrict__ wire_cnt,
                                                                    const int* __restrict__ wire_off,
                                                                    const Visit* __restrict__ visits, long long vcap,
                                                                    GridSet gs, float* __restrict__ Q,
                                                                    unsigned char* __restrict__ row_flag)
{
    extern __shared__ long long grid64[];
    int ip = 0;
    while (ip + 1 < gs.nplanes && (int)blockIdx.x >= gs.p[ip + 1].row_base) ++ip;
    const GridPlane& P = gs.p[ip];
    const int rel = blockIdx.x - P.row_base;
    const int row = rel / P.ntile;
    const int ktile = P.ktile0 + (rel - row * P.ntile);
    raster_tile_fluc(P, ip, row, ktile, 0, gs.ntiles_abs, evt, fp, rec, fluc, draws, wire_cnt, wire_off, visits, vcap, Q,
                     row_flag, grid64);
}

void launch_raster_fluc(const PatchRec* rec, const FlucRec* fluc, const int* draws, const FlucParams& fp,
                        const EventTable& evt,
                        const int* wire_cnt, const int* wire_off, const Visit* visits, long long vcap,
                        const GridSet& gs, float* Q, unsigned char* row_flag, cudaStream_t s)
{
    if (gs.nrows_total <= 0) return;
    size_t smem = 0;
    for (int i = 0; i < gs.nplanes; ++i) smem = std::max(smem, raster_fluc_smem_bytes(gs.p[i].G));
    cudaFuncSetAttribute((const void*)k_raster_fluc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_raster_fluc<<<gs.nrows_total, kFlucRasterThreads, smem, s>>>(rec, fluc, draws, fp, evt, wire_cnt, wire_off, visits,
                                                                     vcap, gs, Q, row_flag);
}

// Independent Binomial(n, p) draws: out[i] from the stream of key (seed,
// ident) and counter (i, kRngSampleTag, 0) -- IRandom::binomial in bulk.
__global__ void k_binomial_samples(unsigned int key0, unsigned int key1, int n, double p, long long count,
                                   int* __restrict__ out)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x) {
        Philox g;
        g.init(key0, key1, (unsigned)(i & 0xffffffffll), kRngSampleTag, (unsigned)(i >> 32));
        out[i] = binomial(n, p, g);
    }
}

void launch_binomial_samples(unsigned long long seed, int ident, int n, double p, long long count, int* out,
                             cudaStream_t s)
{
    if (count <= 0) return;
    const unsigned key0 = (unsigned)(seed & 0xffffffffull);
    const unsigned key1 = (unsigned)(seed >> 32) + 0x9E3779B9u * (unsigned)ident;
    const long long blocks = std::min<long long>((count + 255) / 256, 148LL * 32);
    k_binomial_samples<<<(unsigned)blocks, 256, 0, s>>>(key0, key1, n, p, count, out);
}

// ---------------------------------------------------------------------------
// Real FFT of rows (forward), packed output.  One row per block.
// ---------------------------------------------------------------------------
// One row: x (in_len real values, zero padded to 2M) -> o (M packed bins).
// Called by all threads of the block; sm holds 2M complex values.
__device__ __forceinline__ void rfft_row(const float* x, int in_len, float2* o, const FftDesc& d, float2* sm)
{
    __syncthreads();  // the previous row of a persistent block is done with sm
    float2* a = sm;
    float2* b = sm + d.M;
    const int M = d.M, tid = threadIdx.x, nth = blockDim.x;
    if (in_len >= 2 * M && ((reinterpret_cast<uintptr_t>(x) & 7) == 0)) {
        const float2* x2 = reinterpret_cast<const float2*>(x);
        for (int m = tid; m < M; m += nth) a[m] = x2[m];
    }
    else {
        for (int m = tid; m < M; m += nth) {
            const int k = 2 * m;
            a[m] = make_float2(k < in_len ? x[k] : 0.f, k + 1 < in_len ? x[k + 1] : 0.f);
        }
    }
    __syncthreads();
    float2* Z = fft_c2c<-1>(a, b, d, tid, nth);
    for (int k = tid; k < M; k += nth) o[k] = r2c_bin(Z, k, M, d.twh);
}

__global__ void k_rfft_rows(const float* in, long in_ld, int in_len, float2* out, long out_ld, int nrows, FftDesc d)
{
    extern __shared__ float2 sm[];
    const int row = blockIdx.x;
    if (row >= nrows) return;
    rfft_row(in + (size_t)row * in_ld, in_len, out + (size_t)row * out_ld, d, sm);
}

// Two complex rows of M bins in dynamic shared memory; raise the opt-in limit
// when they exceed the default 48 KB.
static void allow_smem(const void* f, size_t bytes)
{
    if (bytes > 48 * 1024) cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// ---------------------------------------------------------------------------
// Many rows: a persistent block per SM slot loops over rows, with
//  * the first stage (radix 8, no twiddles) run from registers: each thread
//    loads the eight inputs of its butterfly straight from global memory,
//    and loads them for its next row while the later stages of the current
//    row run in shared memory (the row loads never stall the transform);
//  * the twiddle factors of every later stage and the real-packing twiddles
//    copied into shared memory once per block (stage s holds w^(r k) for
//    r = 1..R-1, k < Ns at [(r-1) Ns + k]: M - 1 values over all stages).
// Needs M % 16 == 0 (radix 8 first; swizzled stage buffers), aligned float2
// rows, and M / 8 <= 2 * threads.
// ---------------------------------------------------------------------------
namespace fftk {
// SIGN -1 forward, +1 inverse; tws holds the stage's twiddles of that sign
template <int R, int SIGN, bool SWI, bool SWO>
__device__ __forceinline__ void stage_smtw(const float2* __restrict__ src, float2* __restrict__ dst, int M, int Ns,
                                           const float2* __restrict__ tws, int tid, int nth)
{
    const int nR = M / R;
    const FastMod mod(Ns);
    for (int j = tid; j < nR; j += nth) {
        const int k = mod(j);
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = j + r * nR;
            v[r] = src[SWI ? swz(i) : i];
        }
        if (k) {
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = cmul(v[r], tws[(r - 1) * Ns + k]);
        }
        bfly<R, SIGN>(v);
        const int base = (j - k) * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = base + r * Ns;
            dst[SWO ? swz(i) : i] = v[r];
        }
    }
}

template <int R, int SIGN = -1>
__device__ __forceinline__ void stage_smtw_any(const float2* __restrict__ src, float2* __restrict__ dst, int M,
                                               int Ns, const float2* __restrict__ tws, int tid, int nth, bool swi,
                                               bool swo)
{
    if (swi) {
        if (swo) stage_smtw<R, SIGN, true, true>(src, dst, M, Ns, tws, tid, nth);
        else stage_smtw<R, SIGN, true, false>(src, dst, M, Ns, tws, tid, nth);
    }
    else {
        if (swo) stage_smtw<R, SIGN, false, true>(src, dst, M, Ns, tws, tid, nth);
        else stage_smtw<R, SIGN, false, false>(src, dst, M, Ns, tws, tid, nth);
    }
}

// Stages 1 .. nst-1 of a transform whose first stage (radix 8) wrote src,
// swizzled when more stages follow; returns the buffer with the result in
// natural order.  All threads of the block call it.
template <int SIGN>
__device__ __forceinline__ float2* stages_after_first(float2* src, float2* dst, const FftDesc& d,
                                                      const float2* __restrict__ tws, int tid, int nth)
{
    const int M = d.M;
    int Ns = 8, off = 0;
    bool swi = d.nst > 1;  // the first stage's writes have stride 8
    for (int s = 1; s < d.nst; ++s) {
        const int R = d.radix[s];
        const bool swo = s + 1 < d.nst && Ns < 16;  // strided writes only while Ns < 16
        switch (R) {
            case 2: stage_smtw_any<2, SIGN>(src, dst, M, Ns, tws + off, tid, nth, swi, swo); break;
            case 3: stage_smtw_any<3, SIGN>(src, dst, M, Ns, tws + off, tid, nth, swi, swo); break;
            case 4: stage_smtw_any<4, SIGN>(src, dst, M, Ns, tws + off, tid, nth, swi, swo); break;
            case 5: stage_smtw_any<5, SIGN>(src, dst, M, Ns, tws + off, tid, nth, swi, swo); break;
            case 7: stage_smtw_any<7, SIGN>(src, dst, M, Ns, tws + off, tid, nth, swi, swo); break;
            default: stage_smtw_any<8, SIGN>(src, dst, M, Ns, tws + off, tid, nth, swi, swo); break;
        }
        __syncthreads();
        off += (R - 1) * Ns;
        Ns *= R;
        swi = swo;
        float2* t = src;
        src = dst;
        dst = t;
    }
    return src;
}

// The twiddles of stages 1 .. nst-1 (conjugated for SIGN +1) and the
// real-packing twiddles into shared memory, once per block.
template <int SIGN>
__device__ __forceinline__ void load_stage_twiddles(const FftDesc& d, float2* tws, float2* twh, int tid, int nth)
{
    const int M = d.M;
    int Ns = d.radix[0], off = 0;
    for (int s = 1; s < d.nst; ++s) {
        const int R = d.radix[s], step = M / (Ns * R), n = (R - 1) * Ns;
        for (int e = tid; e < n; e += nth) {
            const int r = e / Ns + 1, k = e - (r - 1) * Ns;
            float2 w = __ldg(d.tw + k * r * step);
            if (SIGN > 0) w.y = -w.y;
            tws[off + e] = w;
        }
        off += n;
        Ns *= R;
    }
    for (int k = tid; k < M; k += nth) twh[k] = __ldg(d.twh + k);
}
}  // namespace fftk

// IT: first-stage butterflies per thread (M / 8 <= IT * 256)
template <int IT>
__global__ void __launch_bounds__(256) k_rfft_rows_pf(const float* __restrict__ in, long in_ld, int in_len,
                                                      float2* __restrict__ out, long out_ld, int nrows, FftDesc d)
{
    extern __shared__ float2 sm[];
    const int M = d.M, tid = threadIdx.x, nth = blockDim.x;
    float2* a = sm;
    float2* b = sm + M;
    float2* tws = sm + 2 * M;
    float2* twh = sm + 3 * M;
    fftk::load_stage_twiddles<-1>(d, tws, twh, tid, nth);
    const int nR = M / 8;
    float2 v[IT][8];
    auto fetch = [&](int row) {
        const float* x = in + (size_t)row * in_ld;
        const float2* x2 = reinterpret_cast<const float2*>(x);
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int j = tid + it * nth;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int m = j + q * nR, k = 2 * m;
                float2 val = make_float2(0.f, 0.f);
                if (j < nR) {
                    if (k + 1 < in_len) val = __ldcs(x2 + m);  // streamed once: evict first
                    else if (k < in_len) val.x = x[k];
                }
                v[it][q] = val;
            }
        }
    };
    int row = blockIdx.x;
    if (row < nrows) fetch(row);
    __syncthreads();  // twiddle tables
    const bool more = d.nst > 1;
    while (row < nrows) {
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int j = tid + it * nth;
            if (j < nR) {
                fftk::bfly8<-1>(v[it]);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int i = j * 8 + q;
                    a[more ? fftk::swz(i) : i] = v[it][q];
                }
            }
        }
        __syncthreads();
        const int next = row + gridDim.x;
        if (next < nrows) fetch(next);
        float2* src = fftk::stages_after_first<-1>(a, b, d, tws, tid, nth);
        float2* o = out + (size_t)row * out_ld;
        for (int k = tid; k < M; k += nth) {
            const float2 zk = src[k];
            float2 res;
            if (k == 0) res = make_float2(zk.x + zk.y, zk.x - zk.y);
            else {
                const float2 zm = cconj(src[M - k]);
                const float2 E = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y + zm.y));
                const float2 D = make_float2(0.5f * (zk.x - zm.x), 0.5f * (zk.y - zm.y));
                res = cadd(E, cmul(twh[k], make_float2(D.y, -D.x)));
            }
            o[k] = res;
        }
        __syncthreads();  // src is the next row's stage-1 output buffer or its stage scratch
        row = next;
    }
}

template <int IT>
static int rfft_pf_blocks(size_t smem)
{
    int dev = 0, nsm = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_rfft_rows_pf<IT>, 256, smem) != cudaSuccess) return 0;
    return per * nsm;
}

template <int IT>
static bool launch_rfft_pf(const float* in, long in_ld, int in_len, float2* out, long out_ld, int nrows,
                           const FftDesc& d, cudaStream_t s)
{
    const size_t smem = 4 * (size_t)d.M * sizeof(float2);
    allow_smem((const void*)k_rfft_rows_pf<IT>, smem);
    const int grid = std::min(nrows, rfft_pf_blocks<IT>(smem));
    if (grid <= 0 || nrows < 2 * grid) return false;  // under two rows per block: the per-row kernel
    k_rfft_rows_pf<IT><<<grid, 256, smem, s>>>(in, in_ld, in_len, out, out_ld, nrows, d);
    return true;
}

void launch_rfft_rows(const float* in, long in_ld, int in_len, float2* out, long out_ld, int nrows, const FftDesc& d,
                      cudaStream_t s, const TileMap& tiles)
{
    if (nrows <= 0) return;
    if (launch_rfft3(in, in_ld, in_len, out, out_ld, nrows, d, tiles, s)) return;
    const bool aligned = ((reinterpret_cast<uintptr_t>(in) & 7) == 0) && (in_ld % 2 == 0);
    if (aligned && d.M % 16 == 0 && d.nst >= 2 && d.radix[0] == 8 && 4 * (size_t)d.M * sizeof(float2) <= 128 * 1024) {
        if (d.M / 8 <= 256 && launch_rfft_pf<1>(in, in_ld, in_len, out, out_ld, nrows, d, s)) return;
        if (d.M / 8 > 256 && d.M / 8 <= 512 && launch_rfft_pf<2>(in, in_ld, in_len, out, out_ld, nrows, d, s)) return;
    }
    allow_smem((const void*)k_rfft_rows, 2 * d.M * sizeof(float2));
    const int nth = d.M >= 2048 ? 512 : 256;
    k_rfft_rows<<<nrows, nth, 2 * d.M * sizeof(float2), s>>>(in, in_ld, in_len, out, out_ld, nrows, d);
}

// ---------------------------------------------------------------------------
// Inverse real FFT of rows + frame write (ImpactTransform.cxx:303-347).
// Row r of Vh is wire wire0 + r; ticks are tick0 + column.
// ---------------------------------------------------------------------------
// One row: v (M packed bins) -> real values written to f[tick0 + c] for
// c < ncols, 0 <= tick0 + c < nticks.  Called by all threads of the block.
__device__ __forceinline__ void irfft_row(const float2* __restrict__ v, const FftDesc& d, float* __restrict__ f,
                                          int tick0, int ncols, int nticks, float2* sm)
{
    __syncthreads();  // the previous row of a persistent block is done with sm
    float2* a = sm;
    float2* b = sm + d.M;
    const int M = d.M, tid = threadIdx.x, nth = blockDim.x;
    for (int k = tid; k < M; k += nth) b[k] = v[k];
    __syncthreads();
    for (int k = tid; k < M; k += nth) a[k] = c2r_bin(b, k, M, d.twh);
    __syncthreads();
    float2* z = fft_c2c<+1>(a, b, d, tid, nth);
    const float sc = 1.0f / (float)M;
    for (int m = tid; m < M; m += nth) {
        const float2 zz = z[m];
        const int c0 = 2 * m;
        const int t0 = tick0 + c0;
        if (c0 < ncols && t0 >= 0 && t0 < nticks) f[t0] = zz.x * sc;
        if (c0 + 1 < ncols && t0 + 1 >= 0 && t0 + 1 < nticks) f[t0 + 1] = zz.y * sc;
    }
}

__global__ void k_irfft_rows(const float2* __restrict__ Vh, int nrows, FftDesc d, int wire0, int wlo, int whi,
                             int tick0, int ncols, int nticks, float* __restrict__ frame,
                             const unsigned char* __restrict__ row_flag, int nwires, int npad)
{
    extern __shared__ float2 sm[];
    const int row = blockIdx.x;
    const int W = wire0 + row;
    if (row >= nrows || W < wlo || W >= whi) return;
    if (row_flag && !row_reached(row_flag, nwires, W, npad)) return;
    irfft_row(Vh + (size_t)row * d.M, d, frame + (size_t)W * nticks, tick0, ncols, nticks, sm);
}

// Many rows: persistent blocks (as k_rfft_rows_pf) over the rows that are
// frame wires, each thread holding its share of the next row's packed
// spectrum in registers while the current row is transformed; the complex
// pre-processing of the real inverse is fused into the first (radix-8)
// stage; twiddles in shared memory.  IT: spectrum values per thread
// (M <= 256 IT).
template <int IT>
__global__ void __launch_bounds__(256) k_irfft_rows_pf(const float2* __restrict__ Vh, int r0, int r1, FftDesc d,
                                                       int wire0, int tick0, int ncols, int nticks,
                                                       float* __restrict__ frame,
                                                       const unsigned char* __restrict__ row_flag, int nwires,
                                                       int npad)
{
    extern __shared__ float2 sm[];
    const int M = d.M, tid = threadIdx.x, nth = blockDim.x;
    float2* a = sm;
    float2* b = sm + M;
    float2* tws = sm + 2 * M;
    float2* twh = sm + 3 * M;
    fftk::load_stage_twiddles<+1>(d, tws, twh, tid, nth);
    float2 pv[IT];
    auto fetch = [&](int row) {
        const float2* v = Vh + (size_t)row * M;
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int k = tid + it * nth;
            pv[it] = k < M ? __ldcs(v + k) : make_float2(0.f, 0.f);
        }
    };
    int row = r0 + blockIdx.x;
    if (row < r1) fetch(row);
    __syncthreads();  // twiddle tables
    const bool more = d.nst > 1;
    const int nR = M / 8;
    const float sc = 1.0f / (float)M;
    while (row < r1) {
        const int next = row + gridDim.x;
        if (row_flag && !row_reached(row_flag, nwires, wire0 + row, npad)) {  // uniform over the block
            if (next < r1) fetch(next);
            row = next;
            continue;
        }
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int k = tid + it * nth;
            if (k < M) b[k] = pv[it];
        }
        __syncthreads();
        if (next < r1) fetch(next);
        // first stage (radix 8, no twiddles) on the pre-processed bins
        for (int j = tid; j < nR; j += nth) {
            float2 v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int k = j + q * nR;
                const float2 xk = b[k];
                if (k == 0) {
                    v[q] = make_float2(0.5f * (xk.x + xk.y), 0.5f * (xk.x - xk.y));
                }
                else {
                    const float2 xm = cconj(b[M - k]);
                    const float2 E = make_float2(0.5f * (xk.x + xm.x), 0.5f * (xk.y + xm.y));
                    const float2 D = make_float2(0.5f * (xk.x - xm.x), 0.5f * (xk.y - xm.y));
                    const float2 O = cmulc(D, twh[k]);
                    v[q] = make_float2(E.x - O.y, E.y + O.x);
                }
            }
            fftk::bfly8<+1>(v);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int i = j * 8 + q;
                a[more ? fftk::swz(i) : i] = v[q];
            }
        }
        __syncthreads();  // b is read by the first stage and written by the second
        const float2* z = fftk::stages_after_first<+1>(a, b, d, tws, tid, nth);
        float* f = frame + (size_t)(wire0 + row) * nticks;
        for (int m = tid; m < M; m += nth) {
            const float2 zz = z[m];
            const int c0 = 2 * m;
            const int t0 = tick0 + c0;
            if (c0 < ncols && t0 >= 0 && t0 < nticks) f[t0] = zz.x * sc;
            if (c0 + 1 < ncols && t0 + 1 >= 0 && t0 + 1 < nticks) f[t0 + 1] = zz.y * sc;
        }
        __syncthreads();  // z is the next row's spectrum or first-stage buffer
        row = next;
    }
}

template <int IT>
static bool launch_irfft_pf(const float2* Vh, int r0, int r1, const FftDesc& d, int wire0, int tick0, int ncols,
                            int nticks, float* frame, const unsigned char* row_flag, int nwires, int npad,
                            cudaStream_t s)
{
    const size_t smem = 4 * (size_t)d.M * sizeof(float2);
    allow_smem((const void*)k_irfft_rows_pf<IT>, smem);
    int dev = 0, nsm = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return false;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_irfft_rows_pf<IT>, 256, smem) != cudaSuccess) return false;
    const int grid = std::min(r1 - r0, per * nsm);
    if (grid <= 0 || r1 - r0 < 2 * grid) return false;  // under two rows per block: one block per row
    k_irfft_rows_pf<IT><<<grid, 256, smem, s>>>(Vh, r0, r1, d, wire0, tick0, ncols, nticks, frame, row_flag, nwires,
                                                npad);
    return true;
}

void launch_irfft_rows(const float2* Vh, int nrows, const FftDesc& d, int wire0, int wlo, int whi, int tick0,
                       int ncols, int nticks, float* frame, cudaStream_t s, const unsigned char* row_flag, int nwires,
                       int npad)
{
    // the rows that are frame wires: wire0 + r in [wlo, whi)
    const int r0 = std::max(0, wlo - wire0), r1 = std::min(nrows, whi - wire0);
    if (nrows <= 0 || r1 <= r0) return;
    if (launch_irfft3(Vh, r0, r1, d, wire0, tick0, ncols, nticks, frame, row_flag, nwires, npad, s)) return;
    if (d.M % 16 == 0 && d.nst >= 2 && d.radix[0] == 8 && 4 * (size_t)d.M * sizeof(float2) <= 128 * 1024) {
        if (d.M <= 1024 && launch_irfft_pf<4>(Vh, r0, r1, d, wire0, tick0, ncols, nticks, frame, row_flag, nwires,
                                               npad, s))
            return;
        if (d.M > 1024 && d.M <= 2048 && launch_irfft_pf<8>(Vh, r0, r1, d, wire0, tick0, ncols, nticks, frame,
                                                                row_flag, nwires, npad, s))
            return;
    }
    allow_smem((const void*)k_irfft_rows, 2 * d.M * sizeof(float2));
    const int nth = d.M >= 2048 ? 512 : 256;
    k_irfft_rows<<<nrows, nth, 2 * d.M * sizeof(float2), s>>>(Vh, nrows, d, wire0, wlo, whi, tick0, ncols, nticks,
                                                                  frame, row_flag, nwires, npad);
}

// ---------------------------------------------------------------------------
// Wire-direction convolution in the (wire, frequency) domain:
//   V[o][f] = sum_g sum_{j=-P}^{P} R_g[j][f] * Q_g[o - P - j][f]
// Input row i is wire row0 + i; output row o is wire row0 - P + o.
// Block: 32 frequencies x 8 row groups, each thread 8 consecutive output
// rows with a register sliding window over the staged input rows.
// Bin 0 (packed DC/Nyquist) is multiplied component-wise.
// ---------------------------------------------------------------------------
constexpr int kConvRB = 8;
constexpr int kConvRG = 8;
constexpr int kConvRows = kConvRB * kConvRG;

// A group's taps are summed apart and then added to the groups before: one sum
// over all of 473 taps (258 mirrored) rounds at its full size from the first
// centre tap on, 3.4e-7 of a frame in all against 1.5 to 2.2e-7 so (full APA and
// planes, tracks and showers; the row transforms' share 1.5e-7).
template <int N>
__device__ __forceinline__ void add_sums(float2* sum, const float2* acc)
{
#pragma unroll
    for (int r = 0; r < N; ++r) sum[r] = make_float2(sum[r].x + acc[r].x, sum[r].y + acc[r].y);
}

// One tile of the wire convolution: frequencies fblk*32 .. +31, output rows
// oblk*64 .. +63.  Called by all threads of a (32, kConvRG) block.
// PAIR: groups g and G-1-g share one response up to a mirror in wire
// (R_{G-1-g}[j] = R_g[-j], the symmetrised impact map of
// gen/src/PlaneImpactResponse.cxx:256-268), so for each tap the two
// mirrored inputs are added before one complex multiply.
template <int PAD, bool PAIR>
__device__ __forceinline__ void wire_conv_tile(const float2* __restrict__ Qh, const float2* __restrict__ Rh,
                                               float2* __restrict__ Vh, int G, int nin, int nout, int M, int fblk,
                                               int oblk, float2* conv_smem)
{
    constexpr int SROWS = kConvRows + 2 * PAD;
    constexpr int NT = 2 * PAD + 1;
    float2 (*Qs)[32] = reinterpret_cast<float2 (*)[32]>(conv_smem);
    float2 (*Qs2)[32] = reinterpret_cast<float2 (*)[32]>(conv_smem + SROWS * 32);
    float2 (*Rs)[32] = reinterpret_cast<float2 (*)[32]>(conv_smem + (PAIR ? 2 : 1) * SROWS * 32);
    const int lane = threadIdx.x, rg = threadIdx.y;
    const int f = fblk * 32 + lane;
    const int o0 = oblk * kConvRows;
    const bool fok = f < M;
    const bool dc = f == 0;
    float2 sum[kConvRB];
#pragma unroll
    for (int r = 0; r < kConvRB; ++r) sum[r] = make_float2(0.f, 0.f);
    const int rb0 = rg * kConvRB;
    const int ng = PAIR ? (G + 1) / 2 : G;
    for (int gi = 0; gi < ng; ++gi) {
        const int g = gi;
        const int g2 = G - 1 - gi;
        const bool pair = PAIR && g2 != g;
        __syncthreads();
        for (int s = rg; s < SROWS; s += kConvRG) {
            const int i = o0 - 2 * PAD + s;
            const bool ok = fok && i >= 0 && i < nin;
            Qs[s][lane] = ok ? Qh[((size_t)g * nin + i) * M + f] : make_float2(0.f, 0.f);
            if (PAIR) Qs2[s][lane] = (ok && pair) ? Qh[((size_t)g2 * nin + i) * M + f] : make_float2(0.f, 0.f);
        }
        for (int jj = rg; jj < NT; jj += kConvRG)
            Rs[jj][lane] = fok ? Rh[((size_t)g * NT + jj) * M + f] : make_float2(0.f, 0.f);
        __syncthreads();
        if (fok) {
            float2 acc[kConvRB], win[kConvRB], win2[kConvRB];  // acc: the group's sums (add_sums)
#pragma unroll
            for (int r = 0; r < kConvRB; ++r) {
                acc[r] = make_float2(0.f, 0.f);
                win[r] = Qs[rb0 + r + 2 * PAD][lane];       // input row o - PAD - j at j = -PAD
                if (PAIR) win2[r] = Qs2[rb0 + r][lane];     // input row o - PAD + j at j = -PAD
            }
#pragma unroll
            for (int jj = 0; jj < NT; ++jj) {
                const float2 rr = Rs[jj][lane];
                // bin 0 packs two real spectra (DC, Nyquist): multiply component-wise there
                const float rc = dc ? 0.f : rr.y;
                const float ry = dc ? rr.y : rr.x;
#pragma unroll
                for (int r = 0; r < kConvRB; ++r) {
                    float2 q = win[r];
                    if (PAIR) q = make_float2(q.x + win2[r].x, q.y + win2[r].y);
                    acc[r].x = fmaf(rr.x, q.x, fmaf(-rc, q.y, acc[r].x));
                    acc[r].y = fmaf(ry, q.y, fmaf(rc, q.x, acc[r].y));
                }
                if (jj < NT - 1) {
#pragma unroll
                    for (int r = kConvRB - 1; r > 0; --r) win[r] = win[r - 1];
                    win[0] = Qs[rb0 + 2 * PAD - jj - 1][lane];
                    if (PAIR) {
#pragma unroll
                        for (int r = 0; r < kConvRB - 1; ++r) win2[r] = win2[r + 1];
                        win2[kConvRB - 1] = Qs2[rb0 + kConvRB + jj][lane];
                    }
                }
            }
            add_sums<kConvRB>(sum, acc);
        }
    }
    if (fok) {
#pragma unroll
        for (int r = 0; r < kConvRB; ++r) {
            const int o = o0 + rb0 + r;
            if (o < nout) Vh[(size_t)o * M + f] = sum[r];
        }
    }
}

template <int PAD, bool PAIR>
__global__ void __launch_bounds__(32 * kConvRG) k_wire_conv(const float2* __restrict__ Qh,
                                                             const float2* __restrict__ Rh, float2* __restrict__ Vh,
                                                             int G, int nin, int nout, int M)
{
    extern __shared__ float2 conv_smem[];
    wire_conv_tile<PAD, PAIR>(Qh, Rh, Vh, G, nin, nout, M, blockIdx.x, blockIdx.y, conv_smem);
}

// One frequency (per lane) of the eight output rows o0 .. with a run-time pad; mask
// are written.
__device__ __forceinline__ void conv_rows_any(const float2* __restrict__ Qh, const float2* __restrict__ Rh,
                                              float2* __restrict__ Vh, int G, int PAD, int nin, int M, int f, int o0,
                                              unsigned mask)
{
    float2 acc[kConvRB];
#pragma unroll
    for (int r = 0; r < kConvRB; ++r) acc[r] = make_float2(0.f, 0.f);
    for (int g = 0; g < G; ++g) {
        const float2* Rg = Rh + (size_t)g * (2 * PAD + 1) * M + f;
        for (int jj = 0; jj <= 2 * PAD; ++jj) {
            const float2 rr = Rg[(size_t)jj * M];
            const float rc = f == 0 ? 0.f : rr.y;
            const float ry = f == 0 ? rr.y : rr.x;
            const int j = jj - PAD;
#pragma unroll
            for (int r = 0; r < kConvRB; ++r) {
                const int i = o0 + r - PAD - j;
                if (i < 0 || i >= nin) continue;
                const float2 q = Qh[((size_t)g * nin + i) * M + f];
                acc[r].x = fmaf(rr.x, q.x, fmaf(-rc, q.y, acc[r].x));
                acc[r].y = fmaf(ry, q.y, fmaf(rc, q.x, acc[r].y));
            }
        }
    }
#pragma unroll
    for (int r = 0; r < kConvRB; ++r)
        if (mask >> r & 1) Vh[(size_t)(o0 + r) * M + f] = acc[r];
}

// Same convolution with a run-time pad (any response width).
__global__ void __launch_bounds__(32 * kConvRG) k_wire_conv_any(const float2* __restrict__ Qh,
                                                                 const float2* __restrict__ Rh,
                                                                 float2* __restrict__ Vh, int G, int PAD, int nin,
                                                                 int nout, int M)
{
    const int f = blockIdx.x * 32 + threadIdx.x, o0 = blockIdx.y * kConvRows + threadIdx.y * kConvRB;
    if (f >= M) return;
    conv_rows_any(Qh, Rh, Vh, G, PAD, nin, M, f, o0, o0 + kConvRB <= nout ? 0xffu : (1u << max(nout - o0, 0)) - 1u);
}

// ---------------------------------------------------------------------------
// The same convolution with the staging of the next group (pair) overlapped
// with the arithmetic of the current one: 16 frequencies x 16 row groups per
// block (128 output rows), the input rows, mirrored rows and taps of group
// gi + 1 copied by cp.async into the second of two shared-memory buffers
// while group gi is multiplied out of the first.  Needs 16-byte aligned
// spectra and an even M (two frequencies per 16-byte copy).
// ---------------------------------------------------------------------------
constexpr int kConv2F = 16;  // frequencies per block
constexpr int kConv2RG = 16; // row groups per block (kConvRB output rows each)
constexpr int kConv2Rows = kConv2RG * kConvRB;
constexpr int kRowsBlocks = 148 * 2;  // resident blocks that take a list's rows


template <bool PAIR, int RG>
constexpr size_t conv2_stage_f2(int pad)  // float2 values per pipeline stage
{
    return (size_t)kConv2F * ((PAIR ? 2 : 1) * (RG * kConvRB + 2 * pad) + (2 * pad + 1));
}

// Output rows at 16 frequencies: a thread's RB rows from o0 + rb0 on (rb0 < 0:
// none), of which mask are written; the block's rows lie within span (at most
// 8 RG) of o0.  PAD 0: run-time pad, the taps rolled by four.  Called by all 16 RG
// threads of the block.
template <int PAD, bool PAIR, int RB, int RG>
__device__ __forceinline__ void conv2_unit(const float2* __restrict__ Qh, const float2* __restrict__ Rh,
                                           float2* __restrict__ Vh, int G, int pad, int nin, int M, int f0, int o0,
                                           int span, int rb0, unsigned mask, float2* conv2_smem)
{
    const int P = PAD ? PAD : pad;
    const int SROWS = RG * kConvRB + 2 * P, NT = 2 * P + 1;
    const size_t STAGE = conv2_stage_f2<PAIR, RG>(P);
    const int tid = threadIdx.x, lane = tid & (kConv2F - 1);
    const int f = f0 + lane;
    const bool dc = f == 0;
    const int ng = PAIR ? (G + 1) / 2 : G;
    // copy of group gi into stage buffer st: 8 16-byte pieces per row of 16 frequencies
    auto issue = [&](int gi, int st) {
        float2* base = conv2_smem + (size_t)st * STAGE;
        float2* Qs = base;
        float2* Qs2 = base + SROWS * kConv2F;
        float2* Rs = base + (PAIR ? 2 : 1) * SROWS * kConv2F;
        const int g = gi, g2 = G - 1 - gi;
        const bool pair = PAIR && g2 != g;
        const int fp = f0 + 2 * (tid & 7);           // first frequency of this thread's piece
        const int fbytes = fp < M ? 16 : 0;          // M even: both or neither of fp, fp + 1
        constexpr int kPieces = kConv2F / 2;
        constexpr int nthr = kConv2F * RG;
        for (int e = tid; e < (span + 2 * P) * kPieces; e += nthr) {
            const int srow = e / kPieces;
            const int i = o0 - 2 * P + srow;
            const bool ok = i >= 0 && i < nin && fbytes;
            const float2* src = ok ? Qh + ((size_t)g * nin + i) * M + fp : Qh;
            cp_async16(Qs + srow * kConv2F + 2 * (e % kPieces), src, ok ? 16 : 0);
            if (PAIR) {
                const bool ok2 = ok && pair;
                const float2* src2 = ok2 ? Qh + ((size_t)g2 * nin + i) * M + fp : Qh;
                cp_async16(Qs2 + srow * kConv2F + 2 * (e % kPieces), src2, ok2 ? 16 : 0);
            }
        }
        for (int e = tid; e < NT * kPieces; e += nthr) {
            const int jj = e / kPieces;
            const float2* src = fbytes ? Rh + ((size_t)g * NT + jj) * M + fp : Rh;
            cp_async16(Rs + jj * kConv2F + 2 * (e % kPieces), src, fbytes);
        }
        cp_async_commit();
    };
    float2 sum[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) sum[r] = make_float2(0.f, 0.f);
    issue(0, 0);
    for (int gi = 0; gi < ng; ++gi) {
        if (gi + 1 < ng) {
            issue(gi + 1, (gi + 1) & 1);
            cp_async_wait<1>();
        }
        else
            cp_async_wait<0>();
        __syncthreads();
        if (rb0 >= 0) {
            float2 acc[RB];  // the group's sums (add_sums)
#pragma unroll
            for (int r = 0; r < RB; ++r) acc[r] = make_float2(0.f, 0.f);
            const float2* base = conv2_smem + (size_t)(gi & 1) * STAGE;
            const float2* Qs = base;
            const float2* Qs2 = base + SROWS * kConv2F;
            const float2* Rs = base + (PAIR ? 2 : 1) * SROWS * kConv2F;
            if constexpr (PAD > 0) {
                float2 win[RB], win2[RB];
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    win[r] = Qs[(rb0 + r + 2 * PAD) * kConv2F + lane];  // input row o - PAD - j at j = -PAD
                    if (PAIR) win2[r] = Qs2[(rb0 + r) * kConv2F + lane];  // input row o - PAD + j at j = -PAD
                }
#pragma unroll
                for (int jj = 0; jj <= 2 * PAD; ++jj) {
                    const float2 rr = Rs[jj * kConv2F + lane];
                    // bin 0 packs two real spectra (DC, Nyquist): multiply component-wise there
                    const float rc = dc ? 0.f : rr.y;
                    const float ry = dc ? rr.y : rr.x;
#pragma unroll
                    for (int r = 0; r < RB; ++r) {
                        float2 q = win[r];
                        if (PAIR) q = make_float2(q.x + win2[r].x, q.y + win2[r].y);
                        acc[r].x = fmaf(rr.x, q.x, fmaf(-rc, q.y, acc[r].x));
                        acc[r].y = fmaf(ry, q.y, fmaf(rc, q.x, acc[r].y));
                    }
                    if (jj < 2 * PAD) {
#pragma unroll
                        for (int r = RB - 1; r > 0; --r) win[r] = win[r - 1];
                        win[0] = Qs[(rb0 + 2 * PAD - jj - 1) * kConv2F + lane];
                        if (PAIR) {
#pragma unroll
                            for (int r = 0; r < RB - 1; ++r) win2[r] = win2[r + 1];
                            win2[RB - 1] = Qs2[(rb0 + RB + jj) * kConv2F + lane];
                        }
                    }
                }
            }
            else {
                float2 w[RB + 4], v[RB + 4];  // rows o - jj and o - 2P + jj of the next four taps
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    w[4 + r] = Qs[(rb0 + r + 2 * P) * kConv2F + lane];
                    if (PAIR) v[r] = Qs2[(rb0 + r) * kConv2F + lane];
                }
                for (int j0 = 0; j0 < NT; j0 += 4) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        w[3 - k] = Qs[max(rb0 + 2 * P - j0 - 1 - k, 0) * kConv2F + lane];
                        if (PAIR) v[RB + k] = Qs2[min(rb0 + RB + j0 + k, SROWS - 1) * kConv2F + lane];
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        if (j0 + k < NT) {
                            const float2 rr = Rs[(j0 + k) * kConv2F + lane];
                            const float rc = dc ? 0.f : rr.y;
                            const float ry = dc ? rr.y : rr.x;
#pragma unroll
                            for (int r = 0; r < RB; ++r) {
                                float2 q = w[4 + r - k];
                                if (PAIR) q = make_float2(q.x + v[r + k].x, q.y + v[r + k].y);
                                acc[r].x = fmaf(rr.x, q.x, fmaf(-rc, q.y, acc[r].x));
                                acc[r].y = fmaf(ry, q.y, fmaf(rc, q.x, acc[r].y));
                            }
                        }
                    }
#pragma unroll
                    for (int r = 0; r < RB; ++r) {
                        w[3 + RB - r] = w[RB - 1 - r];
                        if (PAIR) v[r] = v[r + 4];
                    }
                }
            }
            add_sums<RB>(sum, acc);
        }
        __syncthreads();  // buffer gi & 1 is refilled with group gi + 2 next
    }
    if (f < M && rb0 >= 0) {
#pragma unroll
        for (int r = 0; r < RB; ++r)
            if (mask >> r & 1) Vh[(size_t)(o0 + rb0 + r) * M + f] = sum[r];
    }
}

template <int PAD, bool PAIR>
__global__ void __launch_bounds__(kConv2F * kConv2RG) k_wire_conv2(const float2* __restrict__ Qh,
                                                                  const float2* __restrict__ Rh,
                                                                  float2* __restrict__ Vh, int G, int nin, int nout,
                                                                  int M)
{
    extern __shared__ __align__(16) float2 conv2_smem[];
    const int o0 = blockIdx.y * kConv2Rows, rb0 = threadIdx.x / kConv2F * kConvRB, left = nout - (o0 + rb0);
    conv2_unit<PAD, PAIR, kConvRB, kConv2RG>(Qh, Rh, Vh, G, PAD, nin, M, blockIdx.x * kConv2F, o0, kConv2Rows, rb0,
                          left >= kConvRB ? 0xffu : (1u << max(left, 0)) - 1u, conv2_smem);
}

// A list's chunk at 16 frequencies: a group of rows per 16 threads, where that
// leaves half of the block without one two or four 16 a group (a chunk is a chain
// of copies and sums: few rows take as long as many).
template <int PAD, bool PAIR, int WAYS>
__device__ __forceinline__ void conv2_ways(const float2* __restrict__ Qh, const float2* __restrict__ Rh,
                                           float2* __restrict__ Vh, int G, int pad, int nin, int M, int f0,
                                           const RowList& list, const int4& c, float2* conv2_smem)
{
    constexpr int RB = kConvRB / WAYS;
    const int rg = threadIdx.x / kConv2F, mine = rg / WAYS, first = RB * (rg & (WAYS - 1));
    const int o0 = list.item[c.x].x;
    const int2 it = mine < c.y ? list.item[c.x + mine] : make_int2(0, 0);
    conv2_unit<PAD, PAIR, RB, kConvGroups>(Qh, Rh, Vh, G, pad, nin, M, f0, o0, c.w, mine < c.y ? it.x - o0 + first : -1,
                              (unsigned)it.y >> first & ((1u << RB) - 1u), conv2_smem);
}
template <int PAD, bool PAIR>
__device__ __forceinline__ void conv2_chunk(const float2* __restrict__ Qh, const float2* __restrict__ Rh,
                                            float2* __restrict__ Vh, int G, int pad, int nin, int M, int f0,
                                            const RowList& list, const int4& c, float2* conv2_smem)
{
    if (c.y <= kConvGroups / 4) conv2_ways<PAD, PAIR, 4>(Qh, Rh, Vh, G, pad, nin, M, f0, list, c, conv2_smem);
    else if (c.y <= kConvGroups / 2) conv2_ways<PAD, PAIR, 2>(Qh, Rh, Vh, G, pad, nin, M, f0, list, c, conv2_smem);
    else conv2_ways<PAD, PAIR, 1>(Qh, Rh, Vh, G, pad, nin, M, f0, list, c, conv2_smem);
}

template <int PAD, bool PAIR>
__global__ void __launch_bounds__(kConv2F * kConvGroups) k_wire_rows2(const float2* __restrict__ Qh,
                                                                  const float2* __restrict__ Rh,
                                                                  float2* __restrict__ Vh, int G, int pad, int nin,
                                                                  int M, RowList list)
{
    extern __shared__ __align__(16) float2 conv2_smem[];
    const int nf = (M + kConv2F - 1) / kConv2F, total = list.count[1] * nf;
    for (int u = blockIdx.x; u < total; u += gridDim.x)
        conv2_chunk<PAD, PAIR>(Qh, Rh, Vh, G, pad, nin, M, u % nf * kConv2F, list, list.chunk[u / nf], conv2_smem);
}

void launch_wire_conv(const float2* Qh, const float2* Rh, float2* Vh, int ngroups, int npad, int nrows_in,
                      int nrows_out, int M, bool pair, cudaStream_t s)
{
    if (nrows_out <= 0) return;
    const bool al16 = ((reinterpret_cast<uintptr_t>(Qh) | reinterpret_cast<uintptr_t>(Rh)) & 15) == 0 && M % 2 == 0;
    if (al16 && (npad == 21 || npad == 10)) {
        dim3 grid2((M + kConv2F - 1) / kConv2F, (nrows_out + kConv2Rows - 1) / kConv2Rows);
        const int block2 = kConv2F * kConv2RG;
#define WCT_CONV2(P, B)                                                                                       \
    do {                                                                                                      \
        const size_t sm = 2 * conv2_stage_f2<B, kConv2RG>(P) * sizeof(float2);                                       \
        cudaFuncSetAttribute((const void*)k_wire_conv2<P, B>, cudaFuncAttributeMaxDynamicSharedMemorySize,   \
                             (int)sm);                                                                        \
        k_wire_conv2<P, B><<<grid2, block2, sm, s>>>(Qh, Rh, Vh, ngroups, nrows_in, nrows_out, M);            \
        return;                                                                                               \
    } while (0)
        if (npad == 10 && pair) WCT_CONV2(10, true);
        if (npad == 10) WCT_CONV2(10, false);
        if (npad == 21 && pair) WCT_CONV2(21, true);
        WCT_CONV2(21, false);
#undef WCT_CONV2
    }
    launch_wire_conv_tiles(Qh, Rh, Vh, ngroups, npad, nrows_in, nrows_out, M, pair, s);
}

void launch_wire_conv_tiles(const float2* Qh, const float2* Rh, float2* Vh, int ngroups, int npad, int nrows_in,
                            int nrows_out, int M, bool pair, cudaStream_t s)
{
    if (nrows_out <= 0) return;
    dim3 grid((M + 31) / 32, (nrows_out + kConvRows - 1) / kConvRows);
    dim3 block(32, kConvRG);
    auto smem = [](int pad, bool pr) {
        return sizeof(float2) * 32 * ((size_t)(pr ? 2 : 1) * (kConvRows + 2 * pad) + (2 * pad + 1));
    };
#define WCT_CONV(P, B)                                                                                        \
    do {                                                                                                      \
        const size_t sm = smem(P, B);                                                                         \
        cudaFuncSetAttribute((const void*)k_wire_conv<P, B>, cudaFuncAttributeMaxDynamicSharedMemorySize,    \
                             (int)sm);                                                                        \
        k_wire_conv<P, B><<<grid, block, sm, s>>>(Qh, Rh, Vh, ngroups, nrows_in, nrows_out, M);               \
    } while (0)
    if (npad == 10 && pair) WCT_CONV(10, true);
    else if (npad == 10) WCT_CONV(10, false);
    else if (npad == 21 && pair) WCT_CONV(21, true);
    else if (npad == 21) WCT_CONV(21, false);
#undef WCT_CONV
    else k_wire_conv_any<<<grid, block, 0, s>>>(Qh, Rh, Vh, ngroups, npad, nrows_in, nrows_out, M);
}

// ---------------------------------------------------------------------------
// Trace edges (Waveform::edge, util/src/Waveform.cxx:136-153) of frame rows
// [r0, r0 + nrows) over ticks [t0, t1): out[r] = (first non-zero tick, last
// non-zero tick + 1) relative to t0, or (0, 0) for a row without one.  One
// warp per row.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_row_edges(const float* __restrict__ frame, int ld, int r0, int nrows,
                                                   int t0, int t1, int2* __restrict__ out)
{
    const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= nrows) return;  // whole warps
    const float* row = frame + (size_t)(r0 + r) * ld;
    int lo = INT_MAX, hi = -1;
    for (int t = t0 + lane; t < t1; t += 32)
        if (row[t] != 0.0f) {  // -0.0 counts as zero, as the reference's test
            lo = min(lo, t);
            hi = t;
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) out[r] = hi < 0 ? make_int2(0, 0) : make_int2(lo - t0, hi + 1 - t0);
}

void launch_row_edges(const float* frame, int ld, int r0, int nrows, int t0, int t1, int2* out, cudaStream_t s)
{
    if (nrows <= 0) return;
    k_row_edges<<<(nrows + 7) / 8, 256, 0, s>>>(frame, ld, r0, nrows, t0, t1, out);
}

// ---------------------------------------------------------------------------
// PlaneImpactResponse::build_responses on the device
// (gen/src/PlaneImpactResponse.cxx:89-269), in the reference's single
// precision.  k_pir_bin: each path's field response on the tick grid
// (:185-218): sample r at Binning::center(r) = tstart + (r + 1/2) rawbs falls
// in tick bin (size_t)(time / tick) and adds current * period to that bin, a
// float (Waveform::realseq_t: every add rounded to float); rows of n complex
// values with zero imaginary parts.  One thread per path (the samples of a
// path in order, as the reference adds them).
// ---------------------------------------------------------------------------
__global__ void k_pir_bin(const double* __restrict__ current, int npaths, int nsamples, double tstart, double rawbs,
                          double period, double tick, int n, float2* __restrict__ Z)
{
    const int ip = blockIdx.x * blockDim.x + threadIdx.x;
    if (ip >= npaths) return;
    float2* z = Z + (size_t)ip * n;
    for (int k = 0; k < n; ++k) z[k] = make_float2(0.f, 0.f);
    const double* cur = current + (size_t)ip * nsamples;
    long long bin = -1;
    float acc = 0.f;
    for (int r = 0; r < nsamples; ++r) {
        const double time = __dadd_rn(tstart, __dmul_rn(__dadd_rn((double)r, 0.5), rawbs));
        const long long b = __double2ll_rz(__ddiv_rn(time, tick));
        if (b != bin) {  // a new bin: store the finished one, start from what the new one holds
            if (bin >= 0 && bin < n) z[bin].x = acc;
            bin = b;
            acc = (bin >= 0 && bin < n) ? z[bin].x : 0.f;
        }
        acc = (float)__dadd_rn((double)acc, __dmul_rn(cur[r], period));
    }
    if (bin >= 0 && bin < n) z[bin].x = acc;
}

// The product of nrows spectra of length n, bin by bin in row order, into
// out (the reference's short_spec[bin] *= spec[bin] over its short responses,
// starting from 1).
__global__ void k_spec_chain(const float2* __restrict__ S, int nrows, int n, float2* __restrict__ out)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    float2 a = S[k];
    for (int r = 1; r < nrows; ++r) a = cmul(a, S[(size_t)r * n + k]);
    out[k] = a;
}

// Real parts of the first min(n, ncols) values of each complex row of length
// n into float rows of ncols (zero beyond n): inv_c2r and its resize.
__global__ void k_real_rows(const float2* __restrict__ Z, int nrows, int n, float* __restrict__ out, int ncols)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x, r = blockIdx.y;
    if (c >= ncols || r >= nrows) return;
    out[(size_t)r * ncols + c] = c < n ? Z[(size_t)r * n + c].x : 0.f;
}

void launch_pir_bin(const double* current, int npaths, int nsamples, double tstart, double rawbs, double period,
                    double tick, int n, float2* Z, cudaStream_t s)
{
    if (npaths <= 0) return;
    k_pir_bin<<<(npaths + 63) / 64, 64, 0, s>>>(current, npaths, nsamples, tstart, rawbs, period, tick, n, Z);
}

void launch_spec_chain(const float2* S, int nrows, int n, float2* out, cudaStream_t s)
{
    if (nrows <= 0 || n <= 0) return;
    k_spec_chain<<<(n + 255) / 256, 256, 0, s>>>(S, nrows, n, out);
}

void launch_real_rows(const float2* Z, int nrows, int n, float* out, int ncols, cudaStream_t s)
{
    if (nrows <= 0 || ncols <= 0) return;
    k_real_rows<<<dim3((ncols + 255) / 256, nrows), 256, 0, s>>>(Z, nrows, n, out, ncols);
}

// ---------------------------------------------------------------------------
// Batched row convolution helpers (DftTools::convolve, aux/src/DftTools.cxx:145-168).
// ---------------------------------------------------------------------------
// X[row][k] *= R[k] on packed real spectra (bin 0 component-wise).
__global__ void k_spec_mul(float2* __restrict__ X, long ldx, int nrows, int M, const float2* __restrict__ R)
{
    const int row = blockIdx.y;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < M; k += gridDim.x * blockDim.x) {
        const float2 r = R[k];
        float2 x = X[(size_t)row * ldx + k];
        x = k == 0 ? make_float2(x.x * r.x, x.y * r.y) : cmul(x, r);
        X[(size_t)row * ldx + k] = x;
    }
}

void launch_spec_mul(float2* X, long ldx, int nrows, int M, const float2* R, cudaStream_t s)
{
    if (nrows <= 0) return;
    dim3 grid((M + 255) / 256, nrows);
    k_spec_mul<<<grid, 256, 0, s>>>(X, ldx, nrows, M, R);
}

// exp(-2 pi i m / M) and exp(-2 pi i m / (2M)) in double, stored as float.
__global__ void k_twiddles(float2* __restrict__ tw, float2* __restrict__ twh, int M)
{
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < M; m += gridDim.x * blockDim.x) {
        double sa, ca, sb, cb;
        sincospi(-2.0 * (double)m / (double)M, &sa, &ca);
        sincospi(-(double)m / (double)M, &sb, &cb);
        tw[m] = make_float2((float)ca, (float)sa);
        twh[m] = make_float2((float)cb, (float)sb);
    }
}

void launch_twiddles(float2* tw, float2* twh, int M, cudaStream_t s)
{
    k_twiddles<<<(M + 255) / 256, 256, 0, s>>>(tw, twh, M);
}

// ===========================================================================
// Batched events: a device-planned pipeline with no host round trip, so a
// whole batch is one captured CUDA graph.  After the prep/scan/fill kernels
// (the event-table forms of the single-event ones), k_plan_batch computes
// every (event, plane) window on the device -- ImpactTransform's window
// arithmetic (gen/src/ImpactTransform.cxx:83-115) with the reference's FFT
// length tables -- picks the time-FFT length class, places the event's grids
// in fixed event slots, and writes the work-item prefixes that the persistent
// raster, time-FFT, wire-convolution and inverse kernels walk.
// ===========================================================================
}  // namespace wctb200

#include "fft_lengths.h"

namespace wctb200 {

__constant__ int c_fbl_any[] = {WCT_FFT_LENGTHS_ANY};
__constant__ int c_fbl_even[] = {WCT_FFT_LENGTHS_EVEN};
__constant__ int c_fbl_odd[] = {WCT_FFT_LENGTHS_ODD};

template <int N>
__device__ __forceinline__ int fbl_pick(const int (&t)[N], int n)
{
    if (n <= t[N - 1])
        for (int i = 0; i < N; ++i)
            if (t[i] >= n) return t[i];
    return n;
}

// fft_best_length (util/src/FFTBestLength.cxx:12-59)
__device__ int fft_best_length_dev(int n, bool keep_odd_even)
{
    if (!keep_odd_even) return fbl_pick(c_fbl_any, n);
    return (n % 2 == 0) ? fbl_pick(c_fbl_even, n) : fbl_pick(c_fbl_odd, n);
}

// The window of one (event, plane) from its reduced depo extents: the same
// arithmetic, in the same double operations, as the host path.
__device__ void window_dev(const BatchStatic& bs, int ip, const WindowDev& w, EvPlane& o)
{
    const BatchPlaneStatic& pl = bs.pl[ip];
    double pmin = 0, pmax = 0, tmin = 0, tmax = 0;  // gausdesc_range of an empty set
    if (w.nadded > 0) {
        pmin = dkey_inv(w.pmin);
        pmax = dkey_inv(w.pmax);
        tmin = dkey_inv(w.tmin);
        tmax = dkey_inv(w.tmax);
    }
    auto ibin = [&](double v) { return __double2int_rz(__ddiv_rn(__dsub_rn(v, pl.imp_min), pl.imp_bs)); };
    auto tbin = [&](double v) { return __double2int_rz(__ddiv_rn(__dsub_rn(v, bs.start_time), bs.tbs)); };
    const int i0 = max(ibin(pmin), 0), i1 = min(ibin(pmax) + 1, pl.imp_nbins);
    const int t0 = max(tbin(tmin), 0), t1 = min(tbin(tmax) + 1, bs.nticks);
    const int G = pl.G;
    int start_ch = (int)floor(__ddiv_rn((double)i0, (double)(G - 1))) - 1;
    int end_ch = (int)ceil(__ddiv_rn((double)i1, (double)(G - 1))) + 2;
    if ((end_ch - start_ch) % 2 == 1) end_ch += 1;
    int start_tick = t0 - 1;
    int end_tick = t1 + 2;
    if ((end_tick - start_tick) % 2 == 1) end_tick += 1;
    const int ntw = fft_best_length_dev(end_ch - start_ch + 2 * pl.npad, true);
    const int npad_wire = (ntw - end_ch + start_ch) / 2;
    const int ntt = fft_best_length_dev(end_tick - start_tick + pl.waveform_pad, false);
    const int npad_time = ntt - end_tick + start_tick;
    o.start_ch = start_ch;
    o.end_ch = end_ch;
    o.start_tick = start_tick;
    o.end_tick = end_tick;
    o.m_start_ch = start_ch - npad_wire;
    o.m_end_ch = end_ch + npad_wire;
    o.m_start_tick = start_tick;
    o.m_end_tick = end_tick + npad_time;
    o.nw_ref = end_ch - start_ch + 2 * npad_wire;
    o.nt_ref = o.m_end_tick - o.m_start_tick;
    o.ndepos_added = w.nadded;
    o.outside_time = w.out_time;
    o.outside_pitch = w.out_pitch;
}

__device__ __forceinline__ int fdiv_floor(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

// One block of 256 threads: windows and work counts per (event, plane), then
// the prefixes (thread 0; at most kMaxBatch * kMaxPlanes entries).
__global__ void __launch_bounds__(256) k_plan_batch(BatchPlan* __restrict__ plan, BatchStatic bs, int nev,
                                                    const WindowDev* __restrict__ win,
                                                    long long vcap)
{
    __shared__ int s_status;
    __shared__ int c_raster[kMaxBatch * kMaxPlanes], c_rows[kMaxBatch * kMaxPlanes],
        c_orows[kMaxBatch * kMaxPlanes], c_conv[kMaxBatch * kMaxPlanes], c_wire[kMaxBatch * kMaxPlanes];
    const int np = bs.np, ne = nev * np;
    if (threadIdx.x == 0) s_status = 0;
    __syncthreads();
    for (int k = threadIdx.x; k < ne; k += blockDim.x) {
        const int e = k / np, ip = k - e * np;
        const WindowDev& w = win[k];
        EvPlane o{};
        window_dev(bs, ip, w, o);
        const BatchPlaneStatic& pl = bs.pl[ip];
        int st = 0;
        if (w.oversize) st |= kBatchOversize;
        if (w.bigcharge) st |= kBatchBigCharge;
        o.nin = w.nadded > 0 ? o.end_ch - o.start_ch : 0;
        o.nout = o.nin ? o.nin + 2 * pl.npad : 0;
        o.ncols = o.end_tick - o.start_tick;
        int cls = -1;
        for (int c = 0; c < bs.ncls; ++c)
            if (bs.cls_N[c] >= o.nt_ref) {
                cls = c;
                break;
            }
        if (cls < 0 || o.nin > pl.nin_max) {
            if (o.nin) st |= kBatchNoClass;
            o.nin = o.nout = 0;
            cls = 0;
        }
        o.cls = cls;
        o.N = bs.cls_N[cls];
        o.M = o.N / 2;
        o.ktile0 = fdiv_floor(o.start_tick, kTile);
        o.ntile = fdiv_floor(o.start_tick + o.N - 1, kTile) - o.ktile0 + 1;
        o.qoff = (long long)e * bs.qslot_total + pl.qslot;
        o.voff = (long long)e * bs.vslot_total + pl.vslot;
        plan->ep[k] = o;
        c_raster[k] = o.nin * o.ntile;
        c_rows[k] = bs.cls_fft3[cls] ? 0 : pl.G * o.nin;
        c_orows[k] = bs.cls_fft3[cls] ? 0 : o.nout;
        const bool wire = (pl.wire_cls >> cls) & 1;
        c_conv[k] = wire || !o.nin ? 0 : ((o.M + 31) / 32) * ((o.nout + kConvRows - 1) / kConvRows);
        c_wire[k] = wire && o.nin ? wire_fblocks(o.M) * wire_blocks(o.nout, pl.npad) : 0;
        if (st) atomicOr(&s_status, st);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int a = 0, b = 0, c = 0;
        for (int k = 0; k < ne; ++k) {
            plan->pre_raster[k] = a;
            plan->pre_rows[k] = b;
            plan->pre_orows[k] = c;
            a += c_raster[k];
            b += c_rows[k];
            c += c_orows[k];
        }
        plan->pre_raster[ne] = a;
        plan->pre_rows[ne] = b;
        plan->pre_orows[ne] = c;
        for (int ip = 0; ip < np; ++ip) {
            int t = 0, u = 0;
            for (int e = 0; e < nev; ++e) {
                plan->pre_conv[ip][e] = t;
                plan->pre_wire[ip][e] = u;
                t += c_conv[e * np + ip];
                u += c_wire[e * np + ip];
            }
            plan->pre_conv[ip][nev] = t;
            plan->pre_wire[ip][nev] = u;
        }
        unsigned long long tv = 0;  // visits of the pass, 64-bit (the list offsets are int)
        for (int e = 0; e < nev; ++e) tv += win[(size_t)e * np].nvisits;
        plan->total_visits = (long long)tv;
        plan->nev = nev;
        plan->np = np;
        plan->status = s_status | (tv > (unsigned long long)vcap ? kBatchVisitOverflow : 0) |
                       (tv >= 0x7fffffffull ? kBatchTooBig : 0);
        for (int k = 0; k < 4 + kMaxPlanes; ++k) plan->next[k] = 0;
    }
}

void launch_plan_batch(BatchPlan* plan, const BatchStatic& bs, int nev, const WindowDev* win, long long vcap,
                       cudaStream_t s)
{
    k_plan_batch<<<1, 256, 0, s>>>(plan, bs, nev, win, vcap);
}

// Next work item of a persistent block (all threads get the same value):
// blocks take items from a shared counter, so a block that drew a heavy item
// does not hold back the rest.
__device__ __forceinline__ int next_item(int* counter, int* s_item)
{
    if (threadIdx.x == 0 && threadIdx.y == 0) *s_item = atomicAdd(counter, 1);
    __syncthreads();
    const int item = *s_item;
    __syncthreads();  // every thread has read it before the next draw overwrites it
    return item;
}

// Index of the (event, plane) entry whose item range holds `item`: the last
// k in [0, n) with pre[k] <= item (entries with no items are skipped).
__device__ __forceinline__ int find_entry(const int* __restrict__ pre, int n, int item)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pre[mid] <= item) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The raster parameters of work item `item` of a pass: its event, plane, row and tile.
__device__ __forceinline__ GridPlane batch_tile(const BatchPlan* __restrict__ plan, const BatchStatic& bs,
                                                const PlaneSet& ps, long long recstride, int item, int& e, int& ip,
                                                int& row, int& ktile)
{
    const int k = find_entry(plan->pre_raster, plan->nev * plan->np, item);
    e = k / plan->np;
    ip = k - e * plan->np;
    const EvPlane& E = plan->ep[k];
    GridPlane P;
    P.nimp = ps.p[ip].nimp;
    P.G = bs.pl[ip].G;
    P.nwires = ps.p[ip].nwires;
    P.wire_base = ps.p[ip].wire_base;
    P.start_ch = E.start_ch;
    P.nin = E.nin;
    P.col0 = E.start_tick;
    P.ncols = E.ncols;
    P.N = E.N;
    P.tbs = (float)bs.tbs;
    P.pbs = (float)ps.p[ip].imp_bs;
    P.qoff = E.qoff;
    P.recoff = (long long)ip * recstride;
    P.row_base = 0;
    P.ktile0 = E.ktile0;
    P.ntile = E.ntile;
    P.sparse = bs.cls_fft3[E.cls];  // taken by k_rfft3_batch
    const int rel = item - plan->pre_raster[k];
    row = rel / E.ntile;
    ktile = E.ktile0 + (rel - row * E.ntile);
    return P;
}

template <bool FLUC>
__global__ void __launch_bounds__(FLUC ? kRasterThreads : kLightThreads, FLUC ? 4 : kLightBlocks)
    k_raster_batch(const BatchPlan* __restrict__ plan, BatchStatic bs, PlaneSet ps, const PatchRec* __restrict__ rec,
                   long long recstride, const float* __restrict__ tprof, TprofPool pool,
                   const unsigned char* __restrict__ wide_key, const int* __restrict__ wire_cnt,
                   const int* __restrict__ wire_off, const Visit* __restrict__ visits, long long vcap,
                   const unsigned long long* __restrict__ key_bound, float* __restrict__ Q, EventTable evt,
                   FlucParams fp, const FlucRec* __restrict__ fluc, const int* __restrict__ draws,
                   unsigned char* __restrict__ row_flag, HeavyList heavy)
{
    extern __shared__ int smem_i[];
    __shared__ float scale[kTileBlocks], iscale[kTileBlocks];
    if (plan->status & kBatchSkip) return;
    __shared__ int s_item;
    const int total = plan->pre_raster[plan->nev * plan->np];
    int* ctr = const_cast<int*>(&plan->next[0]);
    for (int item = next_item(ctr, &s_item); item < total; item = next_item(ctr, &s_item)) {
        int e, ip, row, ktile;
        const GridPlane P = batch_tile(plan, bs, ps, recstride, item, e, ip, row, ktile);
        unsigned char* flags = row_flag + (size_t)e * bs.nwires_total;
        if constexpr (FLUC)
            raster_tile_fluc(P, ip, row, ktile, e * bs.nkeys, bs.ntiles, evt, fp, rec, fluc, draws, wire_cnt, wire_off,
                             visits, vcap, Q, flags, reinterpret_cast<long long*>(smem_i));
        else
            raster_tile<false, kLightThreads, true>(P, row, ktile, e * bs.nkeys, bs.ntiles, rec, tprof, pool, wide_key,
                                                    wire_cnt, wire_off, visits, vcap, key_bound, Q, flags, heavy, item,
                                                    0, 1, 0, smem_i, scale, iscale);
    }
}

__global__ void __launch_bounds__(kRasterThreads, kMidBlocks)
    k_raster_mid_batch(const BatchPlan* __restrict__ plan, BatchStatic bs, PlaneSet ps,
                       const PatchRec* __restrict__ rec, long long recstride, const float* __restrict__ tprof,
                       TprofPool pool, const unsigned char* __restrict__ wide_key,
                       const int* __restrict__ wire_cnt, const int* __restrict__ wire_off,
                       const Visit* __restrict__ visits, long long vcap,
                       const unsigned long long* __restrict__ key_bound, float* __restrict__ Q,
                       unsigned char* __restrict__ row_flag, HeavyList heavy)
{
    extern __shared__ int smem_i[];
    __shared__ float scale[kTileBlocks], iscale[kTileBlocks];
    if (plan->status & kBatchSkip) return;
    for (int it = next_mid(heavy); it >= 0; it = next_mid(heavy)) {
        int e, ip, row, ktile;
        const GridPlane P = batch_tile(plan, bs, ps, recstride, it, e, ip, row, ktile);
        raster_tile<false, kRasterThreads, false>(P, row, ktile, e * bs.nkeys, bs.ntiles, rec, tprof, pool, wide_key,
                                                  wire_cnt, wire_off, visits, vcap, key_bound, Q,
                                                  row_flag + (size_t)e * bs.nwires_total, heavy, it, 0, 1, 0, smem_i,
                                                  scale, iscale);
    }
}

__global__ void __launch_bounds__(kRasterThreads, kHeavyBlocks)
    k_raster_heavy_batch(const BatchPlan* __restrict__ plan, BatchStatic bs, PlaneSet ps,
                         const PatchRec* __restrict__ rec, long long recstride, const float* __restrict__ tprof,
                         TprofPool pool, const unsigned char* __restrict__ wide_key,
                         const int* __restrict__ wire_cnt, const int* __restrict__ wire_off,
                         const Visit* __restrict__ visits, long long vcap,
                         const unsigned long long* __restrict__ key_bound, float* __restrict__ Q,
                         unsigned char* __restrict__ row_flag, HeavyList heavy)
{
    extern __shared__ int smem_i[];
    __shared__ float scale[kTileBlocks], iscale[kTileBlocks];
    if (plan->status & kBatchSkip) return;
    const int total = heavy.count[0];
    for (int k = blockIdx.x; k < total; k += gridDim.x) {
        const int4 it = heavy.item[k];
        int e, ip, row, ktile;
        const GridPlane P = batch_tile(plan, bs, ps, recstride, it.x, e, ip, row, ktile);
        raster_tile<true, kRasterThreads, false>(P, row, ktile, e * bs.nkeys, bs.ntiles, rec, tprof, pool, wide_key, wire_cnt, wire_off,
                          visits, vcap, key_bound, Q, row_flag + (size_t)e * bs.nwires_total, heavy, it.x, it.y, it.z,
                          it.w, smem_i, scale, iscale);
    }
}

void launch_raster_batch(const BatchPlan* plan, const BatchStatic& bs, const PlaneSet& ps, const PatchRec* rec,
                         long long recstride, const float* tprof, const TprofPool& pool,
                         const unsigned char* wide_key, const int* wire_cnt, const int* wire_off,
                         const Visit* visits, long long vcap, const unsigned long long* key_bound, float* Q,
                         int nblocks, int maxG, const EventTable& evt, const FlucParams& fp, const FlucRec* fluc,
                         const int* draws, unsigned char* row_flag, const HeavyList& heavy, int nsm,
                         cudaStream_t s)
{
    if (fp.on_patch) {
        k_raster_batch<true><<<nblocks, kRasterThreads, raster_fluc_smem_bytes(maxG), s>>>(
            plan, bs, ps, rec, recstride, tprof, pool, wide_key, wire_cnt, wire_off, visits, vcap, key_bound, Q, evt,
            fp, fluc, draws, row_flag, heavy);
        return;
    }
    k_raster_batch<false><<<kLightBlocks * nsm, kLightThreads, raster_smem(maxG, kLightThreads), s>>>(
        plan, bs, ps, rec, recstride, tprof, pool, wide_key, wire_cnt, wire_off, visits, vcap, key_bound, Q, evt, fp,
        fluc, draws, row_flag, heavy);
    k_raster_mid_batch<<<nblocks, kRasterThreads, raster_smem_bytes(maxG), s>>>(
        plan, bs, ps, rec, recstride, tprof, pool, wide_key, wire_cnt, wire_off, visits, vcap, key_bound, Q, row_flag,
        heavy);
    k_raster_heavy_batch<<<kHeavyBlocks * nsm, kRasterThreads, raster_heavy_smem_bytes(maxG), s>>>(
        plan, bs, ps, rec, recstride, tprof, pool, wide_key, wire_cnt, wire_off, visits, vcap, key_bound, Q, row_flag,
        heavy);
}

// Time FFT of every charge-grid row of the pass, in place (rows of N reals
// become M packed bins), whatever their length class.
__global__ void k_rfft_batch(const BatchPlan* __restrict__ plan, const FftDesc* __restrict__ descs,
                             float* __restrict__ Q)
{
    extern __shared__ float2 sm[];
    if (plan->status & kBatchSkip) return;
    __shared__ int s_item;
    const int ne = plan->nev * plan->np;
    const int total = plan->pre_rows[ne];
    int* ctr = const_cast<int*>(&plan->next[1]);
    for (int item = next_item(ctr, &s_item); item < total; item = next_item(ctr, &s_item)) {
        const int k = find_entry(plan->pre_rows, ne, item);
        const EvPlane& E = plan->ep[k];
        const FftDesc d = descs[E.cls];
        float* x = Q + E.qoff + (size_t)(item - plan->pre_rows[k]) * E.N;
        rfft_row(x, E.N, reinterpret_cast<float2*>(x), d, sm);
    }
}

void launch_rfft_batch(const BatchPlan* plan, const FftDesc* descs, float* Q, int nblocks, int nthreads, int maxM,
                       cudaStream_t s)
{
    const size_t smem = 2 * (size_t)maxM * sizeof(float2);
    k_rfft_batch<<<nblocks, nthreads, smem, s>>>(plan, descs, Q);
}

// PAD < 0: run-time pad (bs.pl[ip].npad) without shared-memory staging.
// Items of planes ip0 .. ip1-1 in order; within a plane, events in order.
template <int PAD, bool PAIR>
__global__ void __launch_bounds__(32 * kConvRG, PAD < 0 ? 1 : 3) k_conv_batch(const BatchPlan* __restrict__ plan, BatchStatic bs,
                                                             int ip0, int ip1, const float2* const* __restrict__ spec,
                                                             const float* __restrict__ Q, float2* __restrict__ V)
{
    extern __shared__ float2 conv_smem[];
    __shared__ int s_item;
    if (plan->status & kBatchSkip) return;
    const int nev = plan->nev, np = plan->np;
    int total = 0;
    for (int ip = ip0; ip < ip1; ++ip) total += plan->pre_conv[ip][nev];
    int* ctr = const_cast<int*>(&plan->next[4 + ip0]);
    for (int item = next_item(ctr, &s_item); item < total; item = next_item(ctr, &s_item)) {
        int ip = ip0, rel = item;
        while (rel >= plan->pre_conv[ip][nev]) {
            rel -= plan->pre_conv[ip][nev];
            ++ip;
        }
        const int* pre = plan->pre_conv[ip];
        const int e = find_entry(pre, nev, rel);
        const EvPlane& E = plan->ep[e * np + ip];
        rel -= pre[e];
        const int nfb = (E.M + 31) / 32;
        const int oblk = rel / nfb, fblk = rel - oblk * nfb;
        const float2* Qh = reinterpret_cast<const float2*>(Q + E.qoff);
        const float2* R = spec[(size_t)ip * bs.ncls + E.cls];
        if constexpr (PAD >= 0)
            wire_conv_tile<PAD, PAIR>(Qh, R, V + E.voff, bs.pl[ip].G, E.nin, E.nout, E.M, fblk, oblk, conv_smem);
        else {
            const int f = fblk * 32 + threadIdx.x, o0 = oblk * kConvRows + threadIdx.y * kConvRB;
            if (f < E.M)
                conv_rows_any(Qh, R, V + E.voff, bs.pl[ip].G, bs.pl[ip].npad, E.nin, E.M, f, o0,
                              o0 + kConvRB <= E.nout ? 0xffu : (1u << max(E.nout - o0, 0)) - 1u);
        }
    }
}

// The same by overlap-save (wire_fft.cuh): the items of every plane.
__global__ void __launch_bounds__(kWThreads, 2) k_conv_fft_batch(const BatchPlan* __restrict__ plan, BatchStatic bs,
                                                                 const float2* const* __restrict__ wspec,
                                                                 const float* __restrict__ Q, float2* __restrict__ V,
                                                                 double* __restrict__ energy)
{
    extern __shared__ float2 wsm[];
    __shared__ int s_item;
    if (plan->status & kBatchSkip) return;
    wfft::load_twiddles(wsm + 2 * kWEx, threadIdx.x);
    const int nev = plan->nev, np = plan->np;
    int total = 0;
    for (int ip = 0; ip < np; ++ip) total += plan->pre_wire[ip][nev];
    int* ctr = const_cast<int*>(&plan->next[3]);
    for (int item = next_item(ctr, &s_item); item < total; item = next_item(ctr, &s_item)) {
        int ip = 0, rel = item;
        while (rel >= plan->pre_wire[ip][nev]) {
            rel -= plan->pre_wire[ip][nev];
            ++ip;
        }
        const int* pre = plan->pre_wire[ip];
        const int e = find_entry(pre, nev, rel);
        const EvPlane& E = plan->ep[e * np + ip];
        rel -= pre[e];
        const int nfb = wire_fblocks(E.M);
        const int oblk = rel / nfb, fblk = rel - oblk * nfb;
        wfft::conv_tile(reinterpret_cast<const float2*>(Q + E.qoff), wspec[(size_t)ip * bs.ncls + E.cls], V + E.voff,
                        bs.pl[ip].G, bs.pl[ip].npad, E.nin, E.nout, E.M, fblk, oblk,
                        energy + e * bs.eslot_total + bs.pl[ip].eslot + (size_t)rel * kWL, wsm);
    }
}

// Their faint rows: block x of a wire row block, y of an entry of the pass.
__global__ void __launch_bounds__(kPickThreads) k_pick_batch(const BatchPlan* __restrict__ plan, BatchStatic bs,
                                                             const double* __restrict__ energy,
                                                             const unsigned char* __restrict__ row_flag, RowList list)
{
    if (plan->status & kBatchSkip) return;
    const int k = blockIdx.y, e = k / bs.np, ip = k - e * bs.np;
    const EvPlane& E = plan->ep[k];
    const BatchPlaneStatic& pl = bs.pl[ip];
    if (!E.nin || !((pl.wire_cls >> E.cls) & 1) || (int)blockIdx.x >= wire_blocks(E.nout, pl.npad)) return;
    const int nfb = wire_fblocks(E.M);
    const WantRows want{E.start_ch - pl.npad, max(0, E.m_start_ch), min(pl.nwires, E.m_end_ch), pl.nwires,
                        row_flag + (size_t)e * bs.nwires_total + pl.wire_base, nullptr, 0};
    wfft::pick_tile<false>(energy + e * bs.eslot_total + pl.eslot + (size_t)blockIdx.x * nfb * kWL, nfb, pl.npad,
                           blockIdx.x, E.nout, want, k, list);
}

// The listed rows of planes ip0 .. ip1-1, all of one pad and pairing (PAD 0: run-time pad).
template <int PAD, bool PAIR>
__global__ void __launch_bounds__(kConv2F * kConvGroups) k_rows_batch(const BatchPlan* __restrict__ plan, BatchStatic bs,
                                                                  int ip0, int ip1, int nf,
                                                                  const float2* const* __restrict__ spec,
                                                                  const float* __restrict__ Q, float2* V, RowList list)
{
    extern __shared__ __align__(16) float2 conv2_smem[];
    if (plan->status & kBatchSkip) return;
    const long long total = (long long)list.count[1] * nf;
    for (long long u = blockIdx.x; u < total; u += gridDim.x) {
        const int i = (int)(u / nf), f0 = (int)(u - (long long)i * nf) * kConv2F;
        const int4 c = list.chunk[i];
        const int e = c.z / bs.np, ip = c.z - e * bs.np;
        const EvPlane& E = plan->ep[c.z];
        if (ip < ip0 || ip >= ip1 || f0 >= E.M) continue;
        const float2* Qh = reinterpret_cast<const float2*>(Q + E.qoff);
        const float2* R = spec[(size_t)ip * bs.ncls + E.cls];
        conv2_chunk<PAD, PAIR>(Qh, R, V + E.voff, bs.pl[ip].G, bs.pl[ip].npad, E.nin, E.M, f0, list, c, conv2_smem);
    }
}

void launch_conv_fft_batch(const BatchPlan* plan, const BatchStatic& bs, int nev, int maxblocks,
                           const float2* const* wspec, const float* Q, float2* V, double* energy,
                           const unsigned char* row_flag, const RowList& list, int nblocks, cudaStream_t s)
{
    k_conv_fft_batch<<<nblocks, kWThreads, kWConvSmem, s>>>(plan, bs, wspec, Q, V, energy);
    k_pick_batch<<<dim3(maxblocks, nev * bs.np), kPickThreads, 0, s>>>(plan, bs, energy, row_flag, list);
}

// f(std::integral_constant PAD, bool_constant PAIR): the pads with taps unrolled,
// 0 (run-time pad) for others.
template <class F>
static void with_pad(int npad, bool pair, F f)
{
    auto go = [&](auto pad) {
        if (pair) f(pad, std::true_type{});
        else f(pad, std::false_type{});
    };
    if (npad == 10) go(std::integral_constant<int, 10>{});
    else if (npad == 21) go(std::integral_constant<int, 21>{});
    else go(std::integral_constant<int, 0>{});
}

void launch_rows_batch(const BatchPlan* plan, const BatchStatic& bs, int ip0, int ip1, bool pair, int maxM,
                       const float2* const* spec, const float* Q, float2* V, const RowList& list, int nblocks,
                       cudaStream_t s)
{
    const int nf = (maxM + kConv2F - 1) / kConv2F, npad = bs.pl[ip0].npad;
    with_pad(npad, pair, [&](auto PAD, auto PAIR) {
        const size_t sm = 2 * conv2_stage_f2<PAIR.value, kConvGroups>(npad) * sizeof(float2);
        k_rows_batch<PAD.value, PAIR.value>
            <<<nblocks, kConv2F * kConvGroups, sm, s>>>(plan, bs, ip0, ip1, nf, spec, Q, V, list);
    });
}

void launch_wire_rows(const float2* Qh, const float2* taps, float2* Vh, int G, int npad, int nin, int nout, int M,
                      bool pair, const RowList& list, cudaStream_t s)
{
    with_pad(npad, pair, [&](auto PAD, auto PAIR) {
        const size_t sm = 2 * conv2_stage_f2<PAIR.value, kConvGroups>(npad) * sizeof(float2);
        allow_smem((const void*)k_wire_rows2<PAD.value, PAIR.value>, sm);
        k_wire_rows2<PAD.value, PAIR.value>
            <<<kRowsBlocks, kConv2F * kConvGroups, sm, s>>>(Qh, taps, Vh, G, npad, nin, M, list);
    });
}

size_t conv_smem_bytes(int npad, bool pair)
{
    if (npad != 10 && npad != 21) return 0;
    return sizeof(float2) * 32 * ((size_t)(pair ? 2 : 1) * (kConvRows + 2 * npad) + (2 * npad + 1));
}

void launch_conv_batch(const BatchPlan* plan, const BatchStatic& bs, int ip0, int ip1, bool pair,
                       const float2* const* spec, const float* Q, float2* V, int nblocks, cudaStream_t s)
{
    const int npad = bs.pl[ip0].npad;
    dim3 block(32, kConvRG);
    const size_t sm = conv_smem_bytes(npad, pair);
#define WCT_CONVB(P, B) k_conv_batch<P, B><<<nblocks, block, sm, s>>>(plan, bs, ip0, ip1, spec, Q, V)
    if (npad == 10 && pair) WCT_CONVB(10, true);
    else if (npad == 10) WCT_CONVB(10, false);
    else if (npad == 21 && pair) WCT_CONVB(21, true);
    else if (npad == 21) WCT_CONVB(21, false);
#undef WCT_CONVB
    else k_conv_batch<-1, false><<<nblocks, block, 0, s>>>(plan, bs, ip0, ip1, spec, Q, V);
}

// Inverse time FFT of every V row of the pass and the frame write of its event.
__global__ void k_irfft_batch(const BatchPlan* __restrict__ plan, BatchStatic bs, const FftDesc* __restrict__ descs,
                              const float2* __restrict__ V, float* __restrict__ frames, long long frame_stride,
                              const unsigned char* __restrict__ row_flag)
{
    extern __shared__ float2 sm[];
    if (plan->status & kBatchSkip) return;
    __shared__ int s_item;
    const int ne = plan->nev * plan->np;
    const int total = plan->pre_orows[ne];
    int* ctr = const_cast<int*>(&plan->next[2]);
    for (int item = next_item(ctr, &s_item); item < total; item = next_item(ctr, &s_item)) {
        const int k = find_entry(plan->pre_orows, ne, item);
        const int e = k / plan->np, ip = k - e * plan->np;
        const EvPlane& E = plan->ep[k];
        const BatchPlaneStatic& pl = bs.pl[ip];
        const int o = item - plan->pre_orows[k];
        const int W = E.start_ch - pl.npad + o;
        const int wlo = max(0, E.m_start_ch), whi = min(pl.nwires, E.m_end_ch);
        if (W < wlo || W >= whi) continue;  // uniform over the block
        if (!row_reached(row_flag + (size_t)e * bs.nwires_total + pl.wire_base, pl.nwires, W, pl.npad)) continue;
        const FftDesc d = descs[E.cls];
        irfft_row(V + E.voff + (size_t)o * E.M, d, frames + (size_t)e * frame_stride + (size_t)(pl.row0 + W) * bs.nticks,
                  E.start_tick, min(E.N, E.nt_ref), bs.nticks, sm);
    }
}

void launch_irfft_batch(const BatchPlan* plan, const BatchStatic& bs, const FftDesc* descs, const float2* V,
                        float* frames, long long frame_stride, int nblocks, int nthreads, int maxM,
                        const unsigned char* row_flag, cudaStream_t s)
{
    const size_t smem = 2 * (size_t)maxM * sizeof(float2);
    k_irfft_batch<<<nblocks, nthreads, smem, s>>>(plan, bs, descs, V, frames, frame_stride, row_flag);
}

// Shared-memory opt-ins of the batched kernels, set before a graph capture
// (the launchers themselves only enqueue).
void batch_kernel_attributes(int maxG, int maxM)
{
    const int sr = (int)std::max(raster_smem_bytes(maxG), raster_fluc_smem_bytes(maxG));
    const int sf = (int)(2 * (size_t)maxM * sizeof(float2));
    cudaFuncSetAttribute((const void*)k_raster_batch<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sr);
    cudaFuncSetAttribute((const void*)k_raster_batch<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sr);
    cudaFuncSetAttribute((const void*)k_raster_mid_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, sr);
    cudaFuncSetAttribute((const void*)k_raster_heavy_batch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)raster_heavy_smem_bytes(maxG));
    cudaFuncSetAttribute((const void*)k_rfft_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, sf);
    cudaFuncSetAttribute((const void*)k_irfft_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, sf);
    cudaFuncSetAttribute((const void*)k_conv_fft_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWConvSmem);
    for (int npad : {10, 21, kWMaxPad})
        for (bool pair : {false, true})
            with_pad(npad, pair, [&](auto PAD, auto PAIR) {
                cudaFuncSetAttribute((const void*)k_rows_batch<PAD.value, PAIR.value>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(2 * conv2_stage_f2<PAIR.value, kConvGroups>(npad) * sizeof(float2)));
            });
    cudaFuncSetAttribute((const void*)k_conv_batch<10, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)conv_smem_bytes(10, true));
    cudaFuncSetAttribute((const void*)k_conv_batch<10, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)conv_smem_bytes(10, false));
    cudaFuncSetAttribute((const void*)k_conv_batch<21, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)conv_smem_bytes(21, true));
    cudaFuncSetAttribute((const void*)k_conv_batch<21, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)conv_smem_bytes(21, false));
}

}  // namespace wctb200
