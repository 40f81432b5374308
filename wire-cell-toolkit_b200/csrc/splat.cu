// DepoFluxSplat (gen/src/DepoFluxSplat.cxx:247-390): the truth frame of the
// depos' diffused charge on (wire, tick), no response.  One warp per depo,
// the planes in order as the reference visits them: a depo whose time span
// misses the window skips the plane, one whose pitch span misses the wire
// plane skips the remaining planes (the reference's `break`).  The patch is
// GaussianDiffusion::set_sampling (gen/src/GaussianDiffusion.cxx:116-182) on
// the window's tick binning and the plane's wire (region) binning
// (util/src/Pimpos.cxx:5-30): double erf bin integrals (GausDesc::binint,
// :30-56), float cells p_k t_j scaled by (float)(Q / sum), the absolute
// value added (double atomics) at row wire, tick toffset + tick offset + j.
#include <algorithm>

#include "kernels.cuh"

namespace wctb200 {

namespace {
__device__ __forceinline__ int sbin(double v, double lo, double bs)
{
    return __double2int_rz(__ddiv_rn(__dsub_rn(v, lo), bs));  // Binning::bin
}
__device__ __forceinline__ double sedge(int i, double lo, double bs)
{
    return __dadd_rn(lo, __dmul_rn((double)i, bs));  // Binning::edge
}
__device__ __forceinline__ double sdist(double x, double c, double s)
{
    return s != 0.0 ? __ddiv_rn(__dsub_rn(x, c), s) : __dsub_rn(x, c);  // GausDesc::distance
}
// Half the erf of bin edge k (start + step * k) from the centre: GausDesc::binint
// is the difference of two neighbours.
__device__ __forceinline__ double half_erf(double start, double step, int k, double c, double d)
{
    return __dmul_rn(0.5, erf(__ddiv_rn(__dsub_rn(__dadd_rn(start, __dmul_rn(step, (double)k)), c), d)));
}
__device__ __forceinline__ double lane_value(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
}  // namespace

// One warp per depo.  Lane ip works out plane ip's widths and windows (FP64
// divisions and square roots: once a depo, not once a plane), then the warp
// takes the planes in turn: an edge per lane (time edges, and the pitch edges
// in the lanes left over where both fit), bins from neighbouring lanes, and
// the cells row by row, a tick per lane.  With a thread per depo every cell
// evaluated four erf, twice over, and the atomics of a warp hit 32 rows:
// 200k depos (60 % tracks, 40 % showers of 100 ticks) on three planes took
// 42 ms and take 0.73 ms, bound by the FP64 edges and the atomics.
constexpr int kSplatWarps = 8;
constexpr int kSplatPitch = 32;  // pitch bins tabulated at a time

__global__ void __launch_bounds__(kSplatWarps * 32) k_splat(const double* __restrict__ dep, int n, PlaneSet ps,
                                                            SplatParams sp, double* __restrict__ acc)
{
    __shared__ double s_pv[kSplatWarps][kSplatPitch];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int i = blockIdx.x * kSplatWarps + wib;
    if (i >= n) return;  // whole warps
    const double* p = dep + 7 * (size_t)i;
    const double t = p[0], q = p[1], x = p[2], y = p[3], z = p[4], el = p[5], et = p[6];
    // a depo with a NaN or infinite value is dropped, as the transform drops it:
    // its bin arithmetic is undefined and it would put NaNs in the frame
    if (!(isfinite(t) && isfinite(q) && isfinite(x) && isfinite(y) && isfinite(z) && isfinite(el) && isfinite(et)))
        return;
    if (ps.nplanes > 0 && ps.p[0].have_bb) {  // the face's sensitive volume
        const double pp[3] = {x, y, z};
        for (int k = 0; k < 3; ++k) {
            const double b1 = ps.p[0].bb_lo[k], b2 = ps.p[0].bb_hi[k];
            if (b1 < b2) { if (pp[k] < b1 || pp[k] > b2) return; }
            else if (b2 < b1) { if (pp[k] < b2 || pp[k] > b1) return; }
        }
    }
    const double nominal = __dadd_rn(t, sp.time_shift);
    const TimeDev& tb = sp.tb;
    // plane `lane`: 0 nothing to add, 1 a patch, 2 a pitch miss (skips the planes after it)
    int state = 0, t0 = 0, p0 = 0, nt = 0, np = 0;
    double st = 0, sT = 0, cp = 0, rbs = 0, rlo = 0;
    if (lane < ps.nplanes) {
        const PlaneDev& pl = ps.p[lane];
        const SplatPlane& spl = sp.pl[lane];
        double sL = el;
        if (spl.smear_long > 0) {
            const double extra = __dmul_rn(__dmul_rn(spl.smear_long, tb.bs), sp.speed);
            sL = __dsqrt_rn(__dadd_rn(__dmul_rn(sL, sL), __dmul_rn(extra, extra)));
        }
        st = __ddiv_rn(sL, sp.speed);
        const double eff_t = el > 0 ? sp.nsigma : 0.0;
        if (!(sdist(tb.tmin, nominal, st) > eff_t || sdist(tb.tmax, nominal, st) < -eff_t)) {
            rlo = pl.imp_min;
            const double rhi = pl.imp_max;
            rbs = __ddiv_rn(__dsub_rn(rhi, rlo), (double)pl.nwires);
            sT = et;
            if (spl.smear_tran > 0) {
                const double extra = __dmul_rn(spl.smear_tran, rbs);
                sT = __dsqrt_rn(__dadd_rn(__dmul_rn(sT, sT), __dmul_rn(extra, extra)));
            }
            cp = __dadd_rn(__dadd_rn(__dmul_rn(pl.ax, __dsub_rn(x, pl.ox)), __dmul_rn(pl.ay, __dsub_rn(y, pl.oy))),
                           __dmul_rn(pl.az, __dsub_rn(z, pl.oz)));
            const double eff_p = et > 0 ? sp.nsigma : 0.0;
            if (sdist(rlo, cp, sT) > eff_p || sdist(rhi, cp, sT) < -eff_p) state = 2;
            else {
                // set_sampling windows (Binning::sample_bin_range)
                t0 = max(sbin(__dsub_rn(nominal, __dmul_rn(st, sp.nsigma)), tb.tmin, tb.bs), 0);
                const int t1 = min(sbin(__dadd_rn(nominal, __dmul_rn(st, sp.nsigma)), tb.tmin, tb.bs) + 1, tb.nbins);
                p0 = max(sbin(__dsub_rn(cp, __dmul_rn(sT, sp.nsigma)), rlo, rbs), 0);
                const int p1 = min(sbin(__dadd_rn(cp, __dmul_rn(sT, sp.nsigma)), rlo, rbs) + 1, pl.nwires);
                if (t1 > t0 && p1 > p0) {
                    state = 1;
                    nt = st == 0.0 ? 1 : t1 - t0;
                    np = sT == 0.0 ? 1 : p1 - p0;
                }
            }
        }
    }
    const double rt2 = 1.41421356237309515;  // sqrt(2.0) rounded to double
    for (int ip = 0; ip < ps.nplanes; ++ip) {
        const int what = __shfl_sync(full, state, ip);
        if (what == 2) break;  // uniform
        if (what == 0) continue;
        const int b_t0 = __shfl_sync(full, t0, ip), b_p0 = __shfl_sync(full, p0, ip);
        const int b_nt = __shfl_sync(full, nt, ip), b_np = __shfl_sync(full, np, ip);
        const double b_st = lane_value(st, ip), b_sT = lane_value(sT, ip), b_cp = lane_value(cp, ip);
        const double b_rbs = lane_value(rbs, ip);
        const double ts = sedge(b_t0, tb.tmin, tb.bs), ps0 = sedge(b_p0, lane_value(rlo, ip), b_rbs);
        const double dt = __dmul_rn(rt2, b_st), dp = __dmul_rn(rt2, b_sT);
        const int nwires = ps.p[ip].nwires;
        const int tstart = (int)((double)b_t0 + sp.pl[ip].tick_offset);
        double* base = acc + (size_t)ps.p[ip].wire_base * tb.nbins;
        // edges: lanes 0 .. nt hold the time edges and the next np + 1 the pitch edges where all fit;
        // else the pitch edges have rounds of their own
        const bool small = b_st > 0.0 && b_sT > 0.0 && b_nt + b_np + 2 <= 32;
        double e = 0.0;
        if (small) {
            const bool is_t = lane <= b_nt;
            const int k = is_t ? lane : lane - b_nt - 1;
            if (k <= b_np || is_t)
                e = half_erf(is_t ? ts : ps0, is_t ? tb.bs : b_rbs, k, is_t ? nominal : b_cp, is_t ? dt : dp);
        }
        // sum of the patch's unit integrals, edge to edge
        double sum_t = 1.0, sum_p = 1.0;
        if (small) {
            sum_t = __dsub_rn(lane_value(e, b_nt), lane_value(e, 0));
            sum_p = __dsub_rn(lane_value(e, b_nt + 1 + b_np), lane_value(e, b_nt + 1));
        }
        else {
            double f = 0.0;  // lanes 0, 1: time; 2, 3: pitch
            if (lane < 2 && b_st > 0.0) f = half_erf(ts, tb.bs, lane ? b_nt : 0, nominal, dt);
            if ((lane == 2 || lane == 3) && b_sT > 0.0) f = half_erf(ps0, b_rbs, lane == 3 ? b_np : 0, b_cp, dp);
            if (b_st > 0.0) sum_t = __dsub_rn(lane_value(f, 1), lane_value(f, 0));
            if (b_sT > 0.0) sum_p = __dsub_rn(lane_value(f, 3), lane_value(f, 2));
        }
        const float scale = (float)__ddiv_rn(q, __dmul_rn(sum_p, sum_t));
        for (int a0 = 0; a0 < b_np; a0 += kSplatPitch - 1) {
            const int na = min(kSplatPitch - 1, b_np - a0);
            double pv = 1.0;
            if (small) {
                const double lo = __shfl_sync(full, e, (b_nt + 1 + lane) & 31);
                const double hi = __shfl_sync(full, e, (b_nt + 2 + lane) & 31);
                pv = __dsub_rn(hi, lo);
            }
            else if (b_sT > 0.0) {
                const double f = lane <= na ? half_erf(ps0, b_rbs, a0 + lane, b_cp, dp) : 0.0;
                pv = __dsub_rn(__shfl_down_sync(full, f, 1), f);
            }
            __syncwarp();
            if (lane < na) s_pv[wib][lane] = pv;
            __syncwarp();
            for (int k0 = 0; k0 < b_nt; k0 += 31) {
                const int nk = min(31, b_nt - k0);
                double tv = 1.0;
                if (small) tv = __dsub_rn(__shfl_down_sync(full, e, 1), e);
                else if (b_st > 0.0) {
                    const double f = lane <= nk ? half_erf(ts, tb.bs, k0 + lane, nominal, dt) : 0.0;
                    tv = __dsub_rn(__shfl_down_sync(full, f, 1), f);
                }
                const int tick = tstart + k0 + lane;
                const bool on = lane < nk && tick >= 0 && tick < tb.nbins;
                for (int a = 0; a < na; ++a) {
                    const int wire = b_p0 + a0 + a;
                    if (wire < 0 || wire >= nwires || !on) continue;
                    const float v = (float)__dmul_rn(s_pv[wib][a], tv) * scale;
                    atomicAdd(base + (size_t)wire * tb.nbins + tick, (double)fabsf(v));
                }
            }
        }
    }
}

__global__ void k_splat_finish(const double* __restrict__ acc, float* __restrict__ frame, long long count)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < count;
         e += (long long)gridDim.x * blockDim.x)
        frame[e] = (float)acc[e];
}

void launch_splat_face(const double* depos, int n, const PlaneSet& ps, const SplatParams& sp, double* acc,
                       cudaStream_t s)
{
    if (n > 0 && ps.nplanes > 0)
        k_splat<<<(n + kSplatWarps - 1) / kSplatWarps, kSplatWarps * 32, 0, s>>>(depos, n, ps, sp, acc);
}

void launch_splat_finish(const double* acc, float* frame, long long count, cudaStream_t s)
{
    if (count <= 0) return;
    const long long blocks = std::min<long long>((count + 255) / 256, 148LL * 32);
    k_splat_finish<<<(unsigned)blocks, 256, 0, s>>>(acc, frame, count);
}

}  // namespace wctb200
