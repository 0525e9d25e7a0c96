// postprocess.cuh -- spectral post-processing on the device: the Gaussian line-spread function
// (apply_LSF / compute_LSF_matrix, src/utils.jl:45-58, 94-106, 132-155) and rotational
// broadening (apply_rotation, src/utils.jl:168-240), each with its reverse mode (both maps are
// linear in the flux, so the reverse mode is the transposed map).
//
//   lsf kernels:       one warp per output wavelength: the window by two binary searches, the
//                      Gaussian weights by lanes, their sum by shuffles; the forward applies
//                      each chunk of weights to every spectrum, the reverse mode scatters them
//                      for a block of up to LSF_SPEC spectra.
//   rotation kernels:  one thread per output wavelength (forward) or point (reverse, a gather): a
//                      walk over the window's offsets, whose kernel integrals are quartics in the
//                      wavelength over a block, applied to up to 16 spectra at once; short windows, and
//                      the reverse mode on coarse grids, by their integrals one by one.
//
// Everything is FP64, as in the reference (post-processing of the FP64 flux).
#pragma once
#include "physics.cuh"

namespace korg {

constexpr int LSF_SPEC = 8;   // spectra per warp pass
constexpr int ROT_TP = 64;    // outputs (forward) or points (reverse) per block
constexpr int ROT_MAX_RANGES = 64;

struct LsfArgs {
    const double* wls;    // synthesis grid (cm), sorted
    int64_t nwl;
    const double* owl;    // output wavelengths (cm)
    int64_t nout;
    const double* R;      // resolving power: R[0] for all outputs, or R[i] per output
    int32_t R_per_point;
    double window;        // window half-width in units of sigma
    double fwhm_to_sigma; // 2 sqrt(2 ln 2), as the reference computes it
};

// _lsf_bounds_and_kernel (src/utils.jl:45-58): sigma = wl0 / R / (2 sqrt(2 ln 2)); window
// [searchsortedfirst(wl0 - w sigma), searchsortedlast(wl0 + w sigma)].
__device__ __forceinline__ void lsf_window(const LsfArgs& a, int64_t i, int64_t& lb, int64_t& ub, double& wl0,
                                           double& sigma) {
    wl0 = a.owl[i];
    sigma = wl0 / a.R[a.R_per_point ? i : 0] / a.fwhm_to_sigma;
    lb = search_first(a.wls, a.nwl, wl0 - a.window * sigma);
    ub = search_last(a.wls, a.nwl, wl0 + a.window * sigma);
}

// normal_pdf (src/utils.jl:5)
__device__ __forceinline__ double lsf_phi(double d, double sigma) {
    return exp(-0.5 * (d * d) / (sigma * sigma)) / 2.5066282746310002 / sigma;
}

// window weight sum of output i, every lane gets it
__device__ __forceinline__ double lsf_norm(const LsfArgs& a, int64_t lb, int64_t ub, double wl0, double sigma,
                                           int lane) {
    double s = 0.0;
    for (int64_t j = lb + lane; j <= ub; j += 32) s += lsf_phi(a.wls[j] - wl0, sigma);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// out[s][i] = sum_j flux[s][j] phi_j / sum phi  (apply_LSF :94-106, compute_LSF_matrix * flux).
// The window is taken in chunks of 32 LSF_CW points; each lane keeps its LSF_CW normalised
// weights of the chunk in registers and applies them to every spectrum, so the Gaussian is
// evaluated twice per window point (sum, then weights) whatever the number of spectra.
constexpr int LSF_CW = 8;
__global__ void __launch_bounds__(256) lsf_apply_kernel(LsfArgs a, const double* flux, int32_t nspec, double* out) {
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (i >= a.nout) return;  // uniform across the warp
    int64_t lb, ub;
    double wl0, sigma;
    lsf_window(a, i, lb, ub, wl0, sigma);
    const double norm = lsf_norm(a, lb, ub, wl0, sigma, lane);
    if (ub < lb) {  // empty window: an empty sum
        for (int s = lane; s < nspec; s += 32) out[int64_t(s) * a.nout + i] = 0.0;
        return;
    }
    for (int64_t c0 = lb; c0 <= ub; c0 += 32 * LSF_CW) {
        double w[LSF_CW];
#pragma unroll
        for (int k = 0; k < LSF_CW; k++) {
            const int64_t j = c0 + lane + 32 * k;
            w[k] = j <= ub ? lsf_phi(a.wls[j] - wl0, sigma) / norm : 0.0;
        }
        for (int s = 0; s < nspec; s++) {
            const double* f = flux + int64_t(s) * a.nwl;
            double v = 0.0;
#pragma unroll
            for (int k = 0; k < LSF_CW; k++) {
                const int64_t j = c0 + lane + 32 * k;
                if (j <= ub) v += f[j] * w[k];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) {
                double* dst = out + int64_t(s) * a.nout + i;
                *dst = c0 == lb ? v : *dst + v;
            }
        }
    }
}

// reverse mode: dflux[s][j] += sum_i dout[s][i] phi_ij / sum_j phi_ij
__global__ void __launch_bounds__(256) lsf_vjp_kernel(LsfArgs a, const double* dout, int32_t nspec, double* dflux) {
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int s0 = blockIdx.y * LSF_SPEC;
    if (i >= a.nout) return;
    int64_t lb, ub;
    double wl0, sigma;
    lsf_window(a, i, lb, ub, wl0, sigma);
    const double norm = lsf_norm(a, lb, ub, wl0, sigma, lane);
    const int ns = min(LSF_SPEC, nspec - s0);
    double g[LSF_SPEC];
#pragma unroll
    for (int k = 0; k < LSF_SPEC; k++) g[k] = k < ns ? dout[int64_t(s0 + k) * a.nout + i] : 0.0;
    for (int64_t j = lb + lane; j <= ub; j += 32) {
        const double w = lsf_phi(a.wls[j] - wl0, sigma) / norm;
#pragma unroll
        for (int k = 0; k < LSF_SPEC; k++)
            if (k < ns && g[k] != 0.0) atomicAdd(dflux + int64_t(s0 + k) * a.nwl + j, g[k] * w);
    }
}

// window bounds per output (0-based, inclusive; ub < lb for an empty window)
__global__ void lsf_windows_kernel(LsfArgs a, int64_t* lb_out, int64_t* ub_out) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.nout) return;
    int64_t lb, ub;
    double wl0, sigma;
    lsf_window(a, i, lb, ub, wl0, sigma);
    lb_out[i] = lb;
    ub_out[i] = ub;
}

// normalised weights of output i at vals[row_ptr[i] + (j - lb)] (compute_LSF_matrix, :150-153)
__global__ void __launch_bounds__(256) lsf_values_kernel(LsfArgs a, const int64_t* row_ptr, double* vals) {
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (i >= a.nout) return;
    int64_t lb, ub;
    double wl0, sigma;
    lsf_window(a, i, lb, ub, wl0, sigma);
    const double norm = lsf_norm(a, lb, ub, wl0, sigma, lane);
    double* v = vals + row_ptr[i];
    for (int64_t j = lb + lane; j <= ub; j += 32) v[j - lb] = lsf_phi(a.wls[j] - wl0, sigma) / norm;
}

struct RotRange {
    int64_t first, n;  // grid indices of the range
    double step;       // step(wls) of the range (cm)
};
struct RotArgs {
    const double* wls;  // grid (cm)
    int64_t nwl;
    int32_t nranges;
    RotRange r[ROT_MAX_RANGES];
    double v_over_c;    // vsini (cm/s) / c
    double c1, c2, c3;  // 2(1 - eps), pi eps / 2, pi (1 - eps / 3)
};

// _rotation_kernel_integral_kernel (src/utils.jl:233-240)
__device__ __forceinline__ double rot_kernel_integral(const RotArgs& a, double c3dl, double d, double dl) {
    if (fabs(d) == dl) return d > 0 ? 0.5 : -0.5;
    return (0.5 * a.c1 * d * sqrt(1 - (d * d) / (dl * dl)) + 0.5 * a.c1 * dl * asin(d / dl) +
            a.c2 * (d - (d * d * d) / (3 * (dl * dl)))) / c3dl;
}

// The rotation of output i (_apply_rotation_core, :204-228): detunings [-dl, (lb - i + 1/2 .. ub - i -
// 1/2) step, dl], kernel integrals K_0 .. K_m+1, new F_i = sum K_{k+1} F_{lb+k} - sum K_k F_{lb+k}: the
// weight of point m is K(m - i + 1/2) - K(m - i - 1/2), with 1/2 above the window's last point and -1/2
// below its first.  K is odd.
//
// K at half-offset h = o + 1/2 is a smooth function of the output's wavelength (through dl), which hardly
// varies over a block of outputs: per block and offset it is evaluated (asin, sqrt: ~80 FP64 operations)
// at ROT_NODE Chebyshev nodes and becomes a quartic, four FMAs per output.  With r the block's relative
// half range over 1 - |x|, x = h step / dl, the quartic is off by about r^5 / 2000 of K: below FP64
// rounding for r <= 1/400; offsets nearer to the window's edge are evaluated one by one.
constexpr int ROT_NODE = 5;
struct RotTable {
    double c[ROT_NODE];  // K(h) in powers of the normalised wavelength; c[0] is NaN where there is no series
};

// Quartics of half-offsets o + 1/2, o in [o0, o0 + n), over the wavelengths [wa, wa + 2 hw], by a block.
__device__ __forceinline__ void rot_table(const RotArgs& a, double step, double wa, double hw, int64_t o0, int n,
                                          RotTable* tab) {
    const double node[3] = {0.0, 0.5877852522924731, 0.9510565162951535};  // cos of 5, 3, 1 tenths of pi
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const double d = (double(o0 + e) + 0.5) * step, dlmin = wa * a.v_over_c;
        RotTable t;
        if (1.0 - fabs(d) / dlmin > 400.0 * hw / wa) {
            double v[ROT_NODE];  // at -u2, -u1, 0, u1, u2
#pragma unroll
            for (int m = 0; m < ROT_NODE; m++) {
                const double u = m < 2 ? -node[2 - m] : node[m - 2], dl = (wa + (hw + hw * u)) * a.v_over_c;
                v[m] = rot_kernel_integral(a, a.c3 * dl, d, dl);
            }
            double c[ROT_NODE];
#pragma unroll
            for (int k = 0; k < ROT_NODE; k++) {
                c[k] = 0.0;
#pragma unroll
                for (int m = 0; m < ROT_NODE; m++) {
                    const double u = m < 2 ? -node[2 - m] : node[m - 2], u2 = u * u;
                    const double T = k == 0 ? 1.0 : k == 1 ? u : k == 2 ? 2 * u2 - 1 : k == 3 ? (4 * u2 - 3) * u
                                                                                           : (8 * u2 - 8) * u2 + 1;
                    c[k] = fma(T, v[m], c[k]);
                }
                c[k] *= k == 0 ? 0.2 : 0.4;
            }
            t.c[0] = c[0] - c[2] + c[4];
            t.c[1] = c[1] - 3 * c[3];
            t.c[2] = 2 * c[2] - 8 * c[4];
            t.c[3] = 4 * c[3];
            t.c[4] = 8 * c[4];
        } else {
            t.c[0] = nan("");
        }
        tab[e] = t;
    }
}
// K(o + 1/2) of an output of wavelength *wl at normalised wavelength u
__device__ __forceinline__ double rot_eval(const RotArgs& a, const RotTable& t, double u, double step, int64_t o,
                                           const double* wl) {
    const double k = fma(fma(fma(fma(t.c[4], u, t.c[3]), u, t.c[2]), u, t.c[1]), u, t.c[0]);
    if ((__double2hiint(t.c[0]) & 0x7ff00000) != 0x7ff00000) return k;
    const double dl = *wl * a.v_over_c;
    return rot_kernel_integral(a, a.c3 * dl, (double(o) + 0.5) * step, dl);
}

// Windows that the quartics do not pay for walk their integrals one after the other, a thread per output,
// two binary searches and one integral per point; the reverse mode scatters with FP64 atomics.  The lines,
// by m = half the window in points and the step over the wavelength (measured: 1, 4 and 16 spectra of 301
// to 100,001 points):
//   forward   m < ROT_FWD_MIN: 2,001 points, m = 1.7: 20 us (quartics 34), m = 3.3: 34 (34), m = 5: 47 (36)
//   reverse   m < ROT_VJP_MIN: m = 5: 49 us (59), m = 10: 87 (63); or a step above ROT_VJP_STEP of the
//             wavelength, where the gather's tables, which span three blocks of outputs, have no series for
//             most offsets and each integral is taken twice: 20,001 points, m = 33: 4e-6 410 us (220),
//             m = 50: 1e-5 628 (650), m = 25: 2e-5 353 (518).
constexpr double ROT_FWD_MIN = 3.0, ROT_VJP_MIN = 10.0, ROT_VJP_STEP = 5e-6;
constexpr int ROT_SPEC = 8;   // spectra per thread of the scatter
__device__ __forceinline__ const RotRange& rot_range(const RotArgs& a, int64_t i) {  // the range of grid index i
    int k = 0;
    while (k + 1 < a.nranges && i >= a.r[k + 1].first) k++;
    return a.r[k];
}
struct RotWindow {
    const double* w;  // the range's wavelengths
    int64_t first, ii, lb, ub;  // the range, the output and its window within it
    double step, dl, c3dl;
    // integral above point m of the window
    __device__ __forceinline__ double above(const RotArgs& a, int64_t m) const {
        return rot_kernel_integral(a, c3dl, m < ub ? (double(m - ii) + 0.5) * step : dl, dl);
    }
};
__device__ __forceinline__ RotWindow rot_window(const RotArgs& a, int64_t i) {
    const RotRange& rg = rot_range(a, i);
    RotWindow q;
    q.w = a.wls + rg.first;
    q.first = rg.first;
    q.ii = i - rg.first;
    q.step = rg.step;
    const double wl = a.wls[i];
    q.dl = wl * a.v_over_c;
    q.c3dl = a.c3 * q.dl;
    q.lb = search_first(q.w, rg.n, wl - q.dl);
    q.ub = search_last(q.w, rg.n, wl + q.dl);
    return q;
}
__global__ void __launch_bounds__(128) rotation_scatter_kernel(RotArgs a, const double* dout, int32_t nspec,
                                                               double* dflux) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.nwl) return;
    const int s0 = blockIdx.y * ROT_SPEC, ns = min(ROT_SPEC, nspec - s0);
    const RotWindow q = rot_window(a, i);
    double g[ROT_SPEC];
#pragma unroll
    for (int k = 0; k < ROT_SPEC; k++) g[k] = k < ns ? dout[int64_t(s0 + k) * a.nwl + i] : 0.0;
    double Kp = rot_kernel_integral(a, q.c3dl, -q.dl, q.dl);
    for (int64_t m = q.lb; m <= q.ub; m++) {
        const double Kn = q.above(a, m);
#pragma unroll
        for (int k = 0; k < ROT_SPEC; k++)
            if (k < ns) atomicAdd(dflux + int64_t(s0 + k) * a.nwl + q.first + m, g[k] * (Kn - Kp));
        Kp = Kn;
    }
}
// Forward: a chunk's weights K_{k+1} - K_k in this thread's own column of shared memory, then every spectrum.
constexpr int ROT_DCH = 8;  // window points per chunk (m < ROT_FWD_MIN: at most 7)
__global__ void __launch_bounds__(ROT_TP) rotation_direct_kernel(RotArgs a, const double* in, int32_t nspec, double* out) {
    __shared__ double s_w[ROT_DCH][ROT_TP];
    const int t = threadIdx.x;
    const int64_t i = int64_t(blockIdx.x) * ROT_TP + t;
    if (i >= a.nwl) return;  // no block-wide synchronisation below
    const RotWindow q = rot_window(a, i);
    const int64_t nwin = q.ub - q.lb + 1;
    double Kp = rot_kernel_integral(a, q.c3dl, -q.dl, q.dl);
    for (int64_t c0 = 0; c0 < nwin; c0 += ROT_DCH) {
        const int n = int(min(int64_t(ROT_DCH), nwin - c0));
        for (int e = 0; e < n; e++) {
            const double Kn = q.above(a, q.lb + c0 + e);
            s_w[e][t] = Kn - Kp;
            Kp = Kn;
        }
        const double* f0 = in + q.first + q.lb + c0;
        for (int s = 0; s < nspec; s++) {
            const double* f = f0 + int64_t(s) * a.nwl;
            double acc = 0.0;
            for (int e = 0; e < n; e++) acc += s_w[e][t] * f[e];
            double* o = out + int64_t(s) * a.nwl + i;
            *o = c0 == 0 ? acc : *o + acc;
        }
    }
    if (nwin <= 0) {  // empty window (cannot happen for a grid point, which is inside its own window)
        for (int s = 0; s < nspec; s++) out[int64_t(s) * a.nwl + i] = 0.0;
    }
}

// first block of each range in a grid of ROT_TP-point blocks that do not straddle ranges
__device__ __forceinline__ const RotRange& rot_block(const RotArgs& a, int64_t* i0) {
    int64_t blk = blockIdx.x;
    int k = 0;
    for (; k + 1 < a.nranges; k++) {
        const int64_t nb = (a.r[k].n + ROT_TP - 1) / ROT_TP;
        if (blk < nb) break;
        blk -= nb;
    }
    *i0 = blk * ROT_TP;
    return a.r[k];
}

// Forward of long windows: one thread per output and up to NS spectra (accumulators in registers), offsets +o and -o
// together.  FP64 pipe bound: 2 NS FMAs and ~8 operations of weights per offset pair.  16 spectra of
// 100,001 points, vsini 10 km/s (214 window points): 3886 -> 944 us (two asin / sqrt a point and output
// before).
constexpr int ROT_CH = 128;  // offsets per table
template <int NS>
__global__ void __launch_bounds__(ROT_TP) rotation_fwd_kernel(RotArgs a, const double* in, int32_t nspec, double* out) {
    __shared__ RotTable s_tab[ROT_CH];
    __shared__ int s_max;
    int64_t i0;
    const RotRange& rg = rot_block(a, &i0);
    const double* w = a.wls + rg.first;
    const int t = threadIdx.x, s0 = blockIdx.y * NS, ns = min(NS, nspec - s0);
    const int64_t i = min(i0 + t, rg.n - 1), il = min(i0 + ROT_TP, rg.n) - 1;  // threads past the end repeat the last
    const double wa = w[i0], hw = 0.5 * (w[il] - wa), wl = w[i], dl = wl * a.v_over_c;
    const double u = hw > 0 ? ((wl - wa) - hw) / hw : 0.0;
    const int64_t lb = search_first(w, rg.n, wl - dl), ub = search_last(w, rg.n, wl + dl);
    if (t == 0) s_max = -1;
    __syncthreads();
    if (ub >= lb) atomicMax(&s_max, int(max(ub - i, i - lb)));
    __syncthreads();
    const int omax = s_max;
    double acc[NS];
#pragma unroll
    for (int s = 0; s < NS; s++) acc[s] = 0.0;
    const double* f = in + int64_t(s0) * a.nwl + rg.first;
    double Kp = 0.0;  // K(o - 1/2)
    for (int c0 = 0; c0 <= omax; c0 += ROT_CH) {
        const int n = min(ROT_CH, omax + 1 - c0);
        __syncthreads();
        rot_table(a, rg.step, wa, hw, c0, n, s_tab);
        __syncthreads();
        for (int q = 0; q < n; q++) {
            const int64_t o = c0 + q, mp = i + o, mm = i - o;
            const bool inp = mp >= lb && mp <= ub, inm = o > 0 && mm >= lb && mm <= ub;
            if (!inp && !inm) continue;
            const double Kn = mp < ub || mm > lb ? rot_eval(a, s_tab[q], u, rg.step, o, w + i) : 0.0;
            if (inp) {
                const double below = o > 0 ? Kp : -Kn;
                const double wt = (mp < ub ? Kn : 0.5) - (mp > lb ? below : -0.5);
#pragma unroll
                for (int s = 0; s < NS; s++)
                    if (s < ns) acc[s] = fma(wt, f[s * a.nwl + mp], acc[s]);
            }
            if (inm) {
                const double wt = (mm < ub ? -Kp : 0.5) - (mm > lb ? -Kn : -0.5);
#pragma unroll
                for (int s = 0; s < NS; s++)
                    if (s < ns) acc[s] = fma(wt, f[s * a.nwl + mm], acc[s]);
            }
            Kp = Kn;
        }
    }
    if (i0 + t < rg.n) {
#pragma unroll
        for (int s = 0; s < NS; s++)
            if (s < ns) out[int64_t(s0 + s) * a.nwl + rg.first + i] = acc[s];
    }
}

// Reverse mode of long windows as a gather: dF_j += sum over the outputs i whose window holds j of dout_i w(i, j), one thread
// per point j and up to NS spectra, outputs j - o and j + o together (o uniform over the block, so the
// offsets without a series do not diverge).  The windows of the outputs at hand and their normalised
// wavelengths go to shared memory; outputs to the left and to the right have a table each where the window
// is wide, else they share one.  16 spectra as above: 6740 -> 1446 us (FP64 atomics, and two asin / sqrt per
// window point and 8 spectra before).
template <int NS>
__global__ void __launch_bounds__(ROT_TP) rotation_vjp_kernel(RotArgs a, const double* dout, int32_t nspec,
                                                              double* dflux) {
    __shared__ RotTable s_tab[2][ROT_CH + 1];
    __shared__ int s_l[2][ROT_CH + ROT_TP], s_r[2][ROT_CH + ROT_TP];  // points of the window on either side
    __shared__ double s_u[2][ROT_CH + ROT_TP];
    int64_t j0;
    const RotRange& rg = rot_block(a, &j0);
    const double* w = a.wls + rg.first;
    const int t = threadIdx.x, s0 = blockIdx.y * NS, ns = min(NS, nspec - s0);
    const int64_t jl = min(j0 + ROT_TP, rg.n) - 1, j = j0 + t;
    // the farthest outputs whose window can reach the block (the margin covers rounding)
    const double v = a.v_over_c;
    const int64_t ia = search_first(w, rg.n, w[j0] / (1.0 + v) * (1.0 - 1e-14));
    const int64_t ib = v < 1.0 ? search_last(w, rg.n, w[jl] / (1.0 - v) * (1.0 + 1e-14)) : rg.n - 1;
    const int64_t omax = max(jl - ia, ib - j0);
    const bool shared_table = omax <= 2 * ROT_CH;
    double acc[NS];
#pragma unroll
    for (int s = 0; s < NS; s++) acc[s] = 0.0;
    const double* g = dout + int64_t(s0) * a.nwl + rg.first;
    for (int64_t c0 = 0; c0 <= omax; c0 += ROT_CH) {
        const int n = int(min(int64_t(ROT_CH), omax + 1 - c0)), back = c0 > 0 ? 1 : 0;
        // outputs j0 - c0 - n + 1 .. jl - c0 (left) and j0 + c0 .. jl + c0 + n - 1 (right), clipped to the range
        const int64_t first[2] = {j0 - c0 - n + 1, j0 + c0};
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int64_t ra = min(max(shared_table ? first[0] : first[h], int64_t(0)), rg.n - 1);
            const int64_t rb = min(max((shared_table || h == 1 ? jl + c0 + n - 1 : jl - c0), int64_t(0)), rg.n - 1);
            const double wa = w[ra], hw = 0.5 * (w[rb] - wa);
            if (h == 0 || !shared_table) rot_table(a, rg.step, wa, hw, c0 - back, n + back, s_tab[h]);
            for (int e = t; e < n + ROT_TP - 1; e += ROT_TP) {
                const int64_t i = first[h] + e;
                int l = -1, r = -1;
                double u = 0.0;
                if (i >= 0 && i < rg.n) {
                    const double wl = w[i], dl = wl * v;
                    l = int(i - search_first(w, rg.n, wl - dl));
                    r = int(search_last(w, rg.n, wl + dl) - i);
                    u = hw > 0 ? ((wl - wa) - hw) / hw : 0.0;
                }
                s_l[h][e] = l;
                s_r[h][e] = r;
                s_u[h][e] = u;
            }
        }
        __syncthreads();
        if (j > jl) continue;
        const RotTable* tabs[2] = {s_tab[0] + back, s_tab[shared_table ? 0 : 1] + back};
        for (int q = 0; q < n; q++) {
            const int64_t o = c0 + q;
            const int e1 = t + n - 1 - q, e2 = t + q;  // outputs j - o and j + o
            const int l1 = s_l[0][e1], r1 = s_r[0][e1], l2 = s_l[1][e2], r2 = s_r[1][e2];
            const bool in1 = l1 >= 0 && o <= r1, in2 = o > 0 && r2 >= 0 && o <= l2;
            if (!in1 && !in2) continue;
            if (in1) {  // point j lies o above output j - o
                const double* wi = w + (j - o);
                const double u = s_u[0][e1], Kn = o < r1 || o == 0 ? rot_eval(a, tabs[0][q], u, rg.step, o, wi) : 0.0;
                const double below = o > 0 ? rot_eval(a, tabs[0][q - 1], u, rg.step, o - 1, wi) : -Kn;
                const double wt = (o < r1 ? Kn : 0.5) - (o + l1 > 0 ? below : -0.5);
#pragma unroll
                for (int s = 0; s < NS; s++)
                    if (s < ns) acc[s] = fma(wt, g[s * a.nwl + (j - o)], acc[s]);
            }
            if (in2) {  // o below output j + o
                const double* wi = w + (j + o);
                const double u = s_u[1][e2], Kn = o < l2 ? rot_eval(a, tabs[1][q], u, rg.step, o, wi) : 0.0;
                const double wt = -rot_eval(a, tabs[1][q - 1], u, rg.step, o - 1, wi) - (o < l2 ? -Kn : -0.5);
#pragma unroll
                for (int s = 0; s < NS; s++)
                    if (s < ns) acc[s] = fma(wt, g[s * a.nwl + (j + o)], acc[s]);
            }
        }
    }
    if (j <= jl) {
#pragma unroll
        for (int s = 0; s < NS; s++)
            if (s < ns) dflux[int64_t(s0 + s) * a.nwl + rg.first + j] += acc[s];
    }
}

}  // namespace korg
