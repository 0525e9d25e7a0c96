// rt.cuh -- planar radiative transfer: anchored optical depth and exponential-integral flux.
// Restates RadiativeTransfer.jl:62-139 for the default planar path (tau_scheme "anchored",
// I_scheme "linear_flux_only" -> "linear_flux_only_expint", mu = [1], weights = [1]).
//
// One thread per wavelength column (a warp, lanes over layers, on grids short for their layers:
// rt_by_warp); the layer recursion (the tau prefix integral of :244-253 and the segment sum of
// :379-388) is sequential per column and entirely FP64.  E2(tau) and exp(-tau) are evaluated once per layer and shared by the two segments
// meeting there.  When a continuum interpolant is given, the continuum-only transfer of synthesize
// (src/synthesize.jl:287-291) runs once per continuum knot interval where its flux is a series in
// wavelength there, else in the same loop.
#pragma once
#include "physics.cuh"
#include "lines.cuh"

namespace korg {

struct RtArgs {
    const double* alpha;     // [nwl][L] full opacity
    const double* S;         // [nwl][L] source function, or null: Planck B(T_l, wl_j)
    const double* T;         // [L] (when S is null)
    const double* wls;       // [nwl] (when S is null or a continuum pass is requested)
    int64_t nwl;
    int32_t L;
    const double* tau_ref;   // [L]
    const double* alpha_ref; // [L]
    const MathTables* math;
    CntmDev cn;              // nk > 0: also run the continuum-only transfer into cntm
    const double* cseg;      // [nk - 1][CSEG_P] continuum flux series per knot interval (cntm_segment_kernel), or null
    double* flux;
    double* cntm;
    double unit;             // multiplies 2*pi*I (1e-8 in synthesize, src/synthesize.jl:315-318)
    int32_t planck;          // rt_kernel: its shared memory holds rows for the Planck series
};

// src/synthesize.jl:412-418 with the column factors hoisted and 1/(kT) per layer precomputed,
// exp(x) - 1 from the table-driven exp and the Newton reciprocal: for x = hc/(lambda k T) >= 0.07
// (lambda <= 2 um, T <= 1e5 K) the subtraction loses under two bits, so the result stays within a
// few ulps of pre / expm1(x), at about half the FP64 work per (layer, wavelength).
__device__ __forceinline__ double planck_t(double pre, double hc_over_wl, double inv_kT, const MathTables& mt) {
    const double x = hc_over_wl * inv_kT;
    return x < 0.05 ? pre / expm1(x) : pre * recip64(fexp64(x, mt) - 1.0);
}

// Once tau at a layer exceeds TAU_STOP, every deeper segment of that column contributes at most
// S_max E2(TAU_STOP) < S_max exp(-TAU_STOP) / TAU_STOP ~ 1e-19 S_max; S_max / F stays below
// ~1e3 for stellar atmospheres (Planck contrast between the top and the bottom), so the
// neglected part is below 1e-16 of the flux: the recursion stops there.
constexpr double TAU_STOP = 40.0;

// One pass of the column recursion; the continuum-only and full passes share the loop.  The
// segment [l-1, l] adds core(tau_l) - core(tau_{l-1}) with the slope m and intercept b of the
// linear source function in tau (RadiativeTransfer.jl:382-385); with core = b G / 2 + m H / 3
// (expint_core) and b = S_{l-1} - m tau_{l-1}:
//   I += S_{l-1} dG / 2 + m (dH / 3 - tau_{l-1} dG / 2),  m = (S_l - S_{l-1}) / dtau.
struct RtPass {
    double ib_prev, tau_prev, G_prev, H_prev, I;
    bool live;
    __device__ __forceinline__ void step(double alpha, double fac, double hdlt, double dS, double half_Sp,
                                         const MathTables& mt) {
        const double ib = alpha * fac;
        const double dtau = (ib + ib_prev) * hdlt;                 // RadiativeTransfer.jl:250-251
        const double tau = tau_prev + dtau;
        const double m = dS * recip64(dtau);                        // :382
        const double ex = fexp64(-tau, mt);
        const double e2 = expint2_ex(tau, ex, mt);
        const double G = fma(tau, e2, -ex), H = fma(tau, G, -ex);
        const double dG = G - G_prev, dH = H - H_prev;
        I = fma(half_Sp, dG, I);                                    // :383-385
        I = fma(m, fma(-0.5 * tau_prev, dG, dH * (1.0 / 3.0)), I);
        ib_prev = ib;
        tau_prev = tau;
        G_prev = G;
        H_prev = H;
        live = tau <= TAU_STOP;
    }
};

// ---- continuum-only transfer, once per knot interval
// Between two continuum knots every layer's opacity is linear in wavelength, so each optical depth is
// too, and the continuum flux is a smooth function of wavelength there, unless a layer's optical depth
// crosses an end of the piecewise E2 (expint2_64), where the flux steps.  Each interval's flux is
// evaluated at CSEG_P Chebyshev-Lobatto points, ends included; if every layer is on the same piece of
// E2 at all of them (and so, linear as they are, in between) and nothing varies by more than CSEG_VAR,
// the interval's flux is their Chebyshev series: with a variation of 2 % the next term is below
// (0.01)^8 / 8 of the flux.  Other intervals are marked by a NaN, and their wavelengths transferred
// one by one.  A grid of 0.01 A has 100 points per 1 A interval: 8 columns in the place of 100.
constexpr int CSEG_P = 8;
constexpr double CSEG_VAR = 0.02;
// cos(pi i / 7), i = 0..7
__device__ __constant__ double c_cos7[8] = {1.0, 0.9009688679024191, 0.6234898018587336, 0.22252093395631445, -0.22252093395631434, -0.6234898018587335, -0.900968867902419, -1.0};
__device__ __forceinline__ double cos_pi7(int i) {
    i %= 14;
    return c_cos7[i <= 7 ? i : 14 - i];
}

// piece of expint2_64 that holds x
__device__ __forceinline__ int expint2_piece(double x) {
    return x == 0 ? 0 : 1 + (x >= 1.1) + (x >= 2.5) + (x >= 3.5) + (x >= 4.5) + (x >= 5.5) + (x >= 6.5) + (x >= 7.5) +
                            (x >= 9);
}

struct RtLayers {  // per-layer constants in shared memory
    double *fac, *hdl, *ikT;
};
// Shared memory that a transfer launch may ask for beside the kernel's math tables: 48 KB in all, 1,792
// layers of constants.  What else a kernel keeps there has to fit too: above 597 layers the columns go
// without Planck rows, above 1,329 without continuum intervals, above 1,775 by threads and not by warps.
constexpr size_t RT_SMEM = 48 * 1024 - sizeof(MathTables);
inline size_t rt_smem(int L) { return sizeof(double) * 3 * size_t(L); }
__device__ __forceinline__ RtLayers rt_layers(const RtArgs& a, double* sh) {
    const int L = a.L;
    RtLayers y{sh, sh + L, sh + 2 * L};
    for (int l = threadIdx.x; l < L; l += blockDim.x) {
        y.fac[l] = a.tau_ref[l] / a.alpha_ref[l] * 1.0;  // RadiativeTransfer.jl:160
        y.hdl[l] = l > 0 ? 0.5 * (log(a.tau_ref[l]) - log(a.tau_ref[l - 1])) : 0.0;  // :114, :250-251
        y.ikT[l] = a.T ? 1.0 / (KBOLTZ_CGS * a.T[l]) : 0.0;
    }
    return y;
}

// expint2_ex with its seven middle pieces as rows of a table (centre, six coefficients; the same operations
// in the same order): lanes of a warp at different optical depths then share one path.
constexpr int E2_ROW = 7;
constexpr size_t E2_BYTES = (sizeof(double) * 7 * E2_ROW + 15) / 16 * 16;  // in shared memory
__device__ __constant__ double c_e2_mid[7 * E2_ROW] = {
    2, 0.037534261820486914, -0.04890051070806112, 0.033833820809153176, -0.016916910404576574, 0.007048712668573576,
    -0.0026785108140579598,
    3, 0.010641925085272673, -0.013048381094197039, 0.008297844727977323, -0.003687930990212144, 0.0013061422257001345,
    -0.0003995258572729822,
    4, 0.0031982292493385146, -0.0037793524098489054, 0.0022894548610917728, -0.0009539395254549051,
    0.00031003034577284415, -8.466213288412284e-5,
    5, 0.000996469042708825, -0.0011482955912753257, 0.0006737946999085467, -0.00026951787996341863,
    8.310134632205409e-5, -2.1202073223788938e-5,
    6, 0.0003182574636904001, -0.0003600824521626587, 0.00020656268138886323, -8.032993165122457e-5,
    2.390771775334065e-5, -5.8334831318151185e-6,
    7, 0.00010350984428214624, -0.00011548173161033826, 6.513442611103688e-5, -2.4813114708966427e-5,
    7.200234178941151e-6, -1.7027366981408086e-6,
    8, 3.413764515111217e-5, -3.76656228439249e-5, 2.096641424390699e-5, -7.862405341465122e-6, 2.2386015208338193e-6,
    -5.173353514609864e-7};
__device__ __forceinline__ double expint2_lanes(double x, double ex, const double* mid, const MathTables& t) {
    if (x >= 1.1 && x < 9) {
        const double* r = mid + E2_ROW * (expint2_piece(x) - 2);
        x -= r[0];
        return r[1] + (r[2] + (r[3] + (r[4] + (r[5] + r[6] * x) * x) * x) * x) * x;
    }
    return expint2_ex(x, ex, t);
}

// One column by one warp, lanes over layers (RtPass's recursion with a prefix sum of the optical depth):
// for grids too short to fill the GPU with one thread per column, whose serial chain of 100 dependent
// FP64 operations a layer takes 3 us a layer.  visit(l, tau) is called for every layer (valid lanes).
template <class Alpha, class Source, class Visit>
__device__ __forceinline__ double rt_column_warp(int L, const RtLayers& y, const MathTables& mt, const double* e2_mid,
                                                 Alpha alpha, Source source, Visit visit) {
    const int lane = threadIdx.x & 31;
    double I = 0.0, c_ib = 0.0, c_S = 0.0, c_tau = 0.0, c_G = -1.0, c_H = -1.0;  // the layer before the chunk
    for (int l0 = 0; l0 < L; l0 += 32) {
        const int l = l0 + lane;
        const bool in = l < L;
        const double ib = in ? alpha(l) * y.fac[l] : 0.0, S = in ? source(l) : 0.0;
        double ibp = __shfl_up_sync(0xffffffffu, ib, 1), Sp = __shfl_up_sync(0xffffffffu, S, 1);
        if (lane == 0) {
            ibp = c_ib;
            Sp = c_S;
        }
        const double dtau = in && l > 0 ? (ib + ibp) * y.hdl[l] : 0.0;  // RadiativeTransfer.jl:250-251
        double tau = dtau;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, tau, o);
            if (lane >= o) tau += v;
        }
        tau += c_tau;
        double taup = __shfl_up_sync(0xffffffffu, tau, 1);
        if (lane == 0) taup = c_tau;
        if (in) visit(l, tau);
        const double ex = fexp64(-tau, mt), e2 = expint2_lanes(tau, ex, e2_mid, mt);
        const double G = fma(tau, e2, -ex), H = fma(tau, G, -ex);
        double Gp = __shfl_up_sync(0xffffffffu, G, 1), Hp = __shfl_up_sync(0xffffffffu, H, 1);
        if (lane == 0) {
            Gp = c_G;
            Hp = c_H;
        }
        if (in && l > 0 && taup <= TAU_STOP) {
            const double m = (S - Sp) * recip64(dtau), dG = G - Gp, dH = H - Hp;  // :382-385
            I = fma(0.5 * Sp, dG, I);
            I = fma(m, fma(-0.5 * taup, dG, dH * (1.0 / 3.0)), I);
        }
        c_ib = __shfl_sync(0xffffffffu, ib, 31);
        c_S = __shfl_sync(0xffffffffu, S, 31);
        c_tau = __shfl_sync(0xffffffffu, tau, 31);
        c_G = __shfl_sync(0xffffffffu, G, 31);
        c_H = __shfl_sync(0xffffffffu, H, 31);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) I += __shfl_xor_sync(0xffffffffu, I, o);
    return I;
}

inline size_t cntm_segment_smem(int L) { return rt_smem(L) + CSEG_P * size_t(L); }  // constants, pieces of E2
// one block per interval at a time, one warp per node
__global__ void __launch_bounds__(32 * CSEG_P) cntm_segment_kernel(RtArgs a, double* cseg) {
    extern __shared__ double s_rt[];
    __shared__ MathTables s_math;
    __shared__ double s_I[CSEG_P], s_e2[7 * E2_ROW];
    load_math_tables(s_math, a.math);
    if (threadIdx.x < 7 * E2_ROW) s_e2[threadIdx.x] = c_e2_mid[threadIdx.x];
    const RtLayers y = rt_layers(a, s_rt);
    unsigned char* s_piece = reinterpret_cast<unsigned char*>(s_rt + 3 * a.L);  // [CSEG_P][L]
    __syncthreads();
    const int m = threadIdx.x >> 5;  // this warp's node
    for (int64_t k = blockIdx.x; k < a.cn.nk - 1; k += gridDim.x) {
        const double w0 = a.cn.knots[k], w1 = a.cn.knots[k + 1];
        const double t = m == 0 ? 0.0 : (m == CSEG_P - 1 ? 1.0 : 0.5 - 0.5 * cos_pi7(m));
        const double wl = w0 + t * (w1 - w0);
        const double pre = 2 * HPLANCK_CGS * (C_CGS * C_CGS) / (wl * wl * wl * wl * wl), hcw = HPLANCK_CGS * C_CGS / wl;
        int ok = 1;
        const double I = rt_column_warp(
            a.L, y, s_math, s_e2,
            [&](int l) {
                const double* v = a.cn.vals + int64_t(l) * a.cn.nk + k;
                const double v0 = v[0], v1 = v[1];
                if (!(fabs(v1 - v0) <= CSEG_VAR * fmin(v0, v1))) ok = 0;
                return v0 * (1.0 - t) + v1 * t;
            },
            [&](int l) {
                if (!((w1 - w0) * (hcw * y.ikT[l] + 5.0) <= CSEG_VAR * wl)) ok = 0;
                return planck_t(pre, hcw, y.ikT[l], s_math);
            },
            // past TAU_STOP every path is on the last piece
            [&](int l, double tau) { s_piece[m * a.L + l] = (unsigned char)(expint2_piece(fmin(tau, TAU_STOP))); });
        if ((threadIdx.x & 31) == 0) s_I[m] = I;
        __syncthreads();
        for (int e = threadIdx.x; e < (CSEG_P - 1) * a.L; e += blockDim.x)
            if (s_piece[e] != s_piece[e + a.L]) ok = 0;  // node by node against the next
        ok = __syncthreads_and(ok);
        if (threadIdx.x < CSEG_P) {
            const int n = threadIdx.x;
            double coef = 0.0;
            for (int q = 0; q < CSEG_P; q++)
                coef = fma((q == 0 || q == CSEG_P - 1 ? 0.5 : 1.0) * s_I[q], cos_pi7(n * q), coef);
            coef *= (n == 0 || n == CSEG_P - 1 ? 1.0 : 2.0) / (CSEG_P - 1);
            cseg[k * CSEG_P + n] = ok ? coef : nan("");
        }
        __syncthreads();  // s_I and s_piece are rewritten for the next interval
    }
}

// continuum flux (without 2 pi and unit) at an interval's position t from its series, or NaN
__device__ __forceinline__ double cntm_series(const double* cseg, const KnotPos& kp) {
    if (!cseg || !(kp.t >= 0.0 && kp.t <= 1.0)) return nan("");
    const double* cs = cseg + kp.i * CSEG_P;
    const double u = 1.0 - 2.0 * kp.t;  // node m of the interval lies at t = (1 - cos(pi m / 7)) / 2
    double t0 = 1.0, t1 = u, v = cs[0];
#pragma unroll
    for (int n = 1; n < CSEG_P; n++) {
        v = fma(cs[n], t1, v);
        const double t2 = fma(2 * u, t1, -t0);
        t0 = t1;
        t1 = t2;
    }
    return v;
}

// Planck function of every layer over a block's wavelengths as a Chebyshev series: PLANCK_P
// evaluations per (layer, block) and PLANCK_P - 1 FMAs per (layer, wavelength) in the place of the
// ~20 FP64 operations of planck_t.  Used where the block spans at most PLANCK_VAR of hc / (lambda kT)
// in the exponent (half range): the next term is below PLANCK_VAR^6 / (2^5 6!) = 4e-17.
constexpr int PLANCK_P = 6;
constexpr double PLANCK_VAR = 0.01;
inline size_t rt_planck_smem(int L) { return rt_smem(L) + sizeof(double) * PLANCK_P * size_t(L); }
// cos(pi i / 12), i = 0..6
__device__ __constant__ double c_cos12[7] = {1.0, 0.9659258262890683, 0.8660254037844387, 0.7071067811865476, 0.5000000000000001, 0.25881904510252074, 0.0};
__device__ __forceinline__ double cos_pi12(int i) {
    i %= 24;
    if (i > 12) i = 24 - i;
    return i <= 6 ? c_cos12[i] : -c_cos12[12 - i];
}

// One thread per column.  FP64 pipe bound (45 operations per pass, layer and wavelength); the Planck
// series and the continuum intervals take the rest of it away.  Both transfers of 700,001 columns x 56
// layers: 8.11 -> 3.86 ms, and 0.5 for the intervals.
constexpr int RT_BLK = 128;
__global__ void __launch_bounds__(RT_BLK) rt_kernel(RtArgs a) {
    extern __shared__ double s_rt[];
    __shared__ MathTables s_math;
    load_math_tables(s_math, a.math);
    const int L = a.L;
    const RtLayers y = rt_layers(a, s_rt);
    double* s_pl = s_rt + 3 * L;  // [L][PLANCK_P] Planck series
    __syncthreads();
    const int64_t j0 = int64_t(blockIdx.x) * RT_BLK, j = j0 + threadIdx.x;
    const bool two = a.cn.nk > 0;
    bool series = false;
    double T1 = 0.0;  // wavelength in [-1, 1] over the block
    if (!a.S && a.planck) {  // uniform
        const double wa = a.wls[j0], hw = 0.5 * (a.wls[min(j0 + RT_BLK, a.nwl) - 1] - wa);
        double xmax = 0.0;
        for (int l = 0; l < L; l++) xmax = fmax(xmax, y.ikT[l]);
        series = hw * (HPLANCK_CGS * C_CGS / wa * xmax + 5.0) <= PLANCK_VAR * wa;
        if (series) {
            for (int e = threadIdx.x; e < L * PLANCK_P; e += RT_BLK) {
                const int l = e / PLANCK_P, m = e - l * PLANCK_P;
                const double w = wa + (hw + hw * cos_pi12(2 * m + 1));
                s_pl[e] = planck_t(2 * HPLANCK_CGS * (C_CGS * C_CGS) / (w * w * w * w * w), HPLANCK_CGS * C_CGS / w,
                                   y.ikT[l], s_math);
            }
            __syncthreads();
            for (int l = threadIdx.x; l < L; l += RT_BLK) {
                double v[PLANCK_P], c[PLANCK_P];
#pragma unroll
                for (int m = 0; m < PLANCK_P; m++) v[m] = s_pl[l * PLANCK_P + m];
#pragma unroll
                for (int n = 0; n < PLANCK_P; n++) {
                    c[n] = 0.0;
#pragma unroll
                    for (int m = 0; m < PLANCK_P; m++) c[n] = fma(v[m], cos_pi12(n * (2 * m + 1)), c[n]);
                    c[n] *= (n == 0 ? 1.0 : 2.0) / PLANCK_P;
                }
                // to powers of the normalised wavelength: T2 = 2u^2 - 1, ..., T5 = 16u^5 - 20u^3 + 5u
                double* d = s_pl + l * PLANCK_P;
                d[0] = c[0] - c[2] + c[4];
                d[1] = c[1] - 3 * c[3] + 5 * c[5];
                d[2] = 2 * c[2] - 8 * c[4];
                d[3] = 4 * c[3] - 20 * c[5];
                d[4] = 8 * c[4];
                d[5] = 16 * c[5];
            }
            __syncthreads();
            T1 = hw > 0 && j < a.nwl ? ((a.wls[j] - wa) - hw) / hw : 0.0;
        }
    }
    if (j >= a.nwl) return;
    double pre = 0, hcw = 0;
    KnotPos kp{0, 0.0};
    bool each = two;  // this wavelength's continuum transfer runs in the layer loop
    if ((!a.S && !series) || two) {
        const double wl = a.wls[j];
        pre = 2 * HPLANCK_CGS * (C_CGS * C_CGS) / (wl * wl * wl * wl * wl);
        hcw = HPLANCK_CGS * C_CGS / wl;
        if (two) {
            kp = knot_pos(a.cn.knots, a.cn.nk, wl);
            const double v = cntm_series(a.cseg, kp);
            if (v == v) {
                a.cntm[j] = 2 * PI * (v * 1.0) * a.unit;
                each = false;
            }
        }
    }
    auto source = [&](int l) {
        if (!series) return planck_t(pre, hcw, y.ikT[l], s_math);
        const double* d = s_pl + l * PLANCK_P;
        return fma(fma(fma(fma(fma(d[5], T1, d[4]), T1, d[3]), T1, d[2]), T1, d[1]), T1, d[0]);
    };
    const double* al = a.alpha + j * L;
    const double* Sc = a.S ? a.S + j * L : nullptr;

    // layer 0: tau = 0, E2(0) = 1, exp(0) = 1, so G = -1 and H = -1
    double S_prev = Sc ? Sc[0] : source(0);
    RtPass full{al[0] * y.fac[0], 0.0, -1.0, -1.0, 0.0, true};
    RtPass cont{each ? knot_eval(a.cn.vals, a.cn.nk, kp) * y.fac[0] : 0.0, 0.0, -1.0, -1.0, 0.0, each};
    for (int l = 1; l < L && (full.live || cont.live); l++) {
        const double S = Sc ? Sc[l] : source(l);
        const double hdl = y.hdl[l], dS = S - S_prev, half_Sp = 0.5 * S_prev;
        if (full.live) full.step(al[l], y.fac[l], hdl, dS, half_Sp, s_math);
        if (cont.live)
            cont.step(knot_eval(a.cn.vals + int64_t(l) * a.cn.nk, a.cn.nk, kp), y.fac[l], hdl, dS, half_Sp, s_math);
        S_prev = S;
    }
    a.flux[j] = 2 * PI * (full.I * 1.0) * a.unit;  // :136
    if (each) a.cntm[j] = 2 * PI * (cont.I * 1.0) * a.unit;
}

// One warp per column, for short grids.  A thread per column takes its serial chain at any size up to 19,456
// columns (a block per SM): 3.05 us a layer (S given), 3.3 to 5 with the Planck function and the continuum.  Warps
// take 3.0 + 4.1 c ns a column, c = ceil(L / 32) (7.0 + 5.8 c), and 20 us.  They meet at n (c + 0.9) = 730 L (500
// to 600 L), measured at S given: 3 layers 1,001 columns, 12: 4,500, 32: 12,600, 33: 9,000, 56: 14,200, 80:
// 15,100, 128: 19,000; in a synthesis: 12 layers 3,800, 24: 6,500, 56: 9,600, 80 and 128: 10,000 to 17,000.
inline bool rt_by_warp(int64_t nwl, int L, bool source_given) {
    return nwl * (10 * ((L + 31) / 32) + 9) <= (source_given ? 7300 : 5000) * int64_t(L);
}
constexpr int RT_WARPS = 4;
__global__ void __launch_bounds__(32 * RT_WARPS) rt_warp_kernel(RtArgs a) {
    extern __shared__ double s_rt[];
    __shared__ MathTables s_math;
    __shared__ double s_e2[7 * E2_ROW];
    load_math_tables(s_math, a.math);
    if (threadIdx.x < 7 * E2_ROW) s_e2[threadIdx.x] = c_e2_mid[threadIdx.x];
    const RtLayers y = rt_layers(a, s_rt);
    __syncthreads();
    const int64_t j = int64_t(blockIdx.x) * RT_WARPS + (threadIdx.x >> 5);
    if (j >= a.nwl) return;  // uniform across the warp
    const int lane = threadIdx.x & 31, L = a.L;
    const bool two = a.cn.nk > 0;
    double pre = 0, hcw = 0;
    if (!a.S || two) {
        const double wl = a.wls[j];
        pre = 2 * HPLANCK_CGS * (C_CGS * C_CGS) / (wl * wl * wl * wl * wl);
        hcw = HPLANCK_CGS * C_CGS / wl;
    }
    const double *al = a.alpha + j * L, *Sc = a.S ? a.S + j * L : nullptr;
    auto source = [&](int l) { return Sc ? Sc[l] : planck_t(pre, hcw, y.ikT[l], s_math); };
    auto nothing = [](int, double) {};
    const double F = rt_column_warp(L, y, s_math, s_e2, [&](int l) { return al[l]; }, source, nothing);
    if (lane == 0) a.flux[j] = 2 * PI * (F * 1.0) * a.unit;  // :136
    if (!two) return;
    const KnotPos kp = knot_pos(a.cn.knots, a.cn.nk, a.wls[j]);
    double C = cntm_series(a.cseg, kp);
    if (!(C == C))
        C = rt_column_warp(
            L, y, s_math, s_e2, [&](int l) { return knot_eval(a.cn.vals + int64_t(l) * a.cn.nk, a.cn.nk, kp); }, source, nothing);
    if (lane == 0) a.cntm[j] = 2 * PI * (C * 1.0) * a.unit;
}

// alpha[j][l] = continuum interpolant of layer l at wl_j (src/synthesize.jl:226-252)
__global__ void __launch_bounds__(256) alpha_init_kernel(double* alpha, const double* wls, int64_t nwl, int32_t L,
                                                         CntmDev cn, TileMarks marks = {}) {
    __shared__ int64_t s_i[64];
    __shared__ double s_t[64], s_u[64];
    const int64_t j0 = int64_t(blockIdx.x) * 64;
    const int64_t jn = min(int64_t(64), nwl - j0);
    if (threadIdx.x < jn) {
        const KnotPos p = knot_pos(cn.knots, cn.nk, wls[j0 + threadIdx.x]);
        s_i[threadIdx.x] = p.i;
        s_t[threadIdx.x] = p.t;
        s_u[threadIdx.x] = 1.0 - p.t;
    }
    __syncthreads();
    const int64_t n = jn * L;
    for (int64_t e = threadIdx.x; e < n; e += blockDim.x) {
        const int jj = int(e / L), l = int(e % L);
        if (marks.skip(j0 + jj)) continue;
        const double* v = cn.vals + int64_t(l) * cn.nk + s_i[jj];
        alpha[j0 * L + e] = cn.nk == 1 ? v[0] : fma(v[1], s_t[jj], v[0] * s_u[jj]);  // knot_eval, two operations
    }
}

// ---------------------------------------------------------------- secondary schemes
// RadiativeTransfer.jl:77-139 and :147-371 for any atmosphere geometry and scheme: rays along
// the surface mu grid (planar or spherical), inward rays seeding the outward ones at the bottom,
// tau by the anchored or the Bezier scheme, intensity by the linear, linear-flux-only or Bezier
// formal solution, or the exponential-integral flux.  One thread per wavelength walks every ray;
// the ray geometry (path, ds/dz, layers reached) is computed once on the host.
constexpr int RTG_LMAX = 128;  // layers per ray
constexpr int RTG_RMAX = 64;   // rays (inward + outward)

struct RtGenArgs {
    const double* alpha;     // [nwl][L]
    const double* S;         // [nwl][L]
    int32_t L;
    int64_t nwl;
    int32_t nrays, n_in, n_mu;
    const int32_t* ray_n;    // [nrays] layers on the ray
    const double* ray_fac;   // [nrays][L] tau_ref/alpha_ref * ds/dz, in ray order
    const double* ray_lt;    // [nrays][L] +-log tau_ref, in ray order
    const double* ray_path;  // [nrays][L] +-s, in ray order
    const double* wmu;       // [n_mu] mu weight * mu of the outward rays
    int32_t tau_scheme;      // 0 anchored, 1 bezier
    int32_t I_scheme;        // 0 linear, 1 linear_flux_only, 2 bezier, 3 linear_flux_only_expint
    const MathTables* math;
    double* flux;            // [nwl] 2 pi sum_mu w mu I_surface
    double* Isurf;           // [n_mu][nwl] surface intensity of the outward rays, or null
};

// fritsch_butland_C (RadiativeTransfer.jl:361-371) evaluated for one interval k of n points
__device__ __forceinline__ double fb_control(const double* x, const double* y, int n, int k) {
    if (n < 3) return 0.5 * (y[0] + y[1]);  // two points: the reference has no interior slope
    auto yp = [&](int q) {  // interior slope estimate at point q + 1
        const double h0 = x[q + 1] - x[q], h1 = x[q + 2] - x[q + 1];
        const double d0 = (y[q + 1] - y[q]) / h0, d1 = (y[q + 2] - y[q + 1]) / h1;
        const double al = 1.0 / 3.0 * (1 + h1 / (h1 + h0));
        return (d0 * d1) / (al * d1 + (1 - al) * d0);
    };
    const double A = k < n - 2 ? y[k + 1] + (x[k + 1] - x[k]) * yp(k) / 2
                               : y[n - 2] - (x[n - 1] - x[n - 2]) * yp(n - 3) / 2;
    const double B = k == 0 ? y[1] + (x[1] - x[0]) * yp(0) / 2 : y[k] - (x[k + 1] - x[k]) * yp(k - 1) / 2;
    return (A + B) / 2;
}

__global__ void __launch_bounds__(128) rt_general_kernel(RtGenArgs a) {
    const int64_t j = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= a.nwl) return;
    const int L = a.L;
    double tau[RTG_LMAX], col[RTG_LMAX], Sc[RTG_LMAX], I[RTG_LMAX];
    double seed[RTG_RMAX];  // per ray: bottom intensity (linear) or start value (flux only)
    for (int r = 0; r < a.nrays; r++) seed[r] = 0.0;
    double F = 0.0;
    for (int r = 0; r < a.nrays; r++) {
        const bool inward = r < a.n_in;
        const int n = a.ray_n[r];
        double Iout = 0.0;
        const double* fac = a.ray_fac + int64_t(r) * L;
        const double* lt = a.ray_lt + int64_t(r) * L;
        const double* path = a.ray_path + int64_t(r) * L;
        if (!(n == 1 && (a.I_scheme == 2 || a.tau_scheme == 1))) {  // :150-154
            for (int k = 0; k < n; k++) {
                const int lk = inward ? n - 1 - k : k;  // reversed path for inward rays (:118-121)
                col[k] = a.alpha[j * L + lk];
                Sc[k] = a.S[j * L + lk];
            }
            if (a.tau_scheme == 0) {  // :244-253
                double prev = col[0] * fac[0];
                tau[0] = 0.0;
                for (int k = 1; k < n; k++) {
                    const double ib = col[k] * fac[k];
                    tau[k] = tau[k - 1] + 0.5 * (ib + prev) * (lt[k] - lt[k - 1]);
                    prev = ib;
                }
            } else {  // :263-273
                double amin = col[0], amax = col[0];
                for (int k = 1; k < n; k++) { amin = fmin(amin, col[k]); amax = fmax(amax, col[k]); }
                tau[0] = 1e-5;
                for (int i = 1; i < n; i++) {
                    const double C = fmin(fmax(fb_control(path, col, n, i - 1), 0.5 * amin), 2 * amax);
                    tau[i] = tau[i - 1] + (path[i - 1] - path[i]) / 3 * (col[i] + col[i - 1] + C);
                }
            }
            if (a.I_scheme == 0) {  // :286-298
                I[n - 1] = seed[r];
                for (int k = n - 2; k >= 0; k--) {
                    const double d = tau[k + 1] - tau[k];
                    const double m = (Sc[k + 1] - Sc[k]) / d;
                    I[k] = (I[k + 1] - Sc[k] - m * (d + 1)) * exp(-d) + m + Sc[k];
                }
                Iout = I[0];
                if (inward && r + a.n_in < a.nrays) seed[r + a.n_in] = I[0];  // :196-198
            } else if (a.I_scheme == 2) {  // :333-350 (the bottom value is not used)
                I[n - 1] = 0.0;
                for (int k = n - 2; k >= 0; k--) {
                    const double d = tau[k + 1] - tau[k], e = exp(-d), d2 = d * d;
                    const double al = (2 + d2 - 2 * d - 2 * e) / d2;
                    const double be = (2 - (2 + 2 * d + d2) * e) / d2;
                    const double ga = (2 * d - 4 + (2 * d + 4) * e) / d2;
                    I[k] = I[k + 1] * e + al * Sc[k] + be * Sc[k + 1] + ga * fb_control(tau, Sc, n, k);
                }
                I[0] *= exp(-tau[0]);
                Iout = I[0];
                if (inward && r + a.n_in < a.nrays) seed[r + a.n_in] = I[0];
            } else {
                double add = 0.0;
                if (a.I_scheme == 1) {  // :307-324
                    double next = exp(-tau[0]);
                    for (int i = 0; i + 1 < n; i++) {
                        double dt = tau[i + 1] - tau[i];
                        dt += (dt == 0);
                        const double m = (Sc[i + 1] - Sc[i]) / dt;
                        const double cur = next;
                        next = exp(-tau[i + 1]);
                        add += (-next * (Sc[i + 1] + m) + cur * (Sc[i] + m));
                    }
                } else {  // :379-388
                    double e2p = 1.0, exp_ = 1.0;
                    for (int i = 0; i + 1 < n; i++) {
                        const double m = (Sc[i + 1] - Sc[i]) / (tau[i + 1] - tau[i]);
                        const double b = Sc[i] - m * tau[i];
                        const double ex = exp(-tau[i + 1]);
                        const double e2 = expint2_64(tau[i + 1]);
                        add += expint_core(tau[i + 1], e2, ex, m, b) - expint_core(tau[i], e2p, exp_, m, b);
                        e2p = e2;
                        exp_ = ex;
                    }
                }
                Iout = seed[r] + add;  // += onto a seeded value (:177-180)
                if (inward && r + a.n_in < a.nrays) seed[r + a.n_in] = Iout * exp(-tau[n - 1]);
            }
        }
        if (!inward) {
            const int u = r - a.n_in;
            F += Iout * a.wmu[u];
            if (a.Isurf) a.Isurf[int64_t(u) * a.nwl + j] = Iout;
        }
    }
    a.flux[j] = 2 * PI * F;
}

// Rays with anchored optical depth and the linear formal solution (I_scheme 0) or its flux-only form (1):
// along a segment of optical depth d with source slope m = (S_deep - S_shallow) / d both give
//   outward  I += T [(S_shallow + m) - e^-d (S_deep + m)],  T = product of e^-d from the surface,
//   inward   I  = I e^-d + (S_deep - m) - e^-d (S_shallow - m)
// (they differ where d = 0: the flux-only form divides by 1), so one pass from the surface down serves an
// outward ray and the inward ray that seeds it (RadiativeTransfer.jl:196-198: the outward ray gets T times
// what the inward ray brings to the deepest layer), without arrays per thread.  Both are evaluated with
// m (1 - e^-d) apart: S + m and S' + m nearly cancel where d is small and m large, which left intensities of rays
// through a shell 1e-8 and more off; now the rounding of e^-d is all that m multiplies, and what a ray gains
// from it on the way in it loses on the way out (500 random shells: 1e-9 -> 4e-12 in the norm, planar 0.4 times).
// A ray ends where T < 1e-27: what lies below contributes less than that much of the largest source
// function, and is left out however far the other columns of the warp walk.  A layer that is not finite
// makes every ray that reaches it NaN, above that depth or below, as the sum over all layers does (but for
// an infinite opacity in the last layer of a flux-only ray, which closes it).
// A block stages 32 columns in shared memory (coalesced loads, read once, transposed); its warps share the
// rays, lanes hold columns.  FP64 pipe bound, 27 operations per (ray, layer, column): 20,001 columns, 20
// rays, 56 layers, the whole call 3.37 -> 2.04 ms (kernel 2.5 ms before: four arrays of 128 doubles per
// thread in local memory).
constexpr int RAY_WARPS = 8;
constexpr double RAY_STOP = 1e-27;
inline size_t rt_rays_smem(int L, int n_mu) { return sizeof(double) * (size_t(2 * L) * 33 + L + size_t(n_mu) * 32); }
__global__ void __launch_bounds__(32 * RAY_WARPS) rt_rays_kernel(RtGenArgs a) {
    extern __shared__ double s_ray[];
    __shared__ MathTables s_math;
    __shared__ int s_bad[32], s_inf[32];  // each column's first layer that is not a number, and infinitely opaque
    load_math_tables(s_math, a.math);
    const int L = a.L, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 32) s_bad[lane] = s_inf[lane] = L;
    __syncthreads();
    double *s_al = s_ray, *s_S = s_al + L * 33, *s_hd = s_S + L * 33, *s_I = s_hd + L;  // [L][33] x 2, [L], [n_mu][32]
    const int64_t j0 = int64_t(blockIdx.x) * 32;
    const int nj = int(min(int64_t(32), a.nwl - j0));
    for (int e = threadIdx.x; e < nj * L; e += blockDim.x) {
        const int jj = e / L, k = e - jj * L;
        const double al = a.alpha[j0 * L + e], S = a.S[j0 * L + e];
        if (isnan(al) || !isfinite(S)) atomicMin(&s_bad[jj], k);
        if (isinf(al)) atomicMin(&s_inf[jj], k);
        s_al[k * 33 + jj] = al;
        s_S[k * 33 + jj] = S;
    }
    // half the steps of log tau_ref, from a ray that holds every layer it needs: outward rays share them
    for (int k = threadIdx.x; k < L; k += blockDim.x) {
        double h = 0.0;
        for (int u = 0; u < a.n_mu; u++)
            if (k > 0 && k < a.ray_n[a.n_in + u]) {
                const double* lt = a.ray_lt + int64_t(a.n_in + u) * L;
                h = 0.5 * (lt[k] - lt[k - 1]);
                break;
            }
        s_hd[k] = h;
    }
    __syncthreads();
    const int c = min(lane, nj - 1);
    for (int u = warp; u < a.n_mu; u += RAY_WARPS) {
        const int n = a.ray_n[a.n_in + u];
        const double* fac = a.ray_fac + int64_t(a.n_in + u) * L;
        const bool inward = u < a.n_in;
        double T = 1.0, Iout = 0.0, Iin = 0.0;
        double ibp = n > 0 ? s_al[c] * fac[0] : 0.0, Sp = s_S[c];
        bool open = true;  // T >= RAY_STOP so far
        for (int k = 1; k < n; k++) {
            if (!__any_sync(0xffffffffu, open)) break;
            const double ib = s_al[k * 33 + c] * fac[k], S = s_S[k * 33 + c];
            const double d = (ib + ibp) * s_hd[k];
            const double m = (S - Sp) * recip64(a.I_scheme == 1 && d == 0 ? 1.0 : d);
            const double e = fexp64(-d, s_math), a1 = 1.0 - e;  // (exact where d < ln 2)
            const double with = fma(T, fma(m, a1, fma(-e, S, Sp)), Iout);
            Iout = open ? with : Iout;
            if (inward) Iin = fma(e, Iin, fma(-m, a1, fma(-e, Sp, S)));
            T *= e;
            open = open && T >= RAY_STOP;
            ibp = ib;
            Sp = S;
        }
        if (inward && open) Iout = fma(T, Iin, Iout);
        if (n > 1 && (s_bad[c] < n || s_inf[c] < (a.I_scheme == 1 && !inward ? n - 1 : n))) Iout = nan("");
        s_I[u * 32 + lane] = Iout;
        if (a.Isurf && lane < nj) a.Isurf[int64_t(u) * a.nwl + j0 + lane] = Iout;
    }
    __syncthreads();
    if (warp == 0 && lane < nj) {
        double F = 0.0;
        for (int u = 0; u < a.n_mu; u++) F += s_I[u * 32 + lane] * a.wmu[u];
        a.flux[j0 + lane] = 2 * PI * F;
    }
}

}  // namespace korg
