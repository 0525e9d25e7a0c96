// lines.cuh -- line opacity: per-(line, layer) prologue, width-tier candidate lists and the
// wavelength-tile accumulation kernels.  Restates line_absorption! (src/line_absorption.jl:33-129).
//
// Work decomposition
//   prep:  per-(line, layer) constants, the continuum-cutoff window (line_absorption.jl:86-119)
//          and, per group of K layers, the distances from the line centre beyond which every
//          layer of the group is in a closed-form wing branch of the Hjerting approximation and
//          (mixed) in its cubic regime, where the branch is a cubic in t' = cref / dl^2.
//   tiers: line indices partitioned by window half-width, each tier ordered by centre, so a
//          wavelength tile finds its candidate lines with two binary searches per tier.
//   tile:  one CTA per tile of wavelengths x one layer group (or, FP64, all groups).  Each thread
//          owns one (FP64) or two (mixed) wavelengths and the K consecutive layers of its group;
//          alpha accumulates in registers (FP64, or FP32 batch sums with Kahan compensation).
//          Lines are visited in list order (deterministic, no atomics on alpha); each chunk of
//          candidates is compacted with warp ballots, and the constants of each batch of lines
//          are copied to shared memory with cp.async, double buffered.
#pragma once
#include <algorithm>
#include <cstddef>

#include "physics.cuh"

namespace korg {

constexpr int STAGE_LINES = 32;  // lines staged in shared memory per batch
constexpr int MAX_GROUPS = 8;    // layer groups per CTA

// FP64 profile constants of one (line, layer): c = 2 sigma^2 (so 1/v^2 = c / x^2), w as in the
// mixed form, inv_s = 1/(sigma sqrt2), a = gamma inv_s, scale = amp inv_s / sqrt(pi)
struct alignas(16) P64 {
    double c, w, inv_s, a, scale, pad;
};

struct LinesDev {
    int64_t n;
    const double *wl, *log_gf, *E_lower, *gamma_rad, *gamma_stark, *vdW1, *vdW2, *mass;
    const int32_t *is_mol, *species;
};
struct LayersDev {
    int32_t L, S;
    const double *T, *ne, *n_eff_vdW, *xi, *n_div_U;
};
struct CntmDev {
    int64_t nk;
    const double *knots, *vals;
};

// Per-layer constants shared by all lines (line_absorption.jl:39 and the temperature scalings
// of :195 and :210), computed once per call.
struct LayerConst {
    double beta;    // 1/(k T)
    double stark6;  // (T/10^4)^(1/6)
    double vdw3;    // (T/10^4)^0.3
    // FP32 copies for the mixed-precision prologue: T, xi, n_e, n_eff_vdW, stark6, vdw3
    float T32, xi32, ne32, nv32, stark6_32, vdw3_32;
};

__device__ __forceinline__ LayerConst layer_const(const LayersDev& lay, int l) {
    double T = lay.T[l];
    LayerConst c;
    c.beta = 1 / (KBOLTZ_EV * T);
    c.stark6 = pow(T / 10000.0, 1.0 / 6.0);
    c.vdw3 = pow(T / 10000.0, 0.3);
    c.T32 = float(T);
    c.xi32 = float(lay.xi[l]);
    c.ne32 = float(lay.ne[l]);
    c.nv32 = float(lay.n_eff_vdW[l]);
    c.stark6_32 = float(c.stark6);
    c.vdw3_32 = float(c.vdw3);
    return c;
}

__global__ void layer_const_kernel(LayersDev lay, LayerConst* out) {
    int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l < lay.L) out[l] = layer_const(lay, l);
}

struct PrepOut {
    void* params;            // [n][Lp] P64 (FP64) or float4 (mixed); layers L..Lp-1 are zero padding
    int32_t* lb;             // [n]
    int32_t* ub;             // [n]
    int32_t* ci;             // [n] index of the first wavelength >= the line centre
    float* xfar;             // [n][G] |wl - wl0| beyond which every layer of group g is in a wing
                             //        branch: v >= 5 (a <= 0.2) or a + v >= 3.2 / a > 1.4 (a > 0.2)
    uint32_t* amask;         // [n] bit g: every layer of group g has a <= 0.2
    int32_t Lp, K, G;
    unsigned long long* evals;   // running totals: evaluations, lines in window
    unsigned long long* nlines;
    float4* params_w;        // [n][G][wing_quads(K)] mixed, or null: wing cubics A1 t' + A2 t'^2 + A3 t'^3 in
                             //   t' = cref / dl^2 (cref = 2 sigma^2 of layer 0), valid beyond the layer's cubic
                             //   boundary; per group three planes A1, A2, A3 of K floats (K padded to 4)
    float* xcub;             // [n][G] mixed, or null: |wl - wl0| beyond which every layer of group g
                             //   is given by its wing cubic to FP32 rounding
};

// 16-byte pieces of one (line, layer group)'s wing cubics: three planes of K floats, K padded to 4.
// Adjacent layers lie next to each other, so packed FP32 arithmetic (two FMAs an instruction) takes
// its operands straight from 16-byte loads: 12 loads and 21 FMAs a line and warp instead of 14 and 42
// (14 layers).  The tile kernel is bound by issue and the shared-memory pipe: full optical synthesis
// 37.5 -> 34.3 ms, bit for bit the same.
__host__ __device__ constexpr int wing_quads(int K) { return 3 * ((K + 3) / 4); }

// Per-line quantities shared by every layer (line_absorption.jl:83,101,105,219).
struct LineConst {
    double wl, m, El, E_upper, strength, wl2c, abo_pre, v1, v2, gstark, grad;
    bool mol;
    int sp;
};

__device__ __forceinline__ LineConst line_const(const LinesDev& ln, int64_t i) {
    LineConst q;
    q.wl = ln.wl[i];
    q.m = ln.mass[i];
    q.El = ln.E_lower[i];
    q.mol = ln.is_mol[i] != 0;
    q.v1 = ln.vdW1[i];
    q.v2 = ln.vdW2[i];
    q.gstark = ln.gamma_stark[i];
    q.grad = ln.gamma_rad[i];
    q.sp = ln.species[i];
    q.E_upper = q.El + C_CGS * HPLANCK_EV / q.wl;
    q.strength = pow(10.0, ln.log_gf[i]) * sigma_line(q.wl);
    q.wl2c = (q.wl * q.wl) / (C_CGS * (4 * PI));
    q.abo_pre = (!q.mol && q.v2 != -1) ? 2 * pow(4 / PI, q.v2 / 2) * tgamma((4 - q.v2) / 2) * 1e6 * q.v1 : 0.0;
    return q;
}

// One (line, layer) in FP64 exactly as line_absorption.jl:86-112 computes it.
struct LineLayer64 {
    double sigma, gamma, amp, dw, lw;
};

__device__ __forceinline__ LineLayer64 line_layer64(const LineConst& q, const LayersDev& lay, const LayerConst& c,
                                                    const CntmDev& cn, const KnotPos& kp, double cutoff, int l,
                                                    const MathTables& mt) {
    LineLayer64 r;
    const double T = lay.T[l];
    r.sigma = doppler_width(q.wl, T, q.m, lay.xi[l]);  // :86
    double G = q.grad;                                 // :90-94
    if (!q.mol) {
        G = G + lay.ne[l] * (q.gstark * c.stark6);
        double vdw;
        if (q.v2 == -1) {
            vdw = q.v1 * c.vdw3;
        } else {
            const double invmu = 1 / (1.008 * AMU_CGS) + 1 / q.m;
            const double vbar = sqrt(8 * KBOLTZ_CGS * T / PI * invmu);
            vdw = q.abo_pre * pow(vbar / 1e6, 1 - q.v2);
        }
        G = G + lay.n_eff_vdW[l] * vdw;
    }
    r.gamma = G * q.wl2c;                                                       // :99
    const double levels = fexp64(-c.beta * q.El, mt) - fexp64(-c.beta * q.E_upper, mt);  // :101-102
    r.amp = q.strength * levels * lay.n_div_U[int64_t(q.sp) * lay.L + l];                // :105-106
    const double acntm = knot_eval(cn.vals + int64_t(l) * cn.nk, cn.nk, kp);    // :108
    const double rho = acntm * cutoff / r.amp;
    r.dw = (rho > 1 / (SQRT_2PI * r.sigma)) ? 0.0                              // :109-112 (:140-145)
                                            : r.sigma * sqrt(-2 * flog64(SQRT_2PI * r.sigma * rho, mt));
    r.lw = inverse_lorentz_density(rho, r.gamma);
    return r;
}

__device__ __forceinline__ void store_window(const PrepOut& out, int64_t i, double lwin, double dwin, double wl,
                                             const double* wls, int64_t nwl, int L) {
    const double window = sqrt(lwin * lwin + dwin * dwin);   // :113
    const int64_t lb = search_first(wls, nwl, wl - window);  // :114-115
    const int64_t ub = search_last(wls, nwl, wl + window);
    out.lb[i] = int32_t(lb);
    out.ub[i] = int32_t(ub);
    out.ci[i] = int32_t(search_first(wls, nwl, wl));
    if (lb <= ub) {
        atomicAdd(out.evals, (unsigned long long)((ub - lb + 1) * L));
        atomicAdd(out.nlines, 1ull);
    }
}

// Per-(line, group) wing boundaries from per-layer ones held in shared memory: lanes g < G
// reduce their group and write xfar / amask.
__device__ __forceinline__ void group_bounds(const PrepOut& out, int64_t i, const float* s_bnd, const int* s_cls,
                                             int lane) {
    unsigned bits = 0;
    float mx = 0.f;
    int allA = 1;
    if (lane < out.G) {
        for (int k = 0; k < out.K; k++) {
            mx = fmaxf(mx, s_bnd[lane * out.K + k]);
            allA &= s_cls[lane * out.K + k];
        }
        out.xfar[i * out.G + lane] = mx;
    }
    bits = __ballot_sync(0xffffffffu, lane < out.G && allA);
    if (lane == 0) out.amask[i] = bits;
}

// FP64 prologue: one warp per line, lanes over layers.
__global__ void __launch_bounds__(256) line_prep64_kernel(LinesDev ln, LayersDev lay, const LayerConst* lc, CntmDev cn,
                                                          const double* wls, int64_t nwl, double cutoff, PrepOut out,
                                                          const MathTables* math) {
    __shared__ MathTables s_math;
    extern __shared__ float s_dyn[];  // [warps][Lp] boundaries, then [warps][Lp] class flags
    load_math_tables(s_math, math);
    __syncthreads();
    const int64_t i = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (i >= ln.n) return;
    const int L = lay.L, Lp = out.Lp;
    float* s_bnd = s_dyn + wib * Lp;
    int* s_cls = reinterpret_cast<int*>(s_dyn + (blockDim.x >> 5) * Lp) + wib * Lp;
    const LineConst q = line_const(ln, i);
    const KnotPos kp = knot_pos(cn.knots, cn.nk, q.wl);
    double dwin = 0.0, lwin = 0.0;
    P64* dst = reinterpret_cast<P64*>(out.params) + i * Lp;
    for (int l = lane; l < Lp; l += 32) {
        if (l >= L) {
            dst[l] = P64{1.0, 0.0, 1.0, 0.0, 0.0, 0.0};
            s_bnd[l] = 0.f;
            s_cls[l] = 1;
            continue;
        }
        const LineLayer64 r = line_layer64(q, lay, lc[l], cn, kp, cutoff, l, s_math);
        dwin = fmax(dwin, r.dw);
        lwin = fmax(lwin, r.lw);
        const double inv_s = 1 / (r.sigma * SQRT_2);  // :246-248
        const double a = r.gamma * inv_s, scale = inv_s / SQRT_PI * r.amp;
        const double c = 1 / (inv_s * inv_s);
        const bool A = a <= 0.2;
        dst[l] = P64{c, A ? a / SQRT_PI * scale : 1 / (r.gamma * r.gamma), inv_s, a, scale, 0.0};
        // v >= 5 (a <= 0.2) or a + v >= 3.2 (0.2 < a <= 1.4) or any v (a > 1.4), v = x inv_s
        s_bnd[l] = float((A ? 5.0 : (a <= 1.4 ? 3.2 - a : 0.0)) / inv_s * 1.0001);
        s_cls[l] = A;
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        dwin = fmax(dwin, __shfl_xor_sync(0xffffffffu, dwin, o));
        lwin = fmax(lwin, __shfl_xor_sync(0xffffffffu, lwin, o));
    }
    group_bounds(out, i, s_bnd, s_cls, lane);
    if (lane == 0) store_window(out, i, lwin, dwin, q.wl, wls, nwl, L);
}

// Lines at one wavelength `*wl_at` (the reference wavelength, src/synthesize.jl:265-283), in FP64: one
// warp per line, lanes over layers, every layer's contribution written to part[i][L] (0 outside the
// line's window); line_point_sum_kernel adds them up.  The tile path (prologue, candidate lists, one
// thread at work per layer group) took 62 + 124 us for 409 lines x 56 layers (80 + 1233 us for 80 layers of
// a cool giant), these two 50 + 6 (66 + 6).
__global__ void __launch_bounds__(256) line_point_kernel(LinesDev ln, LayersDev lay, CntmDev cn, const double* wl_at,
                                                         double cutoff, double* part, unsigned long long* evals,
                                                         unsigned long long* nlines, const MathTables* math) {
    __shared__ MathTables s_math;
    load_math_tables(s_math, math);
    __syncthreads();
    const int64_t i = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= ln.n) return;
    const int L = lay.L;
    const LineConst q = line_const(ln, i);
    const KnotPos kp = knot_pos(cn.knots, cn.nk, q.wl);
    const double wl = *wl_at, x = fabs(wl - q.wl);
    double dwin = 0.0, lwin = 0.0;
    double* dst = part + i * L;
    for (int l = lane; l < L; l += 32) {
        const LayerConst c = layer_const(lay, l);
        const LineLayer64 r = line_layer64(q, lay, c, cn, kp, cutoff, l, s_math);
        dwin = fmax(dwin, r.dw);
        lwin = fmax(lwin, r.lw);
        const double inv_s = 1 / (r.sigma * SQRT_2);  // :246-248
        dst[l] = voigt64(r.gamma * inv_s, x * inv_s) * (inv_s / SQRT_PI * r.amp);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        dwin = fmax(dwin, __shfl_xor_sync(0xffffffffu, dwin, o));
        lwin = fmax(lwin, __shfl_xor_sync(0xffffffffu, lwin, o));
    }
    const double window = sqrt(lwin * lwin + dwin * dwin);    // :113
    if (wl >= q.wl - window && wl <= q.wl + window) {         // :114-115 on a grid of one point
        if (lane == 0) {
            atomicAdd(evals, (unsigned long long)L);
            atomicAdd(nlines, 1ull);
        }
    } else {
        for (int l = lane; l < L; l += 32) dst[l] = 0.0;
    }
}

// alpha[l] += sum over the lines of part[i][l]: one block per layer, a fixed tree (reproducible)
__global__ void __launch_bounds__(128) line_point_sum_kernel(const double* part, int64_t n, int L, double* alpha) {
    __shared__ double s_sum[128];
    const int l = blockIdx.x, t = threadIdx.x;
    double v = 0.0;
    for (int64_t i = t; i < n; i += 128) v += part[i * L + l];
    s_sum[t] = v;
    __syncthreads();
    for (int o = 64; o > 0; o >>= 1) {
        if (t < o) s_sum[t] += s_sum[t + o];
        __syncthreads();
    }
    if (t == 0) alpha[l] += s_sum[0];
}

// FP32 forms of line_absorption.jl:140-161 (used to locate the widest layers)
__device__ __forceinline__ float inverse_gaussian32(float rho, float sigma) {
    if (rho > 1.f / (2.5066282746f * sigma)) return 0.f;
    return sigma * sqrtf(-2.f * __logf(2.5066282746f * sigma * rho));
}
__device__ __forceinline__ float inverse_lorentz32(float rho, float gamma) {
    if (rho > 1.f / (3.14159265f * gamma)) return 0.f;
    return sqrtf(fmaxf(gamma / (3.14159265f * rho) - gamma * gamma, 0.f));
}

__device__ __forceinline__ void argmax_reduce(float& v, int& idx) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
}

// Distance (in units of gamma) beyond which the far-Lorentz branch of voigt_hjerting
// (line_absorption.jl:305-308) equals its cubic series in w = 1/r^2 = gamma^2/dl^2 to FP32
// rounding.  With q = 1/(sqrt2 a) and u = 1/(1 + r^2) the branch is
//   H = sqrt(2/pi) q u (1 + (3 r^2 - 1 + (15 r^4 - 30 r^2 + 2) q^2 u^2) q^2 u^2)
//     = sqrt(2/pi) [q w + (3q^3 - q) w^2 + (q - 10q^3 + 15q^5) w^3 + (-q + 21q^3 - 105q^5) w^4 + ...]
// (u = w - w^2 + w^3 - ...), so the cubic's relative error is about C4 w^3 with
// C4 = |-1 + 21 q^2 - 105 q^4|; w^3 C4 <= 2^-26 gives r >= (2^26 C4)^(1/6).  C4 is clamped at 1
// so that the next term stays negligible near its root (a ~ 2).
__device__ __forceinline__ float far_lorentz_cubic_rmin(float a) {
    const float q2 = 0.5f / (a * a);
    const float C4 = fmaxf(fabsf(fmaf(fmaf(-105.f, q2, 21.f), q2, -1.f)), 1.f);
    return powf(67108864.f * C4, 1.f / 6.f);
}

// Mixed-precision prologue.  sigma, gamma and the profile constants are FP32; the line
// strength (Boltzmann factor, 10^loggf sigma_line, n/U) is FP64 (line_absorption.jl:101-106).
// The window is the FP64 window of the reference rule: FP32 locates the layers with the widest
// Gaussian and Lorentzian windows, and those two layers are re-evaluated in FP64.
// Packed constants: {c = 1/v-scale^2 = 2 sigma^2, a, w, scale} with scale = amp/(sigma sqrt(2 pi))
// and w = a/sqrt(pi)*scale (a <= 0.2, asymptotic wing) or 1/gamma^2 (a > 0.2, far Lorentz).
//
// Each warp handles 32 lines.  The per-line FP64 work (10^loggf, the continuum knot search,
// the exact window at two layers) runs with one lane per line; the per-(line, layer) work runs
// line by line with lanes over layers.  FP64 is 1/64 of the FP32 rate here, so keeping the
// per-line FP64 work lane-parallel is what bounds this kernel.
struct LinePrep32 {
    double El, Eu, strength;   // FP64 line-strength inputs
    float wlc, k_m, wl2c, grad, gstark, v1, abo_pre, vexp, invmu, t32;
    int32_t flags, sp, ki;     // flags: 1 molecule, 2 ABO broadening; ki: continuum knot interval
};
constexpr int PREP_WARPS = 8;  // warps per block, at most

// `lpw` lines per warp (at most 32): 32 lanes of per-line FP64 work where there are lines enough, fewer
// for short lists, whose warps then spread over the SMs (one FP64 warp instruction takes 16 cycles of
// an SM's pipe however few lanes are active, and phase B walks the warp's lines one by one).
__global__ void __launch_bounds__(32 * PREP_WARPS) line_prep_mixed_kernel(LinesDev ln, LayersDev lay,
                                                                          const LayerConst* lc, CntmDev cn,
                                                                          const double* wls, int64_t nwl,
                                                                          double cutoff, PrepOut out,
                                                                          const MathTables* math, int lpw) {
    __shared__ MathTables s_math;
    __shared__ LinePrep32 s_line[PREP_WARPS][32];
    extern __shared__ float s_dyn[];  // [warps][Lp] boundaries, [warps][Lp] class flags, [warps][Lp] cubic boundaries
    load_math_tables(s_math, math);
    __syncthreads();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int64_t base = (int64_t(blockIdx.x) * nwarps + wib) * lpw;
    if (base >= ln.n) return;
    const int nl = int(min(int64_t(lpw), ln.n - base));
    const int L = lay.L, Lp = out.Lp;
    float* s_bnd = s_dyn + wib * Lp;
    int* s_cls = reinterpret_cast<int*>(s_dyn + nwarps * Lp) + wib * Lp;
    float* s_cub = s_dyn + 2 * nwarps * Lp + wib * Lp;
    // phase A: one lane per line
    KnotPos kp_mine{0, 0.0};
    if (lane < nl) {
        const int64_t i = base + lane;
        const LineConst q = line_const(ln, i);
        kp_mine = knot_pos(cn.knots, cn.nk, q.wl);
        LinePrep32 p;
        p.El = q.El;
        p.Eu = q.E_upper;
        p.strength = q.strength;
        p.wlc = float(q.wl / C_CGS);
        p.k_m = float(KBOLTZ_CGS / q.m);
        p.wl2c = float(q.wl2c);
        p.grad = float(q.grad);
        p.gstark = float(q.gstark);
        p.v1 = float(q.v1);
        p.abo_pre = float(q.abo_pre);
        p.vexp = float(1 - q.v2);
        p.invmu = float(1 / (1.008 * AMU_CGS)) + 1.f / float(q.m);
        p.t32 = float(kp_mine.t);
        p.flags = (q.mol ? 1 : 0) | ((!q.mol && q.v2 != -1) ? 2 : 0);
        p.sp = q.sp;
        p.ki = int32_t(kp_mine.i);
        s_line[wib][lane] = p;
    }
    __syncwarp();
    // phase B: line by line, lanes over layers
    int my_dl = 0, my_ll = 0;
    for (int t = 0; t < nl; t++) {
        const int64_t i = base + t;
        const LinePrep32& q = s_line[wib][t];
        const bool mol = q.flags & 1, abo = q.flags & 2;
        float dmax = -1.f, lmax = -1.f;
        int dl = 0, ll = 0;
        float4* dst = reinterpret_cast<float4*>(out.params) + i * Lp;
        const int qb = wing_quads(out.K);
        float* dstw = out.params_w ? reinterpret_cast<float*>(out.params_w + i * out.G * qb) : nullptr;
        float cref = 0.f;
        for (int l0 = 0; l0 < Lp; l0 += 32) {
            const int l = l0 + lane;
            float4 p = make_float4(1.f, 0.f, 0.f, 0.f);  // padding layers contribute nothing
            bool A = true;
            if (l < L) {
                const LayerConst c = lc[l];
                const float sigma = q.wlc * sqrtf(q.k_m * c.T32 + 0.5f * c.xi32 * c.xi32);
                float G = q.grad;
                if (!mol) {
                    float vdw;
                    if (!abo) {
                        vdw = q.v1 * c.vdw3_32;
                    } else {
                        const float vbar = sqrtf(float(8 * KBOLTZ_CGS / PI) * c.T32 * q.invmu);
                        vdw = q.abo_pre * powf(vbar * 1e-6f, q.vexp);
                    }
                    G = G + c.ne32 * (q.gstark * c.stark6_32) + c.nv32 * vdw;
                }
                const float gamma = G * q.wl2c;
                const double levels = fexp64(-c.beta * q.El, s_math) - fexp64(-c.beta * q.Eu, s_math);  // FP64
                const float amp = float(q.strength * levels * lay.n_div_U[int64_t(q.sp) * L + l]);
                const double* row = cn.vals + int64_t(l) * cn.nk;
                const float acntm = cn.nk == 1 ? float(row[0])
                                               : float(row[q.ki]) * (1.f - q.t32) + float(row[q.ki + 1]) * q.t32;
                const float rho = acntm * float(cutoff) / amp;
                const float dw = inverse_gaussian32(rho, sigma), lw = inverse_lorentz32(rho, gamma);
                if (dw > dmax) { dmax = dw; dl = l; }
                if (lw > lmax) { lmax = lw; ll = l; }
                const float s = 1.f / (sigma * 1.41421356f);
                const float a = gamma * s;
                const float scale = s * 0.56418958f * amp;  // 1/sqrt(pi)
                A = a <= 0.2f;
                p.x = 2.f * sigma * sigma;
                p.y = a;
                p.z = A ? a * 0.56418958f * scale : 1.f / (gamma * gamma);
                p.w = scale;
                // v >= 5 (a <= 0.2) or a + v >= 3.2 (0.2 < a <= 1.4) or any v (a > 1.4), v = x / sqrt(c)
                s_bnd[l] = (A ? 5.f : (a <= 1.4f ? 3.2f - a : 0.f)) * sqrtf(p.x) * 1.0001f;
                s_cls[l] = A;
                // the layer's cubic boundary: the asymptotic branch is exactly a cubic in 1/v^2; the
                // far-Lorentz branch is one beyond r_min gamma (far_lorentz_cubic_rmin)
                s_cub[l] = A ? s_bnd[l] : fmaxf(s_bnd[l], far_lorentz_cubic_rmin(a) * gamma * 1.0001f);
            } else if (l < Lp) {
                s_bnd[l] = 0.f;
                s_cls[l] = 1;
                s_cub[l] = 0.f;
            }
            if (l0 == 0) cref = __shfl_sync(0xffffffffu, p.x, 0);  // 2 sigma^2 of layer 0
            if (l < Lp) {
                dst[l] = p;
                if (dstw) {
                    // wing cubic in t' = cref / dl^2: A1 t' + A2 t'^2 + A3 t'^3.  Asymptotic branch:
                    // w u (1 + 1.5 u + 3.75 u^2) with u = 1/v^2 = (c / cref) t'.  Far-Lorentz branch:
                    // sqrt(2/pi) scale [q w + (3q^3 - q) w^2 + (q - 10q^3 + 15q^5) w^3] with
                    // w = gamma^2 / dl^2 = (gamma^2 / cref) t' (see far_lorentz_cubic_rmin).
                    float4 pw = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (l < L) {
                        if (A) {
                            const float rr = p.x / cref;
                            pw.x = p.z * rr;
                            pw.y = 1.5f * pw.x * rr;
                            pw.z = 2.5f * pw.y * rr;
                        } else {
                            const float q = 0.70710678118654752f / p.y, q2 = q * q;
                            const float kap = (1.f / p.z) / cref;  // gamma^2 / cref
                            const float k0 = 0.7978845608028654f * p.w;
                            pw.x = k0 * q * kap;
                            pw.y = k0 * q * fmaf(3.f, q2, -1.f) * kap * kap;
                            pw.z = k0 * q * fmaf(fmaf(15.f, q2, -10.f), q2, 1.f) * kap * kap * kap;
                        }
                    }
                    const int gl = l / out.K, plane = 4 * (qb / 3);
                    float* w = dstw + gl * 4 * qb + (l - gl * out.K);
                    w[0] = pw.x;
                    w[plane] = pw.y;
                    w[2 * plane] = pw.z;
                }
            }
        }
        __syncwarp();
        argmax_reduce(dmax, dl);
        argmax_reduce(lmax, ll);
        group_bounds(out, i, s_bnd, s_cls, lane);
        if (out.xcub && lane < out.G) {
            float mx = 0.f;
            for (int k = 0; k < out.K; k++) mx = fmaxf(mx, s_cub[lane * out.K + k]);
            out.xcub[i * out.G + lane] = mx;
        }
        __syncwarp();  // s_bnd / s_cls / s_cub are rewritten by the next line
        if (lane == t) { my_dl = dl; my_ll = ll; }
    }
    // phase C: the exact FP64 window of each line at its two widest layers, one lane per line
    if (lane < nl) {
        const int64_t i = base + lane;
        const LineConst q = line_const(ln, i);
        const LineLayer64 rd = line_layer64(q, lay, lc[my_dl], cn, kp_mine, cutoff, my_dl, s_math);
        const LineLayer64 rl = line_layer64(q, lay, lc[my_ll], cn, kp_mine, cutoff, my_ll, s_math);
        store_window(out, i, rl.lw, rd.dw, q.wl, wls, nwl, L);
    }
}

// Launch geometry of the prologue kernels.  Up to about two warps per SM (of 152) the FP64 work of a short list
// is spread thin: fewer lines per warp (mixed), then fewer warps per block.  300 lines, mixed: 196 -> 55 us; lists
// of 10,000 lines and more launch as before.  In FP64 a line is a warp: up to 16 warps per SM (2,432 lines) in
// blocks of their own, which spread evenly, above in blocks of 8.  56 layers, 1,000 / 2,000 / 2,300 lines: 66 / 100
// / 109 us; blocks of 8: 70 / 110 / 110, of as many as keep two blocks per SM (3 / 6 / 7): 74 / 119 / 166.
constexpr int64_t PREP_SPREAD_WARPS = 304;
constexpr int64_t PREP64_SPREAD = 16 * 152;
inline int prep_block_warps(int64_t warps) {
    return int(std::min<int64_t>(std::max<int64_t>(warps / PREP_SPREAD_WARPS, 1), PREP_WARPS));
}
struct PrepGeom {
    int lpw, warps;  // lines per warp, warps per block
    unsigned blocks;
};
inline PrepGeom prep_geom(int64_t n, bool mixed) {
    PrepGeom g{mixed ? 4 : 1, 1, 0};
    while (mixed && g.lpw < 32 && n > g.lpw * PREP_SPREAD_WARPS) g.lpw *= 2;
    const int64_t w = (n + g.lpw - 1) / g.lpw;
    g.warps = mixed ? prep_block_warps(w) : (w <= PREP64_SPREAD ? 1 : PREP_WARPS);
    g.blocks = unsigned((w + g.warps - 1) / g.warps);
    return g;
}
// bytes of dynamic shared memory: boundaries and class flags, mixed also cubic boundaries
inline size_t prep_smem(const PrepGeom& g, int Lp, bool mixed) {
    return size_t(g.warps) * Lp * (sizeof(float) + sizeof(int) + (mixed ? sizeof(float) : 0));
}

// Candidate lists.  Lines are split by window half-width into tiers (at most 256, 4096, 65536
// wavelength points, and wider).  Within a tier the lines keep list order, so their centre
// indices are non-decreasing, and the lines that can overlap a tile [j0, j1] are the contiguous
// run with centre index in [j0 - W - 1, j1 + W + 1]: two binary searches per tier.  A single
// list with running max/min window bounds degenerates when a few lines have very wide windows
// (one synthetic line can span the whole grid); the tiers bound the over-scan per tier.
constexpr int NTIER = 4;
__device__ __constant__ int32_t c_tier_w[NTIER] = {256, 4096, 65536, 0x3fffffff};
constexpr int PART_THREADS = 256, PART_ITEMS = 8, PART_CHUNK = PART_THREADS * PART_ITEMS;

__device__ __forceinline__ int line_tier(int32_t lb, int32_t ub, int32_t ci) {
    if (lb > ub) return -1;  // empty window: never a candidate
    const int32_t h = max(ci - lb, ub - ci);
    int k = 0;
    while (k < NTIER - 1 && h > c_tier_w[k]) k++;
    return k;
}

struct TierLists {
    int32_t* idx;       // [n] line indices, tier by tier
    int32_t* ci;        // [n] their centre indices
    int32_t* start;     // [NTIER + 1] tier offsets into idx / ci
    int32_t* unsorted;  // set when centre indices decrease along the list (full scans then)
};

// per-block tier counts, and the sortedness check
__global__ void __launch_bounds__(PART_THREADS) tier_count_kernel(const int32_t* lb, const int32_t* ub,
                                                                  const int32_t* ci, int64_t n, int32_t* bcnt,
                                                                  int32_t* unsorted) {
    __shared__ int32_t s_cnt[NTIER];
    if (threadIdx.x < NTIER) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = int64_t(blockIdx.x) * PART_CHUNK;
    int c[NTIER] = {0, 0, 0, 0};
    bool bad = false;
    for (int k = threadIdx.x; k < PART_CHUNK; k += PART_THREADS) {
        const int64_t i = base + k;
        if (i >= n) break;
        const int t = line_tier(lb[i], ub[i], ci[i]);
        if (t >= 0) c[t]++;
        if (i > 0 && ci[i] < ci[i - 1]) bad = true;
    }
    for (int t = 0; t < NTIER; t++)
        if (c[t]) atomicAdd(&s_cnt[t], c[t]);
    if (bad) atomicOr(unsorted, 1);
    __syncthreads();
    if (threadIdx.x < NTIER) bcnt[blockIdx.x * NTIER + threadIdx.x] = s_cnt[threadIdx.x];
}

// stable scatter: position = tier base + lines of the tier in earlier blocks + rank in the block
__global__ void __launch_bounds__(PART_THREADS) tier_scatter_kernel(const int32_t* lb, const int32_t* ub,
                                                                    const int32_t* ci, int64_t n,
                                                                    const int32_t* bcnt, int nblocks, TierLists out) {
    __shared__ int32_t s_base[NTIER];
    __shared__ int32_t s_scan[NTIER][PART_THREADS];
    const int t0 = threadIdx.x;
    if (t0 < NTIER) {
        int32_t before = 0, total[NTIER] = {0, 0, 0, 0};
        for (int b = 0; b < nblocks; b++) {
            for (int k = 0; k < NTIER; k++) total[k] += bcnt[b * NTIER + k];
            if (b < int(blockIdx.x)) before += bcnt[b * NTIER + t0];
        }
        int32_t tb = 0;
        for (int k = 0; k < t0; k++) tb += total[k];
        s_base[t0] = tb + before;
        if (blockIdx.x == 0) {
            out.start[t0] = tb;
            if (t0 == NTIER - 1) out.start[NTIER] = tb + total[NTIER - 1];
        }
    }
    // each thread owns PART_ITEMS consecutive lines
    const int64_t i0 = int64_t(blockIdx.x) * PART_CHUNK + int64_t(t0) * PART_ITEMS;
    int tier[PART_ITEMS];
    int c[NTIER] = {0, 0, 0, 0};
    for (int k = 0; k < PART_ITEMS; k++) {
        const int64_t i = i0 + k;
        tier[k] = i < n ? line_tier(lb[i], ub[i], ci[i]) : -1;
        if (tier[k] >= 0) c[tier[k]]++;
    }
    for (int k = 0; k < NTIER; k++) s_scan[k][t0] = c[k];
    __syncthreads();
    for (int o = 1; o < PART_THREADS; o <<= 1) {  // inclusive scans of the per-thread counts
        int32_t v[NTIER];
        for (int k = 0; k < NTIER; k++) v[k] = t0 >= o ? s_scan[k][t0 - o] : 0;
        __syncthreads();
        for (int k = 0; k < NTIER; k++) s_scan[k][t0] += v[k];
        __syncthreads();
    }
    int32_t pos[NTIER];
    for (int k = 0; k < NTIER; k++) pos[k] = s_base[k] + s_scan[k][t0] - c[k];
    for (int k = 0; k < PART_ITEMS; k++) {
        if (tier[k] < 0) continue;
        const int32_t p = pos[tier[k]]++;
        out.idx[p] = int32_t(i0 + k);
        out.ci[p] = ci[i0 + k];
    }
}

// Wavelengths that a pass is limited to: those of the marked tiles (tw wavelengths each, a multiple of 32),
// or all of them where there are no marks.
struct TileMarks {
    const unsigned char* on;
    int32_t tw;
    __device__ __forceinline__ bool skip(int64_t j) const { return on && !on[j / tw]; }
};

struct TileArgs {
    double* alpha;        // [nwl][L]
    const double* wls;
    int64_t nwl;
    int32_t L, Lp, G, stage;  // layers, padded layers (G * K), layer groups, lines per batch
    int32_t split;            // 1: each CTA takes one layer group of the tile (blockIdx.y / queue)
    int32_t region;           // bytes of one shared buffer of line constants (x2, double buffered)
    int64_t n;
    const double* wl;     // line centres
    const void* params;
    const float* xfar;
    const uint32_t* amask;
    const int32_t *lb, *ub;
    const int32_t *tier_idx, *tier_ci, *tier_start, *unsorted;
    int32_t far32;            // mixed: line_far_kernel takes the far lines of dense tiles, else they are as the others
    const unsigned char* on;  // tiles to evaluate (line_tile_kernel), or null: all
    const float4* params_w;   // mixed, or null: wing cubics (see PrepOut)
    const float* xcub;        // mixed, or null: cubic boundaries (see PrepOut)
    const MathTables* math;   // FP64: tables of the table-driven exp
};

// first index in [lo, hi) with a[i] >= v (a non-decreasing)
__device__ __forceinline__ int64_t lower_bound_i32(const int32_t* a, int64_t lo, int64_t hi, int32_t v) {
    while (lo < hi) {
        int64_t mid = lo + ((hi - lo) >> 1);
        if (a[mid] < v) lo = mid + 1; else hi = mid;
    }
    return lo;
}
// first index in [lo, hi) with a[i] > v (a non-decreasing)
__device__ __forceinline__ int64_t upper_bound_i32(const int32_t* a, int64_t lo, int64_t hi, int32_t v) {
    while (lo < hi) {
        int64_t mid = lo + ((hi - lo) >> 1);
        if (a[mid] <= v) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Candidate run of width tier `t` for the tile [j0, jlast].
__device__ __forceinline__ void tier_run(const TileArgs& a, int t, int64_t j0, int64_t jlast, int64_t (&run)[2]) {
    const int64_t t0 = a.tier_start[t], t1 = a.tier_start[t + 1];
    if (*a.unsorted) {
        run[0] = t0;
        run[1] = t1;
    } else {
        const int32_t w = c_tier_w[t] + 1;
        const int32_t lo = int32_t(max(int64_t(j0) - w, int64_t(INT32_MIN / 2)));
        const int32_t hi = int32_t(min(int64_t(jlast) + w, int64_t(INT32_MAX / 2)));
        run[0] = lower_bound_i32(a.tier_ci, t0, t1, lo);
        run[1] = upper_bound_i32(a.tier_ci, t0, t1, hi);
    }
}

// A candidate line of the current chunk, as an FP64 tile sees it.
struct LineStage {
    double wl;        // centre
    int32_t lb, ub;   // window (grid indices)
    uint32_t cls;     // 2 bits per layer group: 2 = every layer in a closed-form wing branch, 3 = the same and
                      // far (evaluated at the tile's Chebyshev nodes), 0 = general
    int32_t li;       // line index
};

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_1() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

// Two FP32 values in one 64-bit register, and the packed FMA on them (each half rounds as fmaf does).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float part2(f32x2 v, int h) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    return h ? hi : lo;
}
__device__ __forceinline__ void set2(f32x2& v, int h, float x) {
    v = h ? pack2(part2(v, 0), x) : pack2(x, part2(v, 1));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// Far-Lorentz branch of voigt_hjerting (line_absorption.jl:305-308) with r^2 = x^2/gamma^2.
__device__ __forceinline__ float far_lorentz32(float4 p, float x2) {
    const float r2 = x2 * p.z;
    const float au = __fdividef(0.70710678118654752f, (r2 + 1.f) * p.y);
    const float au2 = au * au;
    return 0.7978845608028654f * au * (1.f + (3.f * r2 - 1.f + ((r2 - 2.f) * 15.f * r2 + 2.f) * au2) * au2) * p.w;
}
__device__ __forceinline__ double far_lorentz64(const P64& p, double x2) {
    const double r2 = __dmul_rn(x2, p.w);
    const double au = __dmul_rn(1 / SQRT_2, recip64(__dmul_rn(__dadd_rn(r2, 1.0), p.a)));
    const double au2 = __dmul_rn(au, au);
    const double c = fma(fma(__dmul_rn(__dadd_rn(r2, -2.0), 15.0), r2, 2.0), au2, fma(3.0, r2, -1.0));
    return __dmul_rn(__dmul_rn(__dmul_rn(0.7978845608028654, au), fma(c, au2, 1.0)), p.scale);
}

// Far lines of a tile.  A line whose window covers the whole tile and whose centre lies at least
// FAR_KAPPA tile widths outside it (and beyond its wing boundary) is a smooth function of
// wavelength there: it is evaluated at the tile's FAR_P Chebyshev nodes only, and the sum over all
// far lines is interpolated to the tile's wavelengths once, as a Chebyshev series of degree
// FAR_P - 1.  The profiles' singularities are at the line centre (asymptotic and far-Lorentz series)
// or beyond it (far-Lorentz: at wl0 +- i gamma), so with z = 2 kappa + 1 the series converges like
// (z + sqrt(z^2 - 1))^-FAR_P.  Measured on 1/x^2 at the closest distance, 16 nodes, largest relative
// error over the tile: kappa 0.75: 7e-10 (mixed; below the 6e-8 rounding of each FP32 evaluation),
// kappa 2.5: at the rounding of FP64 (4e-15 in a plain FP64 evaluation of the series; kappa 2: 8e-15).
// 16 nodes and not fewer: fewer would push kappa, and with it the lines evaluated at every wavelength, up.
// Measured, FP64 (the nodes do an eighth of the far evaluations of a kernel bound by the FP64 pipe): the
// 11 x 51 x 10,001 CO cross-section table 168.6 -> 86.4 ms, line_absorption! of 2,000 lines on 10,001
// points x 56 layers 6.3 -> 4.8 ms, same error against 64 bits.
constexpr int FAR_P = 16;
constexpr float FAR_KAPPA32 = 0.75f;
constexpr double FAR_KAPPA64 = 2.5;
constexpr int FAR_MIN_POINTS = 64;  // shorter tiles: 16 nodes would save less than 3 of 4 evaluations
// Mixed tiles with fewer candidates evaluate every line at every wavelength: there a few lines carry
// the far opacity, and the FP32 rounding of their evaluations (1e-7 each, averaged differently at the
// nodes) would move the flux by up to 6e-9 of itself (above the limit by 2e-9 at single wavelengths and
// 2e-11 in the norm, measured on a cool giant), for a gain of a tenth (full optical synthesis, 4,000
// candidates a tile) or none (sparser lists).
constexpr int64_t FAR_MIN_CAND32 = 8192;

// cos(pi i / 32), i = 0..16; the other angles by symmetry
__device__ __constant__ double c_cos32[17] = {
    1.0, 0.9951847266721969, 0.9807852804032304, 0.9569403357322088,
    0.9238795325112867, 0.881921264348355, 0.8314696123025452, 0.773010453362737,
    0.7071067811865476, 0.6343932841636455, 0.5555702330196023, 0.4713967368259978,
    0.38268343236508984, 0.29028467725446233, 0.19509032201612833, 0.09801714032956077,
    0.0};
__device__ __forceinline__ double cos_pi32(int i) {  // cos(pi i / 32)
    i &= 63;
    if (i > 32) i = 64 - i;
    return i <= 16 ? c_cos32[i] : -c_cos32[32 - i];
}

// Chebyshev coefficient n of a function from its values v[m * stride] at the nodes
// cos(pi (2m + 1) / 32).  A non-finite value makes the series its node value (n = 0) alone, as
// every evaluation of such a line would be non-finite.
__device__ __forceinline__ double far_coef(const double* v, int stride, int n) {
    double c = 0.0, sum = 0.0;
#pragma unroll
    for (int m = 0; m < FAR_P; m++) {
        c = fma(v[m * stride], cos_pi32(n * (2 * m + 1)), c);
        sum += v[m * stride];
    }
    if (!(fabs(sum) < INFINITY)) return n == 0 ? sum : 0.0;
    return c * (n == 0 ? 1.0 / FAR_P : 2.0 / FAR_P);
}

// FP64 tile: TW = blockDim.x / G wavelengths x all layers (or, with gsplit >= 0, x the layers of
// group gsplit), computed by one CTA.  Thread (j, g) owns wavelength j and the K consecutive
// (padded) layers g*K .. g*K+K-1, accumulated in FP64 registers.  `smem` is the dynamic shared
// memory of the launch (two line-constant buffers, then the LineStage array).  SUB > 1: gsplit
// counts SUB-ths of the groups, of K layers each (the classes remain those of the whole group).
template <int K, int SUB = 1>
__device__ __forceinline__ void line_tile_body64(const TileArgs& a, int64_t tile, int gsplit, unsigned char* smem) {
    const int L = a.L, Lp = a.Lp, G = a.G, B = a.stage;
    double* s_alpha = reinterpret_cast<double*>(smem);                          // [TW][SL+1], at the end
    LineStage* s_ln = reinterpret_cast<LineStage*>(smem + 2 * size_t(a.region));  // [blockDim]
    __shared__ int32_t s_warp[32];
    __shared__ int32_t s_count;
    const double* exp2j = a.math->exp2j;  // (read through L1: shared memory belongs to the tile shape)

    // gsplit >= 0: this CTA computes layer group gsplit only (its own candidate list, constants
    // and barriers), so groups of cheap and expensive layers do not wait for each other
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int TW = gsplit >= 0 ? nthr : nthr / G;
    const int jl = tid % TW, g = gsplit >= 0 ? gsplit / SUB : tid / TW;
    const int lfirst = gsplit * K;             // gsplit >= 0: this CTA's first layer
    if (SUB > 1 && lfirst >= L) return;        // nothing but padding
    const int SL = gsplit >= 0 ? K : Lp;       // layers of one staged line
    const int goff = gsplit >= 0 ? 0 : g * K;  // this thread's first layer within a staged line
    const int64_t j0 = tile * TW;
    const int64_t jg = j0 + jl;
    const int64_t jlast = min(j0 + TW, a.nwl) - 1;
    const bool live = jg < a.nwl;
    const double wl_j = live ? a.wls[jg] : 0.0;
    const double wl_ref = a.wls[j0], wl_last = a.wls[jlast];

    // candidate runs of the width tiers (threads 0..NTIER-1 search one tier each)
    __shared__ int64_t s_tier[NTIER][2];
    if (tid < NTIER) tier_run(a, tid, j0, jlast, s_tier[tid]);
    __syncthreads();

    double acc[K];
#pragma unroll
    for (int k = 0; k < K; k++) acc[k] = 0.0;
    // far lines: this thread's Chebyshev node, its line slot and the node's sums; K = 32 (more than
    // 128 layers) has no registers left for them
    constexpr bool FAR = K <= 16;
    const bool use_far = FAR && jlast - j0 + 1 >= FAR_MIN_POINTS;
    const int nslot = TW / FAR_P, fslot = jl / FAR_P;
    // node position as an offset from wl_ref: rounded to the grid's absolute precision it would be off by
    // 1e-12 of the tile
    const double hw = 0.5 * (wl_last - wl_ref), fwl = hw + hw * cos_pi32(2 * (jl % FAR_P) + 1);
    double accn[FAR ? K : 1];
#pragma unroll
    for (int k = 0; k < (FAR ? K : 1); k++) accn[k] = 0.0;

    const int warp = tid >> 5, lane = tid & 31, nwarps = nthr >> 5;
    const int chunks16 = SL * int(sizeof(P64) / 16);  // 16-byte pieces of one line's staged constants
    const int cb0 = tid / chunks16, cr0 = tid - cb0 * chunks16;       // this thread's first staged piece
    const int cdb = nthr / chunks16, cdr = nthr - cdb * chunks16;     // and the step between its pieces
    const int64_t src0 = gsplit >= 0 ? int64_t(lfirst) * int64_t(sizeof(P64) / 16) : 0;
    for (int tier = 0; tier < NTIER; tier++)
    for (int64_t base = s_tier[tier][0]; base < s_tier[tier][1]; base += nthr) {
        const int64_t pidx = base + tid;
        int64_t i = 0;
        bool take = false;
        int32_t lbi = 0, ubi = -1;
        if (pidx < s_tier[tier][1]) {
            i = a.tier_idx[pidx];
            lbi = a.lb[i];
            ubi = a.ub[i];
            take = lbi <= jlast && ubi >= j0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, take);
        if (lane == 0) s_warp[warp] = __popc(m);
        __syncthreads();
        if (tid == 0) {
            int run = 0;
            for (int w = 0; w < nwarps; w++) { int c = s_warp[w]; s_warp[w] = run; run += c; }
            s_count = run;
        }
        __syncthreads();
        if (take) {  // the thread that found the line describes it for the whole CTA
            LineStage st;
            const double wl0 = a.wl[i];
            const double dist = wl0 < wl_ref ? wl_ref - wl0 : (wl0 > wl_last ? wl0 - wl_last : 0.0);
            uint32_t cls = 0;
            const int g_lo = gsplit >= 0 ? g : 0, g_hi = gsplit >= 0 ? g + 1 : G;
            const uint32_t wing = use_far && lbi <= j0 && ubi >= jlast && dist >= FAR_KAPPA64 * (wl_last - wl_ref) ? 3u
                                                                                                                  : 2u;
            for (int gg = g_lo; gg < g_hi; gg++)
                if (dist > double(a.xfar[i * G + gg])) cls |= wing << (2 * gg);
            st.wl = wl0;
            st.lb = lbi;
            st.ub = ubi;
            st.cls = cls;
            st.li = int32_t(i);
            s_ln[s_warp[warp] + __popc(m & ((1u << lane) - 1))] = st;
        }
        const int cnt = s_count;
        __syncthreads();

        // batches of B lines: constants copied with cp.async into two alternating buffers
        const int nq = (cnt + B - 1) / B;
        auto issue = [&](int q) {
            if (q < nq) {
                const int b0 = q * B, nb = min(B, cnt - b0);
                unsigned char* buf = smem + size_t(q & 1) * a.region;
                // piece e = tid + k nthr of the batch is (line b, chunk r) = divmod(e, chunks16),
                // stepped without a division
                int b = cb0, r = cr0;
                for (int e = tid; e < nb * chunks16; e += nthr) {
                    const int64_t li = s_ln[b0 + b].li;
                    cp_async16(buf + (size_t(b) * chunks16 + r) * 16,
                               reinterpret_cast<const unsigned char*>(a.params) +
                                   (li * Lp * int64_t(sizeof(P64) / 16) + src0 + r) * 16);
                    b += cdb;
                    r += cdr;
                    if (r >= chunks16) {
                        r -= chunks16;
                        b++;
                    }
                }
            }
            cp_async_commit();
        };
        issue(0);
        for (int q = 0; q < nq; q++) {
            issue(q + 1);
            cp_async_wait_1();  // batch q has landed (this thread's copies) ...
            __syncthreads();    // ... and everybody else's
            const int b0 = q * B, nb = min(B, cnt - b0);
            const P64* s_par = reinterpret_cast<const P64*>(smem + size_t(q & 1) * a.region);
            // closed-form wing branches of one staged line at distance x
            auto add_wing = [&](double (&sum)[K], const P64* pr, double x) {
                const double x2 = __dmul_rn(x, x), t = recip64(x2);
#pragma unroll
                for (int k = 0; k < K; k++) {
                    if (pr[k].a <= 0.2) {
                        sum[k] = __dadd_rn(sum[k], voigt_wing64(pr[k].w, __dmul_rn(t, pr[k].c)));
                    } else {
                        sum[k] = __dadd_rn(sum[k], far_lorentz64(pr[k], x2));
                    }
                }
            };
            if (live) {
                for (int b = 0; b < nb; b++) {
                    const LineStage& st = s_ln[b0 + b];
                    const uint32_t cls = (st.cls >> (2 * g)) & 3u;
                    if (cls == 3u || jg < st.lb || jg > st.ub) continue;
                    const double x = fabs(wl_j - st.wl);
                    const P64* pr = s_par + b * SL + goff;
                    if (cls) {
                        add_wing(acc, pr, x);
                    } else {
#pragma unroll
                        for (int k = 0; k < K; k++)
                            acc[k] = fma(voigt64t(pr[k].a, __dmul_rn(x, pr[k].inv_s), exp2j), pr[k].scale, acc[k]);
                    }
                }
            }
            if constexpr (FAR) {
                if (use_far) {
                    // a line's slot follows from its index alone, so the sums do not depend on how
                    // the candidates fall into chunks and batches
                    auto next = [&](int b) {
                        while (b < nb && (((s_ln[b0 + b].cls >> (2 * g)) & 3u) != 3u || s_ln[b0 + b].li % nslot != fslot))
                            b++;
                        return b;
                    };
                    for (int b = next(0); b < nb; b = next(b + 1))
                        add_wing(accn, s_par + b * SL + goff, fabs((wl_ref - s_ln[b0 + b].wl) + fwl));
                }
            }
            __syncthreads();  // buffer (q & 1) is refilled by issue(q + 2)
        }
    }
    if constexpr (FAR) {
        if (use_far) {
            // node sums of the line slots -> Chebyshev coefficients -> this thread's wavelength
            double* s_node = s_alpha;  // [SL][TW], then per layer FAR_P node values and FAR_P coefficients
            __syncthreads();
#pragma unroll
            for (int k = 0; k < K; k++) s_node[(goff + k) * TW + jl] = accn[k];
            __syncthreads();
            for (int e = tid; e < SL * FAR_P; e += nthr) {
                double* v = s_node + (e / FAR_P) * TW + e % FAR_P;
                double sum = v[0];
                for (int q = 1; q < nslot; q++) sum += v[q * FAR_P];
                v[0] = sum;
            }
            __syncthreads();
            for (int e = tid; e < SL * FAR_P; e += nthr)
                s_node[(e / FAR_P) * TW + FAR_P + e % FAR_P] = far_coef(s_node + (e / FAR_P) * TW, 1, e % FAR_P);
            __syncthreads();
            const double* cf = s_node + goff * TW + FAR_P;
            const double u = hw > 0 ? fmin(fmax(((wl_j - wl_ref) - hw) / hw, -1.0), 1.0) : 0.0;
            double t0 = 1.0, t1 = u, far[K];
#pragma unroll
            for (int k = 0; k < K; k++) far[k] = cf[k * TW];
            for (int n = 1; n < FAR_P; n++) {
#pragma unroll
                for (int k = 0; k < K; k++) far[k] = fma(cf[k * TW + n], t1, far[k]);
                const double t2 = fma(2 * u, t1, -t0);
                t0 = t1;
                t1 = t2;
            }
#pragma unroll
            for (int k = 0; k < K; k++) acc[k] += far[k];
            __syncthreads();  // s_alpha overlays the coefficients
        }
    }
    // alpha += accumulated lines, staged through shared memory for coalesced updates
    const int stride = SL + 1;
#pragma unroll
    for (int k = 0; k < K; k++) s_alpha[jl * stride + goff + k] = acc[k];
    __syncthreads();
    const int64_t nj = jlast - j0 + 1;
    double* dst = a.alpha + j0 * L;
    if (gsplit >= 0) {
        const int l0 = lfirst, nk = min(K, L - l0);
        for (int64_t e = tid; e < nj * nk; e += nthr) {
            const int j = int(e / nk), k = int(e - int64_t(j) * nk);
            dst[int64_t(j) * L + l0 + k] += s_alpha[j * stride + k];
        }
    } else {
        for (int64_t e = tid; e < nj * L; e += nthr) {
            const int j = int(e / L), l = int(e - int64_t(j) * L);
            dst[e] = dst[e] + s_alpha[j * stride + l];
        }
    }
}

// A candidate line of the current chunk, as a mixed tile sees it (one layer group per CTA).
struct LineStage32 {
    float dhi, dlo;   // centre - first wavelength of the tile, as an FP32 pair
    int32_t lb, ub;   // window (grid indices)
    float cref;       // 2 sigma^2 of layer 0: the wing cubics' variable is t' = cref / dl^2
    float xfar;       // |dl| beyond which every layer of the group is in a closed-form wing branch
    uint32_t cubic;   // 1: every layer of the group is in its cubic regime over the whole tile
    int32_t li;       // line index
};
static_assert(sizeof(LineStage32) == 32, "LineStage32 is two 16-byte loads");

// Whether the mixed tile's far lines go to line_far_kernel (see FAR_MIN_CAND32).  Not with an unsorted list:
// its runs are whole tiers, whose length says nothing about the tile.
__device__ __forceinline__ bool far_tile32(const TileArgs& a, const int64_t (&run)[NTIER][2], int64_t npoints) {
    if (!a.far32 || *a.unsorted || npoints < FAR_MIN_POINTS) return false;
    int64_t n = 0;
    for (int t = 0; t < NTIER; t++) n += max(run[t][1] - run[t][0], int64_t(0));
    return n >= FAR_MIN_CAND32;
}
// Whether line i covers the tile [j0, jlast] from at least kspan away, in its cubic regime for group g.
__device__ __forceinline__ bool far_line32(const TileArgs& a, int64_t i, int g, int32_t lb, int32_t ub, int64_t j0,
                                           int64_t jlast, double wl_ref, float span32, float kspan) {
    if (lb > j0 || ub < jlast) return false;
    const float dh = float(a.wl[i] - wl_ref);
    const float fdist = dh < 0.f ? -dh : (dh > span32 ? dh - span32 : 0.f);
    return fdist >= kspan && fdist > a.xcub[i * a.G + g];
}

// Far lines of a mixed tile of tw wavelengths x the K layers of group g, added to alpha.  Lanes of a
// half-warp hold layers (K = 32: of a warp), each with its wing cubic in registers, and walk the
// FAR_P nodes: a line's constants are one coalesced load, fetched a step ahead, and the nodes' t' are
// shared through shared memory, so there is neither staging nor a block barrier per chunk (the tile
// kernel spends most of its time on both when most of its lines are far).  Packed FP32 sums over at
// most FAR_FLUSH lines, then FP64 sums in shared memory; line order within each half-warp is the
// list's, so results are reproducible.  Whole passes: 80 layers, 286,000 lines, 200,001 points 27.9 ->
// 22.2 ms; 8 infrared spectra of 5,000-50,000 lines on 100,001 points 64.8 -> 48.1 ms.
constexpr int FAR_THREADS = 128, FAR_WARPS = FAR_THREADS / 32, FAR_FLUSH = 64;
template <int K>
struct FarShared {
    double node[FAR_WARPS][FAR_P][K];       // FP64 node sums of each warp
    double v[K][FAR_P], cf[K][FAR_P + 1];
    alignas(16) float tp[FAR_WARPS][2][FAR_P];  // t' of the line(s) at hand, read 16 bytes at a time
    int64_t tier[NTIER][2];
    double stage[32][K + 1];                // alpha of 32 wavelengths
};
template <int K>
__device__ __forceinline__ void line_far_body(const TileArgs& a, int64_t tile, int tw, int g, FarShared<K>& sh) {
    static_assert(alignof(FarShared<K>) % 16 == 0 && offsetof(FarShared<K>, tp) % 16 == 0 && FAR_P % 4 == 0,
                  "tp is read in 16-byte loads");
    constexpr int LPW = K <= 16 ? 2 : 1;    // lines a warp works on at a time
    constexpr int HL = 32 / LPW;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, half = lane / HL, k = lane % HL;
    const int64_t j0 = tile * tw, jlast = min(j0 + tw, a.nwl) - 1;
    const double wl_ref = a.wls[j0], span = a.wls[jlast] - wl_ref;
    const float span32 = float(span);
    if (tid < NTIER) tier_run(a, tid, j0, jlast, sh.tier[tid]);
    __syncthreads();
    if (!far_tile32(a, sh.tier, jlast - j0 + 1)) return;  // uniform
    const float kspan = FAR_KAPPA32 * span32;
    for (int e = tid; e < FAR_WARPS * FAR_P * K; e += FAR_THREADS) (&sh.node[0][0][0])[e] = 0.0;
    __syncthreads();
    const double hw = 0.5 * span, dn = hw + hw * cos_pi32(2 * (lane % FAR_P) + 1);
    const float nh = float(dn), nlo = float(dn - double(nh));
    constexpr int plane = 4 * (wing_quads(K) / 3);
    const float* wing = reinterpret_cast<const float*>(a.params_w) + size_t(g) * 3 * plane + min(k, K - 1);
    f32x2 part[FAR_P / 2];
#pragma unroll
    for (int n = 0; n < FAR_P / 2; n++) part[n] = 0ull;
    int pending = 0;
    auto flush = [&]() {
#pragma unroll
        for (int n = 0; n < FAR_P; n++) {
            float v = part2(part[n / 2], n % 2);
            double d = double(v);
            if (LPW == 2) d += double(__shfl_xor_sync(0xffffffffu, v, 16));
            if (half == 0 && k < K) sh.node[warp][n][k] += d;
        }
#pragma unroll
        for (int n = 0; n < FAR_P / 2; n++) part[n] = 0ull;
        pending = 0;
    };
    for (int tier = 0; tier < NTIER; tier++)
        for (int64_t base = sh.tier[tier][0] + 32 * warp; base < sh.tier[tier][1]; base += FAR_THREADS) {
            int32_t li = 0;
            bool far = false;
            float dhi = 0.f, dlo = 0.f, cref = 0.f;
            if (base + lane < sh.tier[tier][1]) {
                li = a.tier_idx[base + lane];
                far = far_line32(a, li, g, a.lb[li], a.ub[li], j0, jlast, wl_ref, span32, kspan);
                if (far) {
                    const double d = a.wl[li] - wl_ref;
                    dhi = float(d);
                    dlo = float(d - double(dhi));
                    cref = reinterpret_cast<const float4*>(a.params)[int64_t(li) * a.Lp].x;
                }
            }
            unsigned m = __ballot_sync(0xffffffffu, far);
            // the next line of this half-warp (32: none), and its constants
            auto next = [&]() {
                int src = 32;
#pragma unroll
                for (int h = 0; h < LPW; h++) {
                    const int b = m ? __ffs(m) - 1 : 32;
                    if (h == half) src = b;
                    m &= m - 1;
                }
                return src;
            };
            auto load = [&](int src, float (&c)[3]) {
                const int32_t i = __shfl_sync(0xffffffffu, li, src & 31);
                const float* w = wing + size_t(i) * a.G * 3 * plane;
                c[0] = src < 32 ? w[0] : 0.f;
                c[1] = src < 32 ? w[plane] : 0.f;
                c[2] = src < 32 ? w[2 * plane] : 0.f;
            };
            float c[3], cn[3];
            const int n_lines = __popc(m);
            const int steps = (n_lines + LPW - 1) / LPW;
            if (pending + steps > FAR_FLUSH) flush();
            pending += steps;
            int src = next();
            load(src, c);
            for (int r = 0; r < n_lines; r += LPW) {
                const int src_n = next();
                load(src_n, cn);
                const float lh = __shfl_sync(0xffffffffu, dhi, src & 31), ll = __shfl_sync(0xffffffffu, dlo, src & 31),
                            lc = __shfl_sync(0xffffffffu, cref, src & 31);
                const float x = (nh - lh) + (nlo - ll);
                __syncwarp();
                if (src < 32) sh.tp[warp][half][lane % FAR_P] = __fdividef(lc, x * x);
                __syncwarp();
                if (src < 32) {
                    const f32x2 a1 = pack2(c[0], c[0]), a2 = pack2(c[1], c[1]), a3 = pack2(c[2], c[2]);
                    const ulonglong2* tp = reinterpret_cast<const ulonglong2*>(sh.tp[warp][half]);
#pragma unroll
                    for (int n = 0; n < FAR_P / 4; n++) {
                        const ulonglong2 t = tp[n];
                        part[2 * n] = fma2(t.x, fma2(t.x, fma2(t.x, a3, a2), a1), part[2 * n]);
                        part[2 * n + 1] = fma2(t.y, fma2(t.y, fma2(t.y, a3, a2), a1), part[2 * n + 1]);
                    }
                }
                src = src_n;
                c[0] = cn[0];
                c[1] = cn[1];
                c[2] = cn[2];
            }
        }
    flush();
    __syncthreads();
    for (int e = tid; e < K * FAR_P; e += FAR_THREADS) {
        double v = 0.0;
        for (int w = 0; w < FAR_WARPS; w++) v += sh.node[w][e % FAR_P][e / FAR_P];
        sh.v[e / FAR_P][e % FAR_P] = v;
    }
    __syncthreads();
    for (int e = tid; e < K * FAR_P; e += FAR_THREADS)
        sh.cf[e / FAR_P][e % FAR_P] = far_coef(sh.v[e / FAR_P], 1, e % FAR_P);
    __syncthreads();
    // the series at every wavelength, its first four terms in FP64 and the others, at most 2 % of the mean each
    // (term n over term 0 of a line at FAR_KAPPA32: 2 (1 + 0.9 n) 4.8^-n), in FP32.  With all but the mean in
    // FP32 the sum was rounded at 6e-8 of its variation, more coarsely than the Kahan sums of the tile kernel.
    // Each warp's lanes take 32 wavelengths in turn, for a quarter of the layers
    const int l0 = g * K, nk = min(K, a.L - l0);
    for (int64_t jb = j0; jb <= jlast; jb += 32) {
        const int64_t j = jb + lane;
        const double u = hw > 0 ? fmin(fmax(((a.wls[min(j, jlast)] - wl_ref) - hw) / hw, -1.0), 1.0) : 0.0;
        const double T2 = fma(2 * u, u, -1.0), T3 = fma(2 * u, T2, -u);
        const float u2 = float(2 * u);
        for (int q = warp; q < K; q += FAR_WARPS) {
            const double* cf = sh.cf[q];
            float t0 = float(T2), t1 = float(T3), var = 0.f;
#pragma unroll
            for (int n = 4; n < FAR_P; n++) {
                const float t2 = fmaf(u2, t1, -t0);
                t0 = t1;
                t1 = t2;
                var = fmaf(float(cf[n]), t1, var);
            }
            sh.stage[lane][q] = fma(cf[3], T3, fma(cf[2], T2, fma(cf[1], u, cf[0]))) + double(var);
        }
        __syncthreads();
        const int nj = int(min(int64_t(32), jlast - jb + 1));
        for (int e = tid; e < nj * nk; e += FAR_THREADS) {
            const int jj = e / nk, q = e - jj * nk;
            a.alpha[(jb + jj) * a.L + l0 + q] += sh.stage[jj][q];
        }
        __syncthreads();
    }
}

template <int K>
__global__ void __launch_bounds__(FAR_THREADS) line_far_kernel(TileArgs a, int tw) {
    __shared__ FarShared<K> sh;
    line_far_body<K>(a, blockIdx.x, tw, int(blockIdx.y), sh);
}

// on[t] = whether line_far_kernel takes lines of tile t (tw wavelengths), one thread per tile.
__global__ void far_tiles_kernel(TileArgs a, int tw, unsigned char* on) {
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x, j0 = t * tw;
    if (j0 >= a.nwl) return;
    const int64_t jlast = min(j0 + tw, a.nwl) - 1;
    int64_t run[NTIER][2];
    for (int k = 0; k < NTIER; k++) tier_run(a, k, j0, jlast, run[k]);
    on[t] = far_tile32(a, run, jlast - j0 + 1);
}

// Mixed-precision tile: TW = blockDim.x wavelengths x the K layers of group g.  Thread t owns
// wavelength j0 + t and all K layers.  Per staged line:
//   * lines whose layers are all in their cubic regime over the tile (most evaluations: far
//     wings) were staged as wing cubics: t' = cref / dl^2 per wavelength (zero outside the
//     window), then three FMAs per layer;
//   * other lines were staged as packed constants; each warp then checks whether its in-window
//     wavelengths are all beyond the wing boundary (one vote per line and warp) and evaluates
//     the closed-form wing branches, else the full profile.
// Accumulation: FP32 partial sums per batch of B lines, added to the accumulators with Kahan
// compensation.  Lines are visited in list order: results do not depend on the launch shape
// beyond the batch boundaries and the tile origins.  (Two wavelengths per thread, sharing each
// shared-memory load of a layer's constants, measured slower: the third accumulator set costs
// registers and occupancy than the saved loads gain.)
template <int K>
__device__ __forceinline__ void line_tile_body_mixed(const TileArgs& a, int64_t tile, int g, unsigned char* smem) {
    const int Lp = a.Lp, G = a.G, B = a.stage;
    double* s_alpha = reinterpret_cast<double*>(smem);                              // [TW][K+1], at the end
    LineStage32* s_ln = reinterpret_cast<LineStage32*>(smem + 2 * size_t(a.region));  // [blockDim]
    __shared__ int32_t s_warp[32];
    __shared__ int32_t s_count;
    __shared__ int64_t s_tier[NTIER][2];
    const int tid = threadIdx.x, nthr = blockDim.x, TW = nthr;
    const int warp = tid >> 5, lane = tid & 31, nwarps = nthr >> 5;
    const int64_t j0 = tile * TW;
    const int64_t jlast = min(j0 + TW, a.nwl) - 1;
    const double wl_ref = a.wls[j0], wl_last = a.wls[jlast];
    const float span32 = float(wl_last - wl_ref);
    // this thread's wavelength, and its offset from the tile's first one as an FP32 hi + lo pair
    // (formed in FP64), so |wl_j - wl0| is recovered in FP32 to about one rounding; a wavelength
    // past the grid end lies in no window
    const int32_t jm = int32_t(j0 + tid);
    const double dj = (j0 + tid < a.nwl ? a.wls[j0 + tid] : wl_ref) - wl_ref;
    const float xh = float(dj), xl = float(dj - double(xh));
    if (tid < NTIER) tier_run(a, tid, j0, jlast, s_tier[tid]);  // candidate runs of the width tiers
    __syncthreads();

    const float kspan = far_tile32(a, s_tier, jlast - j0 + 1) ? FAR_KAPPA32 * span32 : INFINITY;
    // accumulators of layer pairs (packed FP32 arithmetic on the wing cubics)
    constexpr int KP = K / 2, QB = wing_quads(K);
    float acc[K], comp[K];
#pragma unroll
    for (int k = 0; k < K; k++) { acc[k] = 0.f; comp[k] = 0.f; }

    const int64_t src0 = int64_t(g) * K;  // the group's first float4 within a line's Lp constants
    constexpr int PC = K;                                // 16-byte pieces of a staged line (QB <= K)
    const int cb0 = tid / PC, cr0 = tid - cb0 * PC;      // this thread's first staged (line, piece)
    const int cdb = nthr / PC, cdr = nthr - cdb * PC;    // and the step between its pieces
    for (int tier = 0; tier < NTIER; tier++)
    for (int64_t base = s_tier[tier][0]; base < s_tier[tier][1]; base += nthr) {
        const int64_t pidx = base + tid;
        int64_t i = 0;
        bool take = false;
        int32_t lbi = 0, ubi = -1;
        if (pidx < s_tier[tier][1]) {
            i = a.tier_idx[pidx];
            lbi = a.lb[i];
            ubi = a.ub[i];
            take = lbi <= jlast && ubi >= j0;
            if (take && kspan < INFINITY) take = !far_line32(a, i, g, lbi, ubi, j0, jlast, wl_ref, span32, kspan);
        }
        const unsigned msk = __ballot_sync(0xffffffffu, take);
        if (lane == 0) s_warp[warp] = __popc(msk);
        __syncthreads();
        if (tid == 0) {
            int run = 0;
            for (int w = 0; w < nwarps; w++) { int c = s_warp[w]; s_warp[w] = run; run += c; }
            s_count = run;
        }
        __syncthreads();
        if (take) {  // the thread that found the line describes it for the whole CTA
            LineStage32 st;
            const double d = a.wl[i] - wl_ref;
            const float dh = float(d);
            // distance of the centre from the tile in FP32 (the boundaries carry a 1e-4
            // relative margin, far above the rounding)
            const float fdist = dh < 0.f ? -dh : (dh > span32 ? dh - span32 : 0.f);
            st.dhi = dh;
            st.dlo = float(d - double(dh));
            st.lb = lbi;
            st.ub = ubi;
            st.cref = reinterpret_cast<const float4*>(a.params)[i * Lp].x;  // 2 sigma^2, layer 0
            st.xfar = a.xfar[i * G + g];
            st.cubic = fdist > a.xcub[i * G + g] ? 1u : 0u;
            st.li = int32_t(i);
            s_ln[s_warp[warp] + __popc(msk & ((1u << lane) - 1))] = st;
        }
        const int cnt = s_count;
        __syncthreads();

        // batches of B lines: the group's constants copied with cp.async into two alternating
        // buffers (wing cubics for cubic-regime lines, packed constants otherwise)
        const int nq = (cnt + B - 1) / B;
        auto issue = [&](int q) {
            if (q < nq) {
                const int b0 = q * B, nb = min(B, cnt - b0);
                unsigned char* buf = smem + size_t(q & 1) * a.region;
                int b = cb0, r = cr0;  // piece e = tid + k nthr is (line b, 16-byte piece r), stepped without a division
                for (int e = tid; e < nb * PC; e += nthr) {
                    const LineStage32& sl = s_ln[b0 + b];
                    if (!sl.cubic)
                        cp_async16(buf + (size_t(b) * PC + r) * 16,
                                   reinterpret_cast<const float4*>(a.params) + (int64_t(sl.li) * Lp + src0 + r));
                    else if (r < QB)
                        cp_async16(buf + (size_t(b) * PC + r) * 16, a.params_w + ((int64_t(sl.li) * G + g) * QB + r));
                    b += cdb;
                    r += cdr;
                    if (r >= PC) {
                        r -= PC;
                        b++;
                    }
                }
            }
            cp_async_commit();
        };
        issue(0);
        for (int q = 0; q < nq; q++) {
            issue(q + 1);
            cp_async_wait_1();  // batch q has landed (this thread's copies) ...
            __syncthreads();    // ... and everybody else's
            const int b0 = q * B, nb = min(B, cnt - b0);
            const float4* s_par = reinterpret_cast<const float4*>(smem + size_t(q & 1) * a.region);
            f32x2 part[KP];
#pragma unroll
            for (int k = 0; k < KP; k++) part[k] = 0ull;
            for (int b = 0; b < nb; b++) {
                const LineStage32 st = s_ln[b0 + b];
                const float4* pr = s_par + b * K;
                const bool in = jm >= st.lb && jm <= st.ub;
                const float x = fabsf((xh - st.dhi) + (xl - st.dlo));
                if (st.cubic) {
                    const float tp = in ? __fdividef(st.cref, x * x) : 0.f;
                    const f32x2 t2 = pack2(tp, tp);
                    // planes A1, A2, A3 of K layers (padded to 4): two layer pairs per 16-byte load
#pragma unroll
                    for (int q = 0; q < QB / 3; q++) {
                        const ulonglong2 a1 = reinterpret_cast<const ulonglong2*>(pr)[q],
                                         a2 = reinterpret_cast<const ulonglong2*>(pr)[QB / 3 + q],
                                         a3 = reinterpret_cast<const ulonglong2*>(pr)[2 * (QB / 3) + q];
                        part[2 * q] = fma2(t2, fma2(t2, fma2(t2, a3.x, a2.x), a1.x), part[2 * q]);
                        if (2 * q + 1 < KP) part[2 * q + 1] = fma2(t2, fma2(t2, fma2(t2, a3.y, a2.y), a1.y), part[2 * q + 1]);
                    }
                } else if (__all_sync(0xffffffffu, !in || x > st.xfar)) {
                    // every in-window wavelength of the warp in a closed-form wing branch, chosen
                    // per layer (uniform across the warp)
                    if (in) {
                        const float x2 = x * x, t = __fdividef(1.f, x2);
#pragma unroll
                        for (int k = 0; k < K; k++) {
                            const float4 p = pr[k];
                            float v = part2(part[k / 2], k % 2);
                            if (p.y <= 0.2f) {
                                const float iv = t * p.x;
                                v = fmaf(p.z * iv, fmaf(fmaf(3.75f, iv, 1.5f), iv, 1.f), v);
                            } else {
                                v += far_lorentz32(p, x2);
                            }
                            set2(part[k / 2], k % 2, v);
                        }
                    }
                } else if (in) {
                    const float t = __fdividef(1.f, x * x);
#pragma unroll
                    for (int k = 0; k < K; k++)
                        set2(part[k / 2], k % 2, part2(part[k / 2], k % 2) + profile32x(pr[k], x, t));
                }
            }
            // batch partial sums enter the accumulators with Kahan compensation
#pragma unroll
            for (int k = 0; k < K; k++) {
                const float y = part2(part[k / 2], k % 2) - comp[k];
                const float tt = acc[k] + y;
                comp[k] = (tt - acc[k]) - y;
                acc[k] = tt;
            }
            __syncthreads();  // buffer (q & 1) is refilled by issue(q + 2)
        }
    }
    // alpha += accumulated lines, staged through shared memory for coalesced updates
    const int stride = K + 1;
#pragma unroll
    for (int k = 0; k < K; k++) s_alpha[tid * stride + k] = double(acc[k]) - double(comp[k]);
    __syncthreads();
    const int64_t nj = jlast - j0 + 1;
    double* dst = a.alpha + j0 * a.L;
    const int l0 = g * K, nk = min(K, a.L - l0);
    for (int64_t e = tid; e < nj * nk; e += nthr) {
        const int j = int(e / nk), k = int(e - int64_t(j) * nk);
        dst[int64_t(j) * a.L + l0 + k] += s_alpha[j * stride + k];
    }
}

// One CTA per tile of one spectrum (per tile and layer group in the mixed form).
template <bool MIXED, int K, int MAXT, int MINB, int SUB = 1>
__global__ void __launch_bounds__(MAXT, MINB) line_tile_kernel(TileArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    if (MIXED && a.on && !a.on[blockIdx.x]) return;
    if constexpr (MIXED)
        line_tile_body_mixed<K>(a, blockIdx.x, int(blockIdx.y), smem);
    else
        line_tile_body64<K, SUB>(a, blockIdx.x, a.split ? int(blockIdx.y) : -1, smem);
}

// Work queue of (spectrum, tile) items for a batch of spectra on one wavelength grid.  Item k
// is tile k / nspec of spectrum k % nspec: the queue walks the grid once, visiting every
// spectrum's tile before moving on, so spectra with few and many lines are interleaved.
struct TileQueue {
    const TileArgs* spec;        // [nspec], device
    int32_t nspec;
    int32_t groups;              // layer groups per tile item (G when split, else 1)
    int64_t nitems;              // nspec * tiles * groups
    unsigned long long* next;    // item counter, zero before the launch
};

// Persistent form: a grid sized to the resident CTAs of the GPU takes items from the queue
// until it is empty.
template <bool MIXED, int K, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) line_tile_queue_kernel(TileQueue q) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ TileArgs s_a;
    __shared__ long long s_item;
    for (;;) {
        if (threadIdx.x == 0) {
            const long long it = (long long)atomicAdd(q.next, 1ull);
            s_item = it;
            if (it < q.nitems) s_a = q.spec[it % q.nspec];
        }
        __syncthreads();
        const long long it = s_item;
        if (it >= q.nitems) break;
        const long long r = it / q.nspec;
        if constexpr (MIXED)
            line_tile_body_mixed<K>(s_a, r / q.groups, int(r % q.groups), smem);
        else
            line_tile_body64<K>(s_a, r / q.groups, q.groups > 1 ? int(r % q.groups) : -1, smem);
        __syncthreads();  // s_a and s_item are rewritten for the next item
    }
}


// The far lines of a batch: one CTA per (spectrum, tile, group), spectra interleaved as in the queue.
template <int K>
__global__ void __launch_bounds__(FAR_THREADS) line_far_batch_kernel(const TileArgs* spec, int32_t nspec, int tw) {
    __shared__ FarShared<K> sh;
    __shared__ TileArgs s_a;
    if (threadIdx.x == 0) s_a = spec[blockIdx.x % nspec];
    __syncthreads();
    line_far_body<K>(s_a, blockIdx.x / nspec, tw, int(blockIdx.y), sh);
}

}  // namespace korg
