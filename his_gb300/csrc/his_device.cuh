// Device-side building blocks of the flood-engine step: constants, member and
// tile descriptors, ghost cells, MUSCL/hydrostatic reconstruction, HLLC/HLL flux,
// Kurganov-Petrova velocities and block reductions.
//
// Everything is templated on the storage/arithmetic type R (double for the plain
// method, float for the production form).  The float64 translation unit is built
// with -fmad=false, so a product and a sum are fused only where the code says so; its
// order of rounding is its own (f64_ops.cuh), not that of the reference solver's float64
// torch ops (hydrointel/solver/swe2d.py).
#pragma once
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/his_gb300.h"
#include "f64_ops.cuh"

namespace his {

enum : int { BC_CLOSED = 0, BC_TRANSMISSIVE = 1, BC_STAGE = 2, BC_DISCHARGE = 3 };
enum : int { EDGE_W = 0, EDGE_E = 1, EDGE_S = 2, EDGE_N = 3 };

// Per-tile partial sums written by the stage kernels (one slot per tile, summed in
// tile order by the finalize kernel: deterministic, and for a given decomposition
// independent of the batch).
enum : int {
    P_CLIP1 = 0, P_XIN1, P_XOUT1, P_YIN1, P_YOUT1,
    P_CLIP2, P_XIN2, P_XOUT2, P_YIN2, P_YOUT2,
    P_INFIL, P_RAINW, P_RATE, P_HSUM, P_SSUM, P_HMAX,
    NPART
};

// Rows of the coupled step's float64 volume ledger (8 x members, row-major), in the
// reference's term order with the clip of each model in its own row, so that the 2-D
// and 1-D kernels of a step, which run on two streams, never add to the same element
enum : int { LG_RAIN = 0, LG_INFIL, LG_BND2_IN, LG_BND2_OUT, LG_BND1_IN, LG_BND1_OUT, LG_CLIP2, LG_CLIP1, LEDGER_ROWS };

// Member status in the device-resident engine
enum : int { ST_RUNNING = 0, ST_DONE = 1, ST_NONFINITE = 2, ST_IMPLAUSIBLE = 3, ST_SUBSTEPS = 4 };
constexpr double MAX_PLAUSIBLE_DEPTH_2D = 10.0;   // coupling.py:39

// One member of the device-resident engine: its forcing tables and its evolving
// clock, step statistics and float64 volume accumulators, in the reference's term
// order (rain, infiltration, bnd2d_in, bnd2d_out, bnd1d_in, bnd1d_out, clip).
struct EngMember {
    double rain_t0, rain_step;
    const double* rain;          // m/s per block
    int rain_n, tide_on, tide_n, q_n;
    double tide_base, tide_shift;
    double amp[4], w[4], ph[4];
    double q_t0, q_step;
    const double* q;             // inflow hydrograph, m^3/s
    int edge_src[4];             // 0 constant, 1 tide(t), 2 inflow(t) x edge_val
    double edge_val[4];
    double t_end;
    double t, dt, dt_min, dt_max, rate;
    long long steps;
    int status, n_sub, n_sub_max, n_clamped;
    double acc[7];
    // output times k * out_dt, k = 1 .. n_out - 1 (k = 0, the initial state, is written
    // by the host); k_out is the next one.  Snapshot slots: 2-D depth and KP velocities
    // (n_out x cells), 1-D level and discharge (n_out x n1d), and the times reached.
    double out_dt;
    int n_out, k_out, cells, n1d;
    float *snap_h, *snap_u, *snap_v, *snap_eta, *snap_q;
    double *snap_t, *snap_ledger;    // ledger: LEDGER_N values per output (below)
};

// Volume ledger at an output time, in the order of the reference's snapshot ledger
// (coupling.py:229-242): 2-D surface, 1-D channel and retained volume, then the
// accumulated source terms.
enum : int { L_V2D = 0, L_V1D, L_STORE, L_RAIN, L_INFIL, L_BND2_IN, L_BND2_OUT, L_BND1_IN, L_BND1_OUT, L_CLIP,
             LEDGER_N };

// Piecewise-constant rain, harmonic tide and linearly interpolated inflow, as the
// reference evaluates them (engine.py:145-166, hyetograph.py:42-46, tide.py:29-31,
// catchment.py:32-40).
__device__ __forceinline__ double eng_rain(const EngMember& E, double t) {
    if (E.rain_n <= 0) return 0.0;
    const double k = floor((t - E.rain_t0) / E.rain_step + 1e-9);
    if (k < 0.0 || k >= (double)E.rain_n) return 0.0;
    return E.rain[(int)k];
}
__device__ __forceinline__ double eng_tide(const EngMember& E, double t) {
    const double tt = t + E.tide_shift;
    double eta = 0.0;
    for (int j = 0; j < E.tide_n; ++j) eta = eta + E.amp[j] * cos(E.w[j] * tt - E.ph[j]);
    return E.tide_base + (E.tide_on ? eta : 0.0);
}
__device__ __forceinline__ double eng_inflow(const EngMember& E, double t) {
    if (E.q_n <= 0) return 0.0;
    const double x = (t - E.q_t0) / E.q_step;
    if (x <= 0.0) return E.q[0];
    if (x >= (double)(E.q_n - 1)) return E.q[E.q_n - 1];
    const int k = (int)x;
    const double w = x - k;
    return (1.0 - w) * E.q[k] + w * E.q[k + 1];
}
__device__ __forceinline__ double eng_edge(const EngMember& E, int e, double t) {
    if (E.edge_src[e] == 1) return eng_tide(E, t);
    if (E.edge_src[e] == 2) return eng_inflow(E, t) * E.edge_val[e];
    return E.edge_val[e];
}

struct Consts {
    double g, h_dry, kp_eps, cfl, dt_min, dt_max;
    double cfl_1d, slot_width_frac, weir_cw, exchange_limit, exchange_relax;
    int order, hllc;
};

template <class R>
struct Grid {
    int ny, nx;
    int bc[4];
    double dx, dy, area, t0;
    int tile0, tiles_x, tiles_y, n_tiles;
    R *h, *hu, *hv, *sf, *ic;        // state: depth, momenta, retained water, infiltrated depth
    R *h1, *hu1, *hv1;               // stage-1 state (library scratch)
    const R *z, *n, *S, *f0, *fc, *k, *rw;
    R *pk, *ps;                      // optional running peak depth and speed
    R rdx, rdy, rt0;                 // dx, dy, Horton t0 in the compute type
    R idx, idy;                      // 1/dx, 1/dy (the float32 kernels multiply instead of dividing)
    R rarea;                         // 1 / cell area
};

// Per-member step parameters, in float64 and (for the float32 kernels, which must not
// convert on GB300's slow FP64 pipe) as float32 copies written by the same producer.
struct StepParams {
    double dt, t, rain;
    double bc0[4], bc1[4];
    int active, snap_k;              // snap_k: output slot written by this step, or -1
    float dt_f, t_f, rain_f, pad_f;
    float bc0_f[4], bc1_f[4];
    // this step's snapshot slots (NULL: no output at the end of this step)
    float *snap_h, *snap_u, *snap_v, *snap_eta, *snap_q;
    double* snap_ledger;
    double* vols;                    // the member's 5 step volumes for the caller (finalize), or NULL
};

__host__ __device__ inline void params_set_f32(StepParams& p) {
    p.dt_f = (float)p.dt;
    p.t_f = (float)p.t;
    p.rain_f = (float)p.rain;
    for (int e = 0; e < 4; ++e) {
        p.bc0_f[e] = (float)p.bc0[e];
        p.bc1_f[e] = (float)p.bc1[e];
    }
}

// The step record of one member from the ABI's step parameters: every field set
// (snapshot slot -1 and no snapshot pointers: no output at the end of this step), the
// float32 copies formed here.  Every producer of records on the host uses it.
inline StepParams step_params_from(const his_step_params& q) {
    StepParams sp{};
    sp.snap_k = -1;
    sp.dt = q.dt;
    sp.t = q.t;
    sp.rain = q.rain;
    for (int e = 0; e < 4; ++e) {
        sp.bc0[e] = q.bc_t[e];
        sp.bc1[e] = q.bc_t_dt[e];
    }
    sp.active = 1;
    params_set_f32(sp);
    return sp;
}

// The solver constants in the compute type R, converted on the host and passed by
// value: converting float64 constants inside the kernels put the float32 kernels on
// GB300's FP64 pipe (a small fraction of the float32 rate).
template <class R>
struct KC {
    R g, hg, h_dry, kp_eps;
    R h_kp;                          // depths from here on have h^4 >= kp_eps: no desingularisation
    int order, hllc;
};

template <class R>
inline KC<R> make_kc(const Consts& c) {
    KC<R> k;
    k.g = R(c.g);
    k.hg = R(0.5 * c.g);
    k.h_dry = R(c.h_dry);
    k.kp_eps = R(c.kp_eps);
    k.h_kp = R(std::sqrt(std::sqrt(c.kp_eps)) * (1.0 + 1e-12));
    k.order = c.order;
    k.hllc = c.hllc;
    return k;
}

// Step parameters in the compute type (no conversion in the float32 kernels)
template <class R> __device__ __forceinline__ R par_dt(const StepParams& p);
template <> __device__ __forceinline__ double par_dt<double>(const StepParams& p) { return p.dt; }
template <> __device__ __forceinline__ float par_dt<float>(const StepParams& p) { return p.dt_f; }
template <class R> __device__ __forceinline__ R par_t(const StepParams& p);
template <> __device__ __forceinline__ double par_t<double>(const StepParams& p) { return p.t; }
template <> __device__ __forceinline__ float par_t<float>(const StepParams& p) { return p.t_f; }
template <class R> __device__ __forceinline__ R par_rain(const StepParams& p);
template <> __device__ __forceinline__ double par_rain<double>(const StepParams& p) { return p.rain; }
template <> __device__ __forceinline__ float par_rain<float>(const StepParams& p) { return p.rain_f; }
template <class R> __device__ __forceinline__ R par_bc(const StepParams& p, int stage2, int e);
template <> __device__ __forceinline__ double par_bc<double>(const StepParams& p, int stage2, int e) {
    return stage2 ? p.bc1[e] : p.bc0[e];
}
template <> __device__ __forceinline__ float par_bc<float>(const StepParams& p, int stage2, int e) {
    return stage2 ? p.bc1_f[e] : p.bc0_f[e];
}

// ------------------------------------------------------------------ scalar helpers
// float64: the selections of the reference's torch.maximum/minimum/clamp on finite
// values, spelled out; float32: the native min/max instructions.
template <class R> __device__ __forceinline__ R rmax(R a, R b) {
    if constexpr (sizeof(R) == 4) return fmaxf(a, b);
    else return a > b ? a : (b > a ? b : a);
}
template <class R> __device__ __forceinline__ R rmin(R a, R b) {
    if constexpr (sizeof(R) == 4) return fminf(a, b);
    else return a < b ? a : (b < a ? b : a);
}
template <class R> __device__ __forceinline__ R relu(R x) {
    if constexpr (sizeof(R) == 4) return fmaxf(x, 0.0f);
    else return x > R(0) ? x : R(0);
}
template <class R> __device__ __forceinline__ R clamp0(R x) {
    if constexpr (sizeof(R) == 4) return fmaxf(x, 0.0f);
    else return x < R(0) ? R(0) : x;
}

__device__ __forceinline__ double dsqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float dsqrt(float x) { return sqrtf(x); }

__device__ __forceinline__ double cbrt_pow(double x) { return pow(x, 1.0 / 3.0); }
__device__ __forceinline__ float cbrt_pow(float x) { return powf(x, 1.0f / 3.0f); }

// Kurganov-Petrova desingularised velocity (swe2d.py:161-167):
// sqrt(2) h hu / sqrt(h^4 + max(h^4, eps)).  float64: where h^4 >= eps that is hu / h,
// one reciprocal instead of a power, a root and two divisions (10 FP64 instructions
// instead of 115, and four roundings fewer).
template <class R>
__device__ __forceinline__ void kp_velocity(const KC<R>& c, R h, R hu, R hv, R& u, R& v) {
    const R SQRT2 = R(1.4142135623730951);
    if constexpr (sizeof(R) == 4) {
        // (_rn: products the compiler must not fuse into a sum in one kernel and not another)
        const float h2 = h * h, h4 = __fmul_rn(h2, h2);
        const float s = SQRT2 * h * rsqrtf(h4 + fmaxf(h4, c.kp_eps));
        const bool wet = h >= c.h_dry;
        u = wet ? __fmul_rn(hu, s) : 0.0f;
        v = wet ? __fmul_rn(hv, s) : 0.0f;
    } else {
        u = v = 0.0;
        if (!f64_ge_pos(h, c.h_dry)) return;
        if (f64_ge_pos(h, c.h_kp)) {
            const double r = __drcp_rn(h);
            u = f64_div(hu, h, r);
            v = f64_div(hv, h, r);
        } else {
            const double h2 = h * h, h4 = h2 * h2;
            const double den = sqrt(h4 + (h4 > c.kp_eps ? h4 : c.kp_eps));
            u = SQRT2 * h * hu / den;
            v = SQRT2 * h * hv / den;
        }
    }
}

// Ghost states of stage and discharge edges from the adjacent interior cell
// (boundaries.py:63-78).  un is that cell's outward-normal velocity; the ghost's
// depth, outward-normal and tangential velocity are returned (its bed is the cell's).
template <class R>
__device__ __forceinline__ void stage_ghost(const KC<R>& c, R val, R h, R un, R ut, R z, R& hg_o, R& un_o, R& ut_o) {
    const R g = c.g, hd = c.h_dry;
    R hg = clamp0(val - z);
    R ci = dsqrt(g * h), cg = dsqrt(g * hg);
    bool wet_i = h >= hd;
    R ung = wet_i ? un + R(2) * (ci - cg) : R(0);
    bool sup = wet_i && (un > ci);
    if (sup) { ung = un; hg = h; }
    if (!(hg >= hd)) ung = R(0);
    hg_o = hg;
    un_o = ung;
    ut_o = ung > R(0) ? ut : R(0);
}

template <class R>
__device__ __forceinline__ void discharge_ghost(const KC<R>& c, R val, R h, R& hg_o, R& un_o, R& ut_o) {
    const R g = c.g, hd = c.h_dry;
    R hc = rmax(cbrt_pow(val * val / g), hd);
    R hg = h >= hd ? h : hc;
    hg_o = hg;
    un_o = -val / hg;
    ut_o = R(0);
}

// minmod: the smaller magnitude with the common sign, zero where the signs differ.
// min.xorsign.abs gives the smaller magnitude, negative where the signs differ (three
// instructions; the median of (a, b, 0) by min/max takes four).
//
// Returned doubled: t + |t| is 2 max(t, 0) exactly, and an add goes to another pipe than a
// maximum.  The march issues bursts of maxima, selects and logic that its half-rate pipe
// held up (0.58 of the 6.9 warp cycles an instruction took), so where a maximum with zero can
// be an add it is one (also in face_flux and the limiter); the factors of two go into
// constants.
__device__ __forceinline__ float minmod2(float a, float b) {
    float t;
    asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(t) : "f"(a), "f"(b));
    return __uint_as_float(__float_as_uint(t + fabsf(t)) | (__float_as_uint(a) & 0x80000000u));
}

// MUSCL face states of one cell along one axis (swe2d.py:205-219), float32 production
// form.  Inputs are the cell and its two neighbours along the axis; outputs the minus
// (left face) and plus (right face) reconstructions of h, normal and tangential velocity.
// The reconstruction is in difference form: the surface-elevation differences are
// dE = dh + dz (never forming eta = h + z, whose float32 rounding would be ulp(z) ~ 1e-6 m
// at tens of metres of terrain) and the reconstructed bed enters only through the in-cell
// bed slope sE - sH, so the hydrostatic reconstruction and the bed source keep their exact
// cancellation at rest.  Slopes are kept halved, as every use takes them.  (The float64
// form, with eta = h + z, is face64 in swe2d_tile64.cuh.)
struct Recon {
    float Hm, Hp, Um, Up, Vm, Vp;
    float z, d, h0, sE;                 // cell bed, half in-cell bed slope, depth, half eta slope
};

__device__ __forceinline__ Recon reconstruct(const KC<float>& c, float hm, float h0, float hp, float um, float u0,
                                             float up, float vm, float v0, float vp, float zm, float z0, float zp) {
    Recon r;
    r.z = z0;
    r.h0 = h0;
    r.sE = 0.0f;
    if (c.order == 2) {
        // 0 where the cell or a neighbour is dry
        const float half = fminf(fminf(hm, h0), hp) >= c.h_dry ? 0.25f : 0.0f;      // of a doubled slope
        const float sH = minmod2(h0 - hm, hp - h0) * half;
        const float mU = minmod2(u0 - um, up - u0), mV = minmod2(v0 - vm, vp - v0);
        r.Hm = h0 - sH;
        r.Hp = h0 + sH;
        r.Um = fmaf(-half, mU, u0);
        r.Up = fmaf(half, mU, u0);
        r.Vm = fmaf(-half, mV, v0);
        r.Vp = fmaf(half, mV, v0);
        r.sE = minmod2((h0 - hm) + (z0 - zm), (hp - h0) + (zp - z0)) * half;
        r.d = r.sE - sH;
    } else {
        r.Hm = r.Hp = h0;
        r.Um = r.Up = u0;
        r.Vm = r.Vp = v0;
        r.d = 0.0f;
    }
    return r;
}

// HLLC / HLL flux with two-rarefaction wave speeds and dry-bed fixes (swe2d.py:61-101) in
// well-balanced deviation form (float32 production form).  Instead of the momentum flux F2
// it returns, for each side s in {L, R},
//     D_s = F2 + corr_s - g/2 h_s^2 = F2 - g/2 h*_s^2
// (corr_s = g/2 (h_s^2 - h*_s^2) is the hydrostatic-reconstruction correction), so
// that the cell update -[(F2 + corrL)_east - (F2 + corrR)_west] + bed source becomes
// -[D_L,east - D_R,west] - g/2 (H+ + H-) sE: every term is small at rest and no
// O(g h^2 / 2) quantities cancel in float32.  The pressure difference across the face
// is formed from the depth difference, dp = g/2 (h*_R - h*_L)(h*_R + h*_L).
//
// The step is bound by the issue rate, so the flux is arranged for few instructions:
//  * the star speeds from the Riemann invariants a = uL + 2 cL, b = uR - 2 cR
//    (u* - c* = a/4 + 3b/4, u* + c* = 3a/4 + b/4), which are the dry-bed speeds as well: with
//    a dry side's invariant set to the other side's, its c being 0, the formulas for two wet
//    sides (uL - cL = a - 3 cL, uR + cR = b + 3 cR) give them;
//  * wave speeds clamped to SL <= 0 <= SR give the one-sided fluxes of supercritical faces
//    from the same formula, without branches;
//  * SR - SL > 0 wherever one side is wet, so it needs no guard;
//  * the contact speed's numerator SL hR (uR - SR) - SR hL (uL - SL) is -(SR - SL) F1 and its
//    denominator negative: the contact moves with the mass flux, whose sign picks the
//    tangential velocity;
//  * where both sides are dry, 1 / (SR - SL) := 0 makes every flux zero.
// A step of 64 resident storms of 400 x 325 cells: 363 -> 338 us with these (the contact's
// numerator still formed) and the skipped donor scaling (StripPipe::update); the contact by
// the mass flux, two selects fewer and the friction's and losses' shared quotients 330 -> 328
// us, 1601 x 1301 cells with the CFL rate 189 -> 185, first order 89.7 -> 85.5.
__device__ __forceinline__ void riemann_wb(const KC<float>& c, float hL, float uL, float vL, float hR, float uR,
                                           float vR, float jump, float& F1o, float& DLo, float& DRo, float& F3o) {
    const float tiny = 1e-14f;
    const float cL = sqrtf(c.g * hL), cR = sqrtf(c.g * hR);
    const bool dryL = hL <= tiny, dryR = hR <= tiny;
    const float a = fmaf(2.0f, cL, uL), b = fmaf(-2.0f, cR, uR);
    const float iL = dryL ? b : a, iR = dryR ? a : b;
    const float SL = fminf(fminf(fmaf(-3.0f, cL, iL), fmaf(0.25f, iL, 0.75f * iR)), 0.0f);
    const float SR = fmaxf(fmaxf(fmaf(3.0f, cR, iR), fmaf(0.25f, iR, 0.75f * iL)), 0.0f);
    const float inv = dryL && dryR ? 0.0f : 1.0f / (SR - SL);
    const float qL = __fmul_rn(hL, uL), qR = __fmul_rn(hR, uR);
    const float dp = c.hg * jump * (hR + hL);
    const float wL = SL * inv, wR = SR * inv, ww = wL * SR;
    const float F1 = fmaf(ww, jump, fmaf(-wL, qR, wR * qL));
    const float dyn = fmaf(ww, qR - qL, fmaf(-wL, qR * uR, wR * (qL * uL)));
    F1o = F1;
    DLo = fmaf(-wL, dp, dyn);
    DRo = fmaf(-wR, dp, dyn);
    if (c.hllc) {
        F3o = F1 * (F1 >= 0.0f ? vL : vR);
    } else {
        F3o = fmaf(ww, fmaf(hR, vR, -__fmul_rn(hL, vL)), fmaf(-wL, qR * vR, wR * (qL * vL)));
    }
}

// Face flux between two reconstructed cells (swe2d.py:226-234), float32: hydrostatic
// reconstruction z* = max(zL, zR), h* = max(0, h + z - z*); returns the mass flux,
// the momentum flux plus the left and right pressure corrections, and the
// tangential flux.
__device__ __forceinline__ void face_flux(const KC<float>& c, const Recon& L, const Recon& Rr, float& F1, float& F2L,
                                          float& F2R, float& F3) {
    const float hL = L.Hp, hR = Rr.Hm;
    // z* - zL = max(0, zR - zL), z* - zR = max(0, zL - zR), with
    // zR - zL = (z_R - z_L) - (half bed slopes) formed from the cell-bed difference
    const float zz = Rr.z - L.z;
    const float dz = zz - (L.d + Rr.d);
    const float aL = fmaf(-0.5f, dz + fabsf(dz), hL), aR = fmaf(-0.5f, fabsf(dz) - dz, hR);
    const float hLs = clamp0(aL), hRs = clamp0(aR);
    // surface jump h*_R - h*_L = (eta_R - eta_L) - (half eta slopes) when neither side is
    // clamped, formed from cell differences rather than from two rounded depths
    const float jump = fminf(aL, aR) > 0.0f ? ((Rr.h0 - L.h0) + zz) - (L.sE + Rr.sE) : hRs - hLs;
    riemann_wb(c, hLs, L.Up, L.Vp, hRs, Rr.Um, Rr.Vm, jump, F1, F2L, F2R, F3);
}

// ------------------------------------------------------------ block reductions
__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
// The same sum at the price of one vote where every lane holds zero
__device__ __forceinline__ double warp_sum_sparse(double v) {
    return __any_sync(0xffffffffu, f64_bits(v) << 1 != 0) ? warp_sum(v) : 0.0;
}
__device__ __forceinline__ double warp_max(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

}  // namespace his
