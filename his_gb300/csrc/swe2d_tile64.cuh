// 2-D finite-volume step of the plain float64 method: one CTA per strip-chunk, worked off
// in sub-tiles of up to TILE64_W x TILE64_H cells held in shared memory.
//
// What bounds it: the FP64 pipe (f64_ops.cuh), at about 310 FP64 instructions per cell in
// stage 1 and 430 in stage 2; DRAM and the integer pipe are far from their limits.  So
//  * a sub-tile is a list of independent items per phase (cells, slopes, faces, limiters,
//    updates) that all eight warps share, where a march up the rows keeps one warp per
//    column on a chain of 64-cycle instructions and leaves most of an SM's FP64 issue
//    slots empty on the small grids this method runs on;
//  * only what another item needs is computed: faces around the sub-tile's cells and their
//    four neighbours, slopes on the cells of those faces;
//  * the arithmetic is arranged for few FP64 instructions: slopes kept instead of the eight
//    reconstructed values of a cell, dt/dx instead of divisions by dx, one reciprocal per
//    flux and per velocity, no flux where both sides are dry, no limiter where nothing is
//    limited, and the momentum a cell loses with its water folded into its velocity.
// Phases of a sub-tile, a barrier between each: cells {h, u, v, h + z} with a three-cell
// halo (swe2d.py:161-167, boundaries.py:81-128); slopes in x and y (swe2d.py:205-219);
// face fluxes (swe2d.py:61-101, 226-234); the positivity limiter (swe2d.py:259-264); the
// update with, in the last stage, rain, infiltration, retention, friction, CFL rate and
// peaks (swe2d.py:305-371).
//
// This kernel does a stage in one launch; face64_kernel and cell64_kernel below do it in two
// with each face computed once, and serve every set with room for its faces.
//
// Measured (one member, 400 x 325 cells, infiltration and retention on, 58 x 16 chunks):
// 1340 us per step with the row-marching kernel this replaces, at 2000 FP64 instructions
// per cell and one warp on half of the schedulers; 250 us here, at 780 per cell with the
// FP64 pipe 80 % busy.
#pragma once
#include "swe2d_strip.cuh"

namespace his {

constexpr int TILE64_W = 58, TILE64_H = 16;     // largest sub-tile: 199 KB of shared memory
constexpr int TILE64_THREADS = 256;

// Shared memory of a w x h sub-tile: cells, slopes in x and y (second order), x- and
// y-faces, limiter.
__host__ __device__ constexpr size_t tile64_smem(int w, int h, bool second) {
    return 32 * ((size_t)(w + 6) * (h + 6) + (second ? (size_t)(w + 4) * (h + 2) + (size_t)(w + 2) * (h + 4) : 0) +
                 (size_t)(w + 3) * (h + 2) + (size_t)(w + 2) * (h + 3)) +
           8 * (size_t)(w + 2) * (h + 2);
}
static_assert(tile64_smem(TILE64_W, TILE64_H, true) <= 227 * 1024, "a sub-tile must fit one SM");

// Equal parts of at most `most` cells along one axis of n cells.  A member's sub-tile is
// the part of its full strip-chunk; a narrower last strip or lower last chunk is split
// into parts of at most that sub-tile.
__host__ __device__ inline int tile64_part(int n, int most) {
    const int k = (n + most - 1) / most;
    return (n + k - 1) / k;
}

// i / d and i % d for the items of a sub-tile: exact for i * d < 2^20
struct Div20 {
    unsigned m, d;
    __device__ __forceinline__ explicit Div20(int d_) : m(((1u << 20) + (unsigned)d_ - 1u) / (unsigned)d_), d((unsigned)d_) {}
    __device__ __forceinline__ int quot(int i) const { return (int)(((unsigned)i * m) >> 20); }
};
static_assert((TILE64_W + 6) * (TILE64_H + 6) * (TILE64_W + 6) < (1 << 20), "item division must be exact");

// Flux through one face from the cells {h, u, v, e} and slopes below and above it:
// hydrostatic reconstruction and HLLC / HLL with two-rarefaction speeds and dry fixes,
// {F1, F2 + left correction, F2 + right correction, F3}.
template <bool SECOND>
__device__ __forceinline__ Q4<double> face64(const KC<double>& c, const Q4<double>& cl, const Q4<double>& cr,
                                             const Q4<double>& sl, const Q4<double>& sr) {
    double HL = cl.a, uL = cl.b, vL = cl.c, EL = cl.d, HR = cr.a, uR = cr.b, vR = cr.c, ER = cr.d;
    if (SECOND) {
        HL = fma(0.5, sl.a, HL); uL = fma(0.5, sl.b, uL); vL = fma(0.5, sl.c, vL); EL = fma(0.5, sl.d, EL);
        HR = fma(-0.5, sr.a, HR); uR = fma(-0.5, sr.b, uR); vR = fma(-0.5, sr.c, vR); ER = fma(-0.5, sr.d, ER);
    }
    // h + z - z* in the reference's own order of rounding: written EL - z*, a front that
    // wets and dries (Thacker's bowl, second order) strays 5 times further from the recorded
    // run after two periods
    const double ZL = EL - HL, ZR = ER - HR;
    const double zf = f64_max(ZL, ZR);
    const double hL = f64_clamp0(HL + ZL - zf), hR = f64_clamp0(HR + ZR - zf);
    const double aL = c.g * hL, aR = c.g * hR;
    const double pL = 0.5 * (aL * hL), pR = 0.5 * (aR * hR);
    const double corrL = fma(c.hg, HL * HL, -pL), corrR = fma(c.hg, HR * HR, -pR);
    const double tiny = 1e-14;
    const bool dryL = f64_bits(hL) <= f64_bits(tiny), dryR = f64_bits(hR) <= f64_bits(tiny);
    if (dryL && dryR) return Q4<double>{0.0, corrL, corrR, 0.0};
    // (no root of zero: sqrt leaves its fast path there)
    const double cL = dryL ? 0.0 : sqrt(aL), cR = dryR ? 0.0 : sqrt(aR);
    const double s = uL + uR;
    double SL, SR;
    if (dryL) { SL = fma(-2.0, cR, uR); SR = uR + cR; }
    else if (dryR) { SL = uL - cL; SR = fma(2.0, cL, uL); }
    else {
        const double us = fma(0.5, s, cL - cR), t = fma(0.5, uL - uR, cL + cR);     // u*, 2 c*
        SL = f64_min(uL - cL, fma(-0.5, t, us));
        SR = f64_max(uR + cR, fma(0.5, t, us));
    }
    const double qL = hL * uL, qR = hR * uR;
    const double mL = fma(qL, uL, pL), mR = fma(qR, uR, pR);
    double F1, F2, F3 = 0.0;
    if (f64_plus(SL)) {
        F1 = qL; F2 = mL;
        if (!c.hllc) F3 = qL * vL;
    } else if (f64_minus(SR)) {
        F1 = qR; F2 = mR;
        if (!c.hllc) F3 = qR * vR;
    } else {
        double den = SR - SL;
        if (f64_mag_lt(den, tiny)) den = 1.0;
        const double r = __drcp_rn(den), SS = SL * SR;
        F1 = fma(SS, hR - hL, fma(-SL, qR, SR * qL)) * r;
        F2 = fma(SS, qR - qL, fma(-SL, mR, SR * mL)) * r;
        if (!c.hllc) F3 = fma(SS, hR * vR - hL * vL, fma(-SL, qR * vR, SR * (qL * vL))) * r;
    }
    if (c.hllc) {
        // the contact speed num / dd enters by its sign alone.  num = -(SR - SL) F1 and dd < 0, so
        // it is the sign of F1 wherever a side is deep enough (dd of -1e-13 and below) that the
        // guard of a vanishing dd has no part in it.  Seven FP64 instructions fewer per face: a
        // step of 400 x 325 cells with its CFL rate 273 -> 264 us, 4 resident ones 990 -> 953.
        // (F1's sign for every film: second-order Thacker strays 5 times further from the record.)
        bool east = !f64_neg(F1);
        if (f64_bits(hL) < f64_bits(1e-9) && f64_bits(hR) < f64_bits(1e-9)) {
            const double A = hR * (uR - SR), B = hL * (uL - SL);
            const double num = fma(SL, A, -(SR * B)), dd = A - B;
            east = f64_mag_lt(dd, tiny) ? !f64_neg(s)
                                        : (long long)(f64_bits(num) ^ f64_bits(dd)) >= 0 || f64_bits(num) << 1 == 0;
        }
        F3 = F1 * (east ? vL : vR);
    }
    return Q4<double>{F1, F2 + corrL, F2 + corrR, F3};
}

__device__ __forceinline__ double warp_max_run(double v) {
    for (int o = 16; o > 0; o >>= 1) v = f64_max_run(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// Constants of a member's step, the same for all its cells
struct Step64 {
    double dt, lamx, lamy, rdt, dtg, tt;
    unsigned feat;
    const StepParams& pr;
    __device__ __forceinline__ Step64(const KC<double>& c, const Grid<double>& gd, const StepParams& p, int stage)
        : dt(p.dt), lamx(p.dt / gd.dx), lamy(p.dt / gd.dy), rdt(p.rain * p.dt), dtg(p.dt * c.g),
          tt(clamp0(p.t - gd.rt0)), feat(grid_features(gd) | (stage != 1 && p.snap_h ? FEAT_SNAP : 0u)), pr(p) {}
};

// Running sums of one thread's cells
struct Acc64 {
    double clip = 0, xin = 0, xout = 0, yin = 0, yout = 0, infil = 0, rainw = 0, rate = 0, hsum = 0, ssum = 0, hmax = 0;
};

struct Pos64 {
    int gx, gy;
};

// Limiter of one cell inside the grid from its faces' mass fluxes (swe2d.py:259-264)
__device__ __forceinline__ double theta64(const Step64& k, double h, double Fw, double Fe, double Fs, double Fn) {
    const double need = fma(k.lamx, f64_relu(Fe) + f64_relu(-Fw), k.lamy * (f64_relu(Fn) + f64_relu(-Fs)));
    return f64_pos(need) && f64_key(need) > f64_key(h) ? h / need : 1.0;
}

// Update of cell j from its faces, the limiters around it, its depth hc and the bed terms
// (slope of h + z less slope of h, in x and y) (swe2d.py:305-371)
template <int STAGE>
__device__ __forceinline__ void update64(const KC<double>& c, const Grid<double>& gd, const Step64& k, Acc64& acc, Pos64 p,
                                         unsigned j, double hc, Q4<double> W, Q4<double> E, Q4<double> S, Q4<double> N,
                                         double thC, double thW, double thE, double thS, double thN, double bx,
                                         double by) {
    const unsigned long long one = f64_bits(1.0);
    if (((f64_bits(thC) ^ one) | (f64_bits(thW) ^ one) | (f64_bits(thE) ^ one) | (f64_bits(thS) ^ one) |
         (f64_bits(thN) ^ one)) != 0ull) {
        const double sw = f64_pos(W.a) ? thW : thC, se = f64_pos(E.a) ? thC : thE;
        const double ss = f64_pos(S.a) ? thS : thC, sn = f64_pos(N.a) ? thC : thN;
        W.a *= sw; W.d *= sw; E.a *= se; E.d *= se;
        S.a *= ss; S.d *= ss; N.a *= sn; N.d *= sn;
    }
    if (p.gx == 0) { acc.xin += f64_relu(W.a); acc.xout += f64_relu(-W.a); }
    if (p.gx == gd.nx - 1) { acc.xin += f64_relu(-E.a); acc.xout += f64_relu(E.a); }
    if (p.gy == 0) { acc.yin += f64_relu(S.a); acc.yout += f64_relu(-S.a); }
    if (p.gy == gd.ny - 1) { acc.yin += f64_relu(-N.a); acc.yout += f64_relu(N.a); }
    double px = W.c - E.b, py = S.c - N.b;
    if (STAGE != 0) {
        // bed source -g/2 (H- + H+)(Z+ - Z-) = -g h (slope of h + z less slope of h)
        const double gh = -(c.g * hc);
        px = fma(gh, bx, px);
        py = fma(gh, by, py);
    }
    const double dh = fma(k.lamx, W.a - E.a, k.lamy * (S.a - N.a));
    const double dhu = fma(k.lamx, px, k.lamy * (S.d - N.d));
    const double dhv = fma(k.lamx, W.d - E.d, k.lamy * py);
    double hn, hun, hvn;
    if (STAGE == 2) {
        hn = 0.5 * (gd.h[j] + (hc + dh));
        hun = 0.5 * (gd.hu[j] + (gd.hu1[j] + dhu));
        hvn = 0.5 * (gd.hv[j] + (gd.hv1[j] + dhv));
    } else {
        hn = hc + dh;
        hun = gd.hu[j] + dhu;
        hvn = gd.hv[j] + dhv;
    }
    if (f64_neg(hn)) { acc.clip -= hn; hn = 0.0; }
    if (STAGE == 1) {
        gd.h1[j] = hn; gd.hu1[j] = hun; gd.hv1[j] = hvn;
        return;
    }
    // ---- rain, Horton infiltration, retention store (swe2d.py:330-360)
    if (k.feat & FEAT_RAINW) {
        const double add = k.rdt * gd.rw[j];
        hn = hn + add;
        acc.rainw += add;
    } else {
        hn = hn + k.rdt;
    }
    const double hp = hn;              // depth the momentum belongs to
    double sf = 0.0;
    if (k.feat & FEAT_STORE) sf = gd.sf[j];
    if (k.feat & FEAT_HORTON) {
        const double fc = gd.fc[j];
        const double pot = fma(gd.f0[j] - fc, exp(-gd.k[j] * k.tt), fc) * k.dt;
        const double take = f64_min(pot, hn);
        hn = hn - take;
        double taken = take;
        if (k.feat & FEAT_STORE) {
            const double tks = f64_min(pot - take, sf);
            sf = sf - tks;
            taken = taken + tks;
        }
        acc.infil += taken;
        gd.ic[j] = gd.ic[j] + taken;
    }
    if (k.feat & FEAT_STORE) {
        const double fill = f64_min(f64_clamp0(gd.S[j] - sf), hn);
        hn = hn - fill;
        sf = sf + fill;
        gd.sf[j] = sf;
        acc.ssum += sf;
    }
    // ---- semi-implicit Manning friction (swe2d.py:362-370).  Water lost takes its
    // momentum along, so the velocity is that before the losses; dry cells rest
    double u2 = 0.0, v2 = 0.0;
    if (f64_ge_pos(hn, c.h_dry)) {
        const double r = __drcp_rn(hn);
        const bool plain = f64_ge_pos(hn, c.h_kp);
        double u, v;
        if (plain) {
            const double rp = f64_bits(hp) == f64_bits(hn) ? r : __drcp_rn(hp);
            u = v = 0.0;
            if (f64_pos(hp)) {             // (infiltration below zero wets dry cells)
                u = f64_div(hun, hp, rp);
                v = f64_div(hvn, hp, rp);
            }
        } else {
            const double keep = f64_pos(hp) ? hn / hp : 0.0;
            kp_velocity(c, hn, hun * keep, hvn * keep, u, v);
        }
        const double sq = fma(u, u, v * v);
        if (f64_pos(sq)) {             // water at rest has no friction (nor a fast root)
            const double nm = gd.n[j];
            const double p43 = f64_pow43(hn);
            const double fac = p43 / fma(k.dtg * nm * nm, sqrt(sq), p43);
            u = u * fac;
            v = v * fac;
        }
        hun = hn * u;
        hvn = hn * v;
        // KP velocities of the new state, for the CFL rate of the next step, the running
        // peak speed and the outputs (swe2d.py:161-167, coupling.py:229-242)
        if (plain) {
            u2 = f64_div(hun, hn, r);
            v2 = f64_div(hvn, hn, r);
        } else {
            kp_velocity(c, hn, hun, hvn, u2, v2);
        }
    } else {
        hun = 0.0;
        hvn = 0.0;
    }
    if (STAGE == 2) {
        gd.h[j] = hn; gd.hu[j] = hun; gd.hv[j] = hvn;
    } else {
        gd.h1[j] = hn; gd.hu1[j] = hun; gd.hv1[j] = hvn;
    }
    // (the caller's fields, of any start: not f64_max_run's)
    if (k.feat & FEAT_PEAK) gd.pk[j] = rmax(gd.pk[j], hn);
    if (k.feat & FEAT_PSPEED) gd.ps[j] = rmax(gd.ps[j], sqrt(fma(u2, u2, v2 * v2)));
    if (k.feat & FEAT_SNAP) {
        k.pr.snap_h[j] = (float)hn;
        k.pr.snap_u[j] = (float)u2;
        k.pr.snap_v[j] = (float)v2;
    }
    if (f64_ge_pos(hn, c.h_dry) && f64_bits(hn) != f64_bits(c.h_dry))
        acc.rate = f64_max_run(acc.rate, rate64(c, hn, u2, v2, gd.rdx, gd.rdy, gd.idx, gd.idy));
    acc.hsum += hn;
    acc.hmax = f64_max_run(acc.hmax, hn);
}

// Partial sums of a strip-chunk: lanes, then warps in order
template <int STAGE>
__device__ __forceinline__ void store_acc64(const Acc64& acc, double* out) {
    constexpr int NT = TILE64_THREADS, NV = STAGE == 1 ? 5 : 11;
    __shared__ double red[NT / 32][NV];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double v[NV] = {warp_sum_sparse(acc.clip), warp_sum_sparse(acc.xin), warp_sum_sparse(acc.xout),
                    warp_sum_sparse(acc.yin), warp_sum_sparse(acc.yout)};
    if constexpr (STAGE != 1) {
        v[5] = warp_sum_sparse(acc.infil);
        v[6] = warp_sum_sparse(acc.rainw);
        v[7] = warp_max_run(acc.rate);
        v[8] = warp_sum_sparse(acc.hsum);
        v[9] = warp_sum_sparse(acc.ssum);
        v[10] = warp_max_run(acc.hmax);
    }
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < NV; ++q) red[warp][q] = v[q];
    }
    __syncthreads();
    if (tid < NV) {
        double a = red[0][tid];
        if (tid == 7 || tid == 10) {
            for (int w = 1; w < NT / 32; ++w) a = f64_max_run(a, red[w][tid]);
        } else {
            for (int w = 1; w < NT / 32; ++w) a += red[w][tid];
        }
        const int b = STAGE == 2 ? P_CLIP2 : P_CLIP1;
        out[tid < 5 ? b + tid : P_INFIL + (tid - 5)] = a;
    }
}

// Slopes of the middle cell o of three {h, u, v, e} along an axis; zero beside dry cells
// (swe2d.py:205-219)
__device__ __forceinline__ Q4<double> slope64(const KC<double>& c, const Q4<double>& m, const Q4<double>& o,
                                              const Q4<double>& q) {
    Q4<double> s{0.0, 0.0, 0.0, 0.0};
    if (f64_ge_pos(m.a, c.h_dry) && f64_ge_pos(o.a, c.h_dry) && f64_ge_pos(q.a, c.h_dry)) {
        s.a = f64_minmod(o.a - m.a, q.a - o.a);
        s.b = f64_minmod(o.b - m.b, q.b - o.b);
        s.c = f64_minmod(o.c - m.c, q.c - o.c);
        s.d = f64_minmod(o.d - m.d, q.d - o.d);
    }
    return s;
}

// The face's flux along y: normal velocity first
template <bool SECOND>
__device__ __forceinline__ Q4<double> face64_along(bool alongx, const KC<double>& c, Q4<double> L, Q4<double> R,
                                                   Q4<double> sl, Q4<double> sr) {
    if (!alongx) {
        double t = L.b; L.b = L.c; L.c = t;
        t = R.b; R.b = R.c; R.c = t;
        t = sl.b; sl.b = sl.c; sl.c = t;
        t = sr.b; sr.b = sr.c; sr.c = t;
    }
    return face64<SECOND>(c, L, R, sl, sr);
}

// STAGE: 0 = first-order full step (into the stage buffers), 1 = RK stage 1, 2 = RK stage
// 2 and sources, as strip_kernel's.
template <int STAGE>
__global__ void __launch_bounds__(TILE64_THREADS, 1) tile64_kernel(const Grid<double>* __restrict__ grids,
                                                                   const StripRef* __restrict__ strips,
                                                                   const StepParams* __restrict__ params,
                                                                   const KC<double> kc, double* __restrict__ partials) {
    constexpr bool SECOND = STAGE != 0;
    constexpr int NT = TILE64_THREADS;
    extern __shared__ __align__(32) unsigned char smem_raw[];
    __shared__ Grid<double> gd;
    __shared__ double bcv[4];
    KC<double> c = kc;
    c.order = SECOND ? 2 : 1;
    const StripRef sr = strips[blockIdx.x];
    const StepParams& pr = params[sr.member];
    if (!pr.active) return;
    const int tid = threadIdx.x;
    {
        const unsigned* src = reinterpret_cast<const unsigned*>(grids + sr.member);
        unsigned* dst = reinterpret_cast<unsigned*>(&gd);
        for (int k = tid; k < (int)(sizeof(Grid<double>) / 4); k += NT) dst[k] = src[k];
    }
    if (tid < 4) bcv[tid] = par_bc<double>(pr, STAGE == 2, tid);
    __syncthreads();
    const double* __restrict__ H = STAGE == 2 ? gd.h1 : gd.h;
    const double* __restrict__ HU = STAGE == 2 ? gd.hu1 : gd.hu;
    const double* __restrict__ HV = STAGE == 2 ? gd.hv1 : gd.hv;
    const int nx = gd.nx, ny = gd.ny;
    const Step64 k(c, gd, pr, STAGE);
    Acc64 acc;

    // parts of at most the member's sub-tile, which the launch's shared memory is sized for
    const int cw = tile64_part(sr.w, sr.sub_w), ch = tile64_part(sr.y1 - sr.y0, sr.sub_h);
    for (int Y0 = sr.y0; Y0 < sr.y1; Y0 += ch)
        for (int X0 = sr.x0; X0 < sr.x0 + sr.w; X0 += cw) {
            const int w = min(cw, sr.x0 + sr.w - X0), h = min(ch, sr.y1 - Y0);
            // cells at (x + 3, y + 3), x-slopes (x + 2, y + 1), y-slopes (x + 1, y + 2), x-faces
            // (x + 1, y + 1), y-faces (x + 1, y + 1), limiter (x + 1, y + 1) of sub-tile cell (x, y);
            // a face lies below (west, south of) the cell it is named by
            const int LC = w + 6, LX = w + 4, LY = w + 2, LF = w + 3, LG = w + 2, LT = w + 2;
            Q4<double>* s_c = reinterpret_cast<Q4<double>*>(smem_raw);
            Q4<double>* s_sx = s_c + LC * (h + 6);
            Q4<double>* s_sy = s_sx + (SECOND ? LX * (h + 2) : 0);
            Q4<double>* s_fx = s_sy + (SECOND ? LY * (h + 4) : 0);
            Q4<double>* s_fy = s_fx + LF * (h + 2);
            double* s_th = reinterpret_cast<double*>(s_fy + LG * (h + 3));
            __syncthreads();                       // the last sub-tile's readers are done
            {
                const Div20 by(LC);
                for (int i = tid; i < LC * (h + 6); i += NT) {
                    const int iy = by.quot(i), y = iy - 3, x = i - iy * LC - 3;
                    // cells more than three faces away from the sub-tile have no part in it
                    const int away = max(max(-x, x - (w - 1)), 0) + max(max(-y, y - (h - 1)), 0);
                    if (away > 3) continue;
                    const HaloRaw<double> a = halo_fetch(c, gd, H, HU, HV, X0 + x, Y0 + y);
                    Q4<double> q;
                    halo_build(c, gd, bcv, a, X0 + x, Y0 + y, q.a, q.b, q.c, q.d);
                    q.d = q.a + q.d;
                    s_c[i] = q;
                }
            }
            __syncthreads();
            if (SECOND) {
                const Div20 bx(LX), by(LY);
                const int nsx = LX * (h + 2), nsx32 = (nsx + 31) & ~31, n = nsx32 + LY * (h + 4);
                for (int i = tid; i < n; i += NT) {
                    const bool alongx = i < nsx32;
                    if (alongx && i >= nsx) continue;
                    const int e = alongx ? i : i - nsx32;
                    const int iy = alongx ? bx.quot(e) : by.quot(e);
                    const int x = alongx ? e - iy * LX - 2 : e - iy * LY - 1, y = iy - (alongx ? 1 : 2);
                    // on the cells of the faces below, within the rows (columns) of the grid
                    if (alongx) {
                        if ((unsigned)(Y0 + y) >= (unsigned)ny || ((y < 0 || y >= h) && (x < -1 || x > w))) continue;
                    } else {
                        if ((unsigned)(X0 + x) >= (unsigned)nx || ((x < 0 || x >= w) && (y < -1 || y > h))) continue;
                    }
                    const int p = (y + 3) * LC + x + 3, d = alongx ? 1 : LC;
                    const Q4<double> m = s_c[p - d], o = s_c[p], q = s_c[p + d];
                    const Q4<double> s = slope64(c, m, o, q);
                    if (alongx) s_sx[e] = s;
                    else s_sy[e] = s;
                }
                __syncthreads();
            }
            {
                const Div20 bx(LF), by(LG);
                const int nfx = LF * (h + 2), nfx32 = (nfx + 31) & ~31, n = nfx32 + LG * (h + 3);
                for (int i = tid; i < n; i += NT) {
                    const bool alongx = i < nfx32;
                    if (alongx && i >= nfx) continue;
                    const int e = alongx ? i : i - nfx32;
                    const int iy = alongx ? bx.quot(e) : by.quot(e);
                    const int x = e - iy * (alongx ? LF : LG) - 1, y = iy - 1;
                    // the faces of the sub-tile's cells and of their four neighbours inside the grid
                    if (alongx) {
                        if ((unsigned)(Y0 + y) >= (unsigned)ny || (unsigned)(X0 + x) > (unsigned)nx ||
                            ((y < 0 || y >= h) && (x < 0 || x > w))) continue;
                    } else {
                        if ((unsigned)(X0 + x) >= (unsigned)nx || (unsigned)(Y0 + y) > (unsigned)ny ||
                            ((x < 0 || x >= w) && (y < 0 || y > h))) continue;
                    }
                    const int p = (y + 3) * LC + x + 3;
                    Q4<double> sl{}, sr_{};
                    if (SECOND) {
                        const Q4<double>* s = alongx ? s_sx + (y + 1) * LX + x + 2 : s_sy + (y + 2) * LY + x + 1;
                        sl = s[alongx ? -1 : -LY];
                        sr_ = s[0];
                    }
                    const Q4<double> f = face64_along<SECOND>(alongx, c, s_c[p - (alongx ? 1 : LC)], s_c[p], sl, sr_);
                    if (alongx) s_fx[e] = f;
                    else s_fy[e] = f;
                }
            }
            __syncthreads();
            {
                const Div20 by(LT);
                for (int i = tid; i < LT * (h + 2); i += NT) {
                    const int iy = by.quot(i), y = iy - 1, x = i - iy * LT - 1;
                    const bool xi = x >= 0 && x < w, yi = y >= 0 && y < h;
                    if (!xi && !yi) continue;
                    double th = 1.0;               // outside the grid
                    if ((unsigned)(X0 + x) < (unsigned)nx && (unsigned)(Y0 + y) < (unsigned)ny) {
                        const int fx = (y + 1) * LF + x + 1, fy = (y + 1) * LG + x + 1;
                        th = theta64(k, s_c[(y + 3) * LC + x + 3].a, s_fx[fx].a, s_fx[fx + 1].a, s_fy[fy].a,
                                     s_fy[fy + LG].a);
                    }
                    s_th[i] = th;
                }
            }
            __syncthreads();
            const Div20 by(w);
            for (int i = tid; i < w * h; i += NT) {
                const int y = by.quot(i), x = i - y * w, gx = X0 + x, gy = Y0 + y;
                const int fx = (y + 1) * LF + x + 1, fy = (y + 1) * LG + x + 1, t0 = (y + 1) * LT + x + 1;
                double ex = 0.0, ey = 0.0;
                if (SECOND) {
                    const Q4<double> sx = s_sx[(y + 1) * LX + x + 2], sy = s_sy[(y + 2) * LY + x + 1];
                    ex = sx.d - sx.a;
                    ey = sy.d - sy.a;
                }
                update64<STAGE>(c, gd, k, acc, Pos64{gx, gy}, (unsigned)gy * (unsigned)nx + (unsigned)gx,
                                s_c[(y + 3) * LC + x + 3].a, s_fx[fx], s_fx[fx + 1], s_fy[fy], s_fy[fy + LG], s_th[t0],
                                s_th[t0 - 1], s_th[t0 + 1], s_th[t0 - LT], s_th[t0 + LT], ex, ey);
            }
        }
    store_acc64<STAGE>(acc, partials + (size_t)blockIdx.x * NPART);
}

// ------------------------------------------------ faces and cells in two kernels
// The sub-tile above computes the faces around its cells' neighbours as well, 2.4 to 3.3
// faces per cell, because the limiter of a neighbour enters a cell's update.  With room for
// the faces in memory, one kernel computes each face once and a second one limits and
// updates from them: 2 faces per cell, 220 FP64 instructions per cell in stage 1 against 330,
// for 80 bytes per cell written and about 200 read (mostly from L2) per stage, which a kernel
// at 2 FP64 lanes per cycle and SM hardly notices.  The cells' arithmetic and the order of
// their sums are the fused kernel's: the same bits.  A step of 400 x 325 cells 249 -> 228 us,
// of four such members 901 -> 752, of 16 of 100 x 81 273 -> 236; 100 x 81 alone 55 -> 52.
// (512 threads per CTA: faces 72 -> 69 us, cells 52 -> 55 and 17 -> 18.)
struct Faces64 {
    Q4<double>*fx, *fy;              // west faces (ny x (nx + 1)) and south faces ((ny + 1) x nx)
    double2* bed;                    // per cell: slope of h + z less slope of h, in x and y
};
// Shared memory of the face kernel over a w x h sub-tile (cells with a two-cell halo, slopes)
__host__ __device__ constexpr size_t face64_smem(int w, int h, bool second) {
    return 32 * ((size_t)(w + 4) * (h + 4) + (second ? (size_t)(w + 2) * h + (size_t)w * (h + 2) : 0));
}
__host__ __device__ constexpr size_t cell64_smem(int w, int h) { return 8 * (size_t)(w + 2) * (h + 2); }

template <int STAGE>
__global__ void __launch_bounds__(TILE64_THREADS, 2) face64_kernel(const Grid<double>* __restrict__ grids,
                                                                   const Faces64* __restrict__ faces,
                                                                   const StripRef* __restrict__ strips,
                                                                   const StepParams* __restrict__ params,
                                                                   const KC<double> kc) {
    constexpr bool SECOND = STAGE != 0;
    constexpr int NT = TILE64_THREADS;
    extern __shared__ __align__(32) unsigned char smem_raw[];
    __shared__ Grid<double> gd;
    __shared__ double bcv[4];
    KC<double> c = kc;
    c.order = SECOND ? 2 : 1;
    const StripRef sr = strips[blockIdx.x];
    const StepParams& pr = params[sr.member];
    if (!pr.active) return;
    const int tid = threadIdx.x;
    {
        const unsigned* src = reinterpret_cast<const unsigned*>(grids + sr.member);
        unsigned* dst = reinterpret_cast<unsigned*>(&gd);
        for (int k = tid; k < (int)(sizeof(Grid<double>) / 4); k += NT) dst[k] = src[k];
    }
    if (tid < 4) bcv[tid] = par_bc<double>(pr, STAGE == 2, tid);
    const Faces64 out = faces[sr.member];
    __syncthreads();
    const double* __restrict__ H = STAGE == 2 ? gd.h1 : gd.h;
    const double* __restrict__ HU = STAGE == 2 ? gd.hu1 : gd.hu;
    const double* __restrict__ HV = STAGE == 2 ? gd.hv1 : gd.hv;
    const int nx = gd.nx, ny = gd.ny;
    const int cw = tile64_part(sr.w, sr.sub_w), ch = tile64_part(sr.y1 - sr.y0, sr.sub_h);
    for (int Y0 = sr.y0; Y0 < sr.y1; Y0 += ch)
        for (int X0 = sr.x0; X0 < sr.x0 + sr.w; X0 += cw) {
            const int w = min(cw, sr.x0 + sr.w - X0), h = min(ch, sr.y1 - Y0);
            // the grid's last column and row carry the faces beyond them as well
            const int xe = X0 + w == nx, ye = Y0 + h == ny;
            // cells at (x + 2, y + 2), x-slopes (x + 1, y), y-slopes (x, y + 1) of cell (x, y)
            const int LC = w + 4, LX = w + 2;
            Q4<double>* s_c = reinterpret_cast<Q4<double>*>(smem_raw);
            Q4<double>* s_sx = s_c + LC * (h + 4);
            Q4<double>* s_sy = s_sx + LX * h;
            __syncthreads();                       // the last sub-tile's readers are done
            {
                const Div20 by(LC);
                for (int i = tid; i < LC * (h + 4); i += NT) {
                    const int iy = by.quot(i), y = iy - 2, x = i - iy * LC - 2;
                    const bool xin = x >= 0 && x < w, yin = y >= 0 && y < h;
                    if (!(yin && x <= w + xe) && !(xin && y <= h + ye)) continue;
                    const HaloRaw<double> a = halo_fetch(c, gd, H, HU, HV, X0 + x, Y0 + y);
                    Q4<double> q;
                    halo_build(c, gd, bcv, a, X0 + x, Y0 + y, q.a, q.b, q.c, q.d);
                    q.d = q.a + q.d;
                    s_c[i] = q;
                }
            }
            __syncthreads();
            if (SECOND) {
                // x-slopes of columns -1 .. w - 1 (+ 1), y-slopes of rows -1 .. h - 1 (+ 1)
                const int wx = w + 1 + xe, hy = h + 1 + ye;
                const Div20 bx(wx), by(w);
                const int nsx = wx * h, nsx32 = (nsx + 31) & ~31, n = nsx32 + w * hy;
                for (int i = tid; i < n; i += NT) {
                    const bool alongx = i < nsx32;
                    if (alongx && i >= nsx) continue;
                    const int e = alongx ? i : i - nsx32, iy = alongx ? bx.quot(e) : by.quot(e);
                    const int x = alongx ? e - iy * wx - 1 : e - iy * w, y = alongx ? iy : iy - 1;
                    const int p = (y + 2) * LC + x + 2, d = alongx ? 1 : LC;
                    const Q4<double> s = slope64(c, s_c[p - d], s_c[p], s_c[p + d]);
                    if (alongx) s_sx[y * LX + x + 1] = s;
                    else s_sy[(y + 1) * w + x] = s;
                }
                __syncthreads();
            }
            const int wx = w + xe, hy = h + ye;
            const Div20 bx(wx), by(w);
            const int nfx = wx * h, nfx32 = (nfx + 31) & ~31, n = nfx32 + w * hy;
            for (int i = tid; i < n; i += NT) {
                const bool alongx = i < nfx32;
                if (alongx && i >= nfx) continue;
                const int e = alongx ? i : i - nfx32, y = alongx ? bx.quot(e) : by.quot(e);
                const int x = e - y * (alongx ? wx : w);
                const int p = (y + 2) * LC + x + 2;
                Q4<double> sl{}, sr_{};
                if (SECOND) {
                    const Q4<double>* s = alongx ? s_sx + y * LX + x + 1 : s_sy + (y + 1) * w + x;
                    sl = s[alongx ? -1 : -w];
                    sr_ = s[0];
                }
                const Q4<double> f = face64_along<SECOND>(alongx, c, s_c[p - (alongx ? 1 : LC)], s_c[p], sl, sr_);
                if (alongx) out.fx[(size_t)(Y0 + y) * (nx + 1) + (X0 + x)] = f;
                else out.fy[(size_t)(Y0 + y) * nx + (X0 + x)] = f;
            }
            if (SECOND) {
                const Div20 bw(w);
                for (int i = tid; i < w * h; i += NT) {
                    const int y = bw.quot(i), x = i - y * w;
                    const Q4<double> sx = s_sx[y * LX + x + 1], sy = s_sy[(y + 1) * w + x];
                    out.bed[(size_t)(Y0 + y) * nx + (X0 + x)] = double2{sx.d - sx.a, sy.d - sy.a};
                }
            }
        }
}

template <int STAGE>
__global__ void __launch_bounds__(TILE64_THREADS, STAGE == 1 ? 2 : 1)
cell64_kernel(const Grid<double>* __restrict__ grids, const Faces64* __restrict__ faces,
              const StripRef* __restrict__ strips, const StepParams* __restrict__ params, const KC<double> kc,
              double* __restrict__ partials) {
    constexpr int NT = TILE64_THREADS;
    extern __shared__ __align__(32) unsigned char smem_raw[];
    __shared__ Grid<double> gd;
    KC<double> c = kc;
    c.order = STAGE != 0 ? 2 : 1;
    const StripRef sr = strips[blockIdx.x];
    const StepParams& pr = params[sr.member];
    if (!pr.active) return;
    const int tid = threadIdx.x;
    {
        const unsigned* src = reinterpret_cast<const unsigned*>(grids + sr.member);
        unsigned* dst = reinterpret_cast<unsigned*>(&gd);
        for (int k = tid; k < (int)(sizeof(Grid<double>) / 4); k += NT) dst[k] = src[k];
    }
    const Faces64 in = faces[sr.member];
    __syncthreads();
    const double* __restrict__ H = STAGE == 2 ? gd.h1 : gd.h;
    const Q4<double>* __restrict__ fx = in.fx;
    const Q4<double>* __restrict__ fy = in.fy;
    const int nx = gd.nx, ny = gd.ny;
    const Step64 k(c, gd, pr, STAGE);
    Acc64 acc;
    const int cw = tile64_part(sr.w, sr.sub_w), ch = tile64_part(sr.y1 - sr.y0, sr.sub_h);
    double* s_th = reinterpret_cast<double*>(smem_raw);
    for (int Y0 = sr.y0; Y0 < sr.y1; Y0 += ch)
        for (int X0 = sr.x0; X0 < sr.x0 + sr.w; X0 += cw) {
            const int w = min(cw, sr.x0 + sr.w - X0), h = min(ch, sr.y1 - Y0), LT = w + 2;
            __syncthreads();                       // the last sub-tile's readers are done
            {
                const Div20 by(LT);
                for (int i = tid; i < LT * (h + 2); i += NT) {
                    const int iy = by.quot(i), y = iy - 1, x = i - iy * LT - 1;
                    if (!(x >= 0 && x < w) && !(y >= 0 && y < h)) continue;
                    const int gx = X0 + x, gy = Y0 + y;
                    double th = 1.0;               // outside the grid
                    if ((unsigned)gx < (unsigned)nx && (unsigned)gy < (unsigned)ny) {
                        const size_t jx = (size_t)gy * (nx + 1) + gx, j = (size_t)gy * nx + gx;
                        th = theta64(k, H[j], fx[jx].a, fx[jx + 1].a, fy[j].a, fy[j + nx].a);
                    }
                    s_th[i] = th;
                }
            }
            __syncthreads();
            const Div20 by(w);
            for (int i = tid; i < w * h; i += NT) {
                const int y = by.quot(i), x = i - y * w, gx = X0 + x, gy = Y0 + y, t0 = (y + 1) * LT + x + 1;
                const size_t jx = (size_t)gy * (nx + 1) + gx, j = (size_t)gy * nx + gx;
                double2 bed{0.0, 0.0};
                if (STAGE != 0) bed = in.bed[j];
                update64<STAGE>(c, gd, k, acc, Pos64{gx, gy}, (unsigned)j, H[j], fx[jx], fx[jx + 1], fy[j], fy[j + nx],
                                s_th[t0], s_th[t0 - 1], s_th[t0 + 1], s_th[t0 - LT], s_th[t0 + LT], bed.x, bed.y);
            }
        }
    store_acc64<STAGE>(acc, partials + (size_t)blockIdx.x * NPART);
}

}  // namespace his
