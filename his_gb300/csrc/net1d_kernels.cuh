// 1-D St. Venant network step and 1-D <-> 2-D weir exchange (one CTA per member).
//
// The channel network is small (10^2 - 10^3 cells): a member's whole network lives
// in shared memory for all of its substeps.  Scatter-adds of the reference
// (torch index_add over faces / links) become per-cell gathers over CSR lists kept
// in the reference's index order, so every sum has the reference's association
// and the result does not depend on thread scheduling.
//
// The drop-in 1-D step (net_step_kernel) is float64 in both precisions.  The
// device-resident engine's float32 form (net_engine_kernel_f32) computes section
// geometry, wave speeds, HLL fluxes, limiter and friction in float32 over float64
// area and discharge state, float64 updates and tallies, and float64 junction depths
// (the level-pool solve); its float64 form (net_engine_kernel) is float64 throughout.
// The weir exchange is float64 in the plain method; in the production form its
// per-link arithmetic is float32 (GB300's float64 pipe runs at a small fraction of the
// float32 rate and this work sits on every step's critical path), with the 1-D area
// update and the exchanged-volume tallies kept in float64.
//
// Reference: hydrointel/solver/swe1d.py:51-107, :253-368; coupling.py:73-124.
#pragma once
#include "his_device.cuh"

namespace his {

struct Net {
    int n_cells, n_faces;
    const int *kind, *gsrc, *fl, *fr;
    const double* gsign;
    const int *lstart, *lidx, *rstart, *ridx;      // faces where the cell is left / right (face order)
    const double *z, *nman, *dx;
    const double *b, *m, *yb, *ts;                 // cell sections
    const double *fb, *fm, *fyb, *fts;             // face sections
    const float *zf, *dxf, *bf, *mf, *ybf, *tsf;   // float32 copies of z, dx and the cell sections
    const float *nmanf, *gsignf;                   // float32 roughness and ghost signs
    const float *fbf, *fmf, *fybf, *ftsf;          // float32 face sections
    double *A, *Q;
};

struct Lnk {
    // Links in the order of their 1-D cell (within a cell in the caller's order), so that a
    // cell's links are contiguous; orig: the caller's index
    int n_links, n_unique, v_offset, pad;
    const int *cell1d, *inv, *uniq, *orig;
    const double *zbank, *length, *z2;
    const float *zbank_f, *length_f, *z2_f;        // float32 copies for the production form
    const int *ustart, *uidx;                      // unique 2-D cell -> links (caller's order)
    const int *ufirst;                             // its link where it has exactly one, else -1
    const int *cstart;                             // 1-D cell -> its links
};

// ---------------------------------------------------------------- sections (swe1d.py:51-84)
struct Sec {
    const double *b, *m, *yb, *ts;
};

__device__ __forceinline__ double sec_area(const Sec& s, int i, double y) {
    double yt = fmin(y, s.yb[i]);
    double at = yt * (s.b[i] + s.m[i] * yt);
    return at + s.ts[i] * clamp0(y - s.yb[i]);
}
__device__ __forceinline__ double sec_top(const Sec& s, int i, double y) {
    return y <= s.yb[i] ? s.b[i] + 2.0 * s.m[i] * y : s.ts[i];
}
__device__ __forceinline__ double sec_i1(const Sec& s, int i, double y) {
    double yt = fmin(y, s.yb[i]);
    double above = clamp0(y - s.yb[i]);
    double it = s.b[i] * yt * yt / 2.0 + s.m[i] * (yt * yt * yt) / 3.0;
    double at = yt * (s.b[i] + s.m[i] * yt);
    return it + at * above + s.ts[i] * above * above / 2.0;
}
__device__ __forceinline__ double sec_perim(const Sec& s, int i, double y) {
    double yt = fmin(y, s.yb[i]);
    return s.b[i] + 2.0 * yt * sqrt(1.0 + s.m[i] * s.m[i]);
}
__device__ __forceinline__ double sec_bank_area(const Sec& s, int i) { return s.yb[i] * (s.b[i] + s.m[i] * s.yb[i]); }
__device__ __forceinline__ double sec_depth(const Sec& s, int i, double A) {
    A = clamp0(A);
    double ab = sec_bank_area(s, i);
    double b = s.b[i];
    double y_t = 2.0 * A / (b + sqrt(b * b + 4.0 * s.m[i] * A));
    return A <= ab ? y_t : s.yb[i] + (A - ab) / s.ts[i];
}
__device__ __forceinline__ double vel1d(const Consts& c, const Sec& s, int i, double A, double Q) {
    double y = sec_depth(s, i, A);
    return y >= c.h_dry ? Q / fmax(A, 1e-12) : 0.0;
}

// HLL flux of the 1-D equations (swe1d.py:87-107)
__device__ __forceinline__ void hll_1d(double AL, double QL, double pL, double cL, double AR, double QR, double pR,
                                       double cR, double uL, double uR, double& F1o, double& F2o) {
    const double tiny = 1e-14;
    bool dryL = AL <= tiny, dryR = AR <= tiny;
    double SL = rmin(uL - cL, uR - cR);
    double SR = rmax(uL + cL, uR + cR);
    if (dryL) { SL = uR - 2.0 * cR; SR = uR + cR; }
    if (dryR) { SL = uL - cL; SR = uL + 2.0 * cL; }
    double FL1 = QL, FR1 = QR;
    double FL2 = QL * uL + pL, FR2 = QR * uR + pR;
    double den = SR - SL;
    if (fabs(den) < tiny) den = 1.0;
    bool left = SL >= 0.0, right = SR <= 0.0;
    double F1, F2;
    if (left) { F1 = FL1; F2 = FL2; }
    else if (right) { F1 = FR1; F2 = FR2; }
    else {
        F1 = (SR * FL1 - SL * FR1 + SL * SR * (AR - AL)) / den;
        F2 = (SR * FL2 - SL * FR2 + SL * SR * (QR - QL)) / den;
    }
    if (dryL && dryR) { F1 = 0.0; F2 = 0.0; }
    F1o = F1;
    F2o = F2;
}

// Deterministic block sum of NV doubles; result valid in thread 0.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = warp_sum(v[j]);
    if (lane == 0)
        for (int j = 0; j < NV; ++j) red[warp * NV + j] = v[j];
    __syncthreads();
    if (threadIdx.x == 0)
        for (int j = 0; j < NV; ++j) {
            double a = red[j];
            for (int w = 1; w < nw; ++w) a += red[w * NV + j];
            v[j] = a;
        }
    __syncthreads();
}

__host__ __device__ inline size_t net_smem_bytes(int n_cells, int n_faces) {
    return sizeof(double) * (7 * (size_t)n_cells + 4 * (size_t)n_faces + 32 * 4);
}

// n_sub substeps of dt/n_sub each for the network N, run by the whole CTA.
// forcing: per substep (inflow, stage).  vols (thread 0, if non-NULL): bnd_in,
// bnd_out, clip summed over the substeps.  sm: net_smem_bytes() of shared memory.
__device__ __forceinline__ void net_substeps_dev(const Net& N, const Consts& c, double dt_total, int n_sub,
                                                 const double* __restrict__ forcing, double* vols, double* sm,
                                                 float* snap_eta = nullptr, float* snap_q = nullptr,
                                                 double* snap_v1d = nullptr) {
    const int nc = N.n_cells, nf = N.n_faces, tid = threadIdx.x, nt = blockDim.x;
    double *A = sm, *Q = A + nc, *Ag = Q + nc, *Qg = Ag + nc, *yv = Qg + nc, *uv = yv + nc, *th = uv + nc;
    double *F1 = th + nc, *F2 = F1 + nf, *pL = F2 + nf, *pR = pL + nf, *red = pR + nf;
    const Sec s{N.b, N.m, N.yb, N.ts}, fs{N.fb, N.fm, N.fyb, N.fts};
    const double g = c.g, dt = dt_total / n_sub;
    for (int i = tid; i < nc; i += nt) { A[i] = N.A[i]; Q[i] = N.Q[i]; }
    __syncthreads();
    double tot_in = 0.0, tot_out = 0.0, tot_clip = 0.0;
    for (int k = 0; k < n_sub; ++k) {
        const double q_in = forcing[2 * k + 0];
        const double eta = forcing[2 * k + 1];
        // ghost cells from the interior neighbour (swe1d.py:265-294)
        for (int i = tid; i < nc; i += nt) {
            const int kd = N.kind[i];
            if (kd < 2) { Ag[i] = A[i]; Qg[i] = Q[i]; continue; }
            const int src = N.gsrc[i];
            const double As = A[src], Qs = Q[src], sg = N.gsign[i];
            const double ys = sec_depth(s, i, As);
            const double un = sg * vel1d(c, s, i, As, Qs);
            const bool wet_i = ys >= c.h_dry;
            double An, Qn;
            if (kd == 3) {
                double yst = clamp0(eta - N.z[i]);
                double Ast = sec_area(s, i, yst);
                double ci = sqrt(g * As / sec_top(s, i, ys));
                double cg = sqrt(g * Ast / sec_top(s, i, yst));
                double un_st = wet_i ? un + 2.0 * (ci - cg) : 0.0;
                if (wet_i && (un > ci)) { un_st = un; Ast = As; }
                if (!(sec_depth(s, i, Ast) >= c.h_dry)) un_st = 0.0;
                An = Ast;
                Qn = sg * Ast * un_st;
            } else if (kd == 2) {
                double yc = fmax(pow(q_in * q_in / (g * N.b[i] * N.b[i]), 1.0 / 3.0), c.h_dry);
                An = wet_i ? As : sec_area(s, i, yc);
                Qn = -sg * q_in;
            } else {
                An = As;
                Qn = -Qs;
            }
            Ag[i] = An;
            Qg[i] = Qn;
        }
        __syncthreads();
        for (int i = tid; i < nc; i += nt) {
            yv[i] = sec_depth(s, i, Ag[i]);
            uv[i] = vel1d(c, s, i, Ag[i], Qg[i]);
        }
        __syncthreads();
        // face fluxes with hydrostatic reconstruction (swe1d.py:326-336)
        for (int f = tid; f < nf; f += nt) {
            const int l = N.fl[f], r = N.fr[f];
            const double zL = N.z[l], zR = N.z[r], zf = rmax(zL, zR);
            const double yL = clamp0(zL + yv[l] - zf), yR = clamp0(zR + yv[r] - zf);
            const double AL = sec_area(fs, f, yL), AR = sec_area(fs, f, yR);
            const double uL = uv[l], uR = uv[r];
            pL[f] = g * sec_i1(fs, f, yL);
            pR[f] = g * sec_i1(fs, f, yR);
            const double cL = sqrt(g * AL / sec_top(fs, f, yL));
            const double cR = sqrt(g * AR / sec_top(fs, f, yR));
            hll_1d(AL, AL * uL, pL[f], cL, AR, AR * uR, pR[f], cR, uL, uR, F1[f], F2[f]);
        }
        __syncthreads();
        // outflow limiter; ghosts unlimited (swe1d.py:337-344)
        for (int i = tid; i < nc; i += nt) {
            double out = 0.0;
            for (int j = N.lstart[i]; j < N.lstart[i + 1]; ++j) out += relu(F1[N.lidx[j]]);
            for (int j = N.rstart[i]; j < N.rstart[i + 1]; ++j) out += relu(-F1[N.ridx[j]]);
            const double vol = Ag[i] * N.dx[i];
            const double need = out * dt;
            const double t = need > vol ? vol / (need > 0.0 ? need : 1.0) : 1.0;
            th[i] = N.kind[i] >= 2 ? 1.0 : t;
        }
        __syncthreads();
        double bsum[3] = {0.0, 0.0, 0.0};
        for (int f = tid; f < nf; f += nt) {
            const double sc = F1[f] > 0.0 ? th[N.fl[f]] : th[N.fr[f]];
            const double Fs = F1[f] * sc;
            F1[f] = Fs;
            if (N.kind[N.fl[f]] >= 2) { bsum[0] += relu(Fs); bsum[1] += relu(-Fs); }
            if (N.kind[N.fr[f]] >= 2) { bsum[0] += relu(-Fs); bsum[1] += relu(Fs); }
        }
        __syncthreads();
        // update, clip, semi-implicit friction; ghosts keep their filled state (swe1d.py:345-368)
        for (int i = tid; i < nc; i += nt) {
            double dA = 0.0, dQ = 0.0;
            for (int j = N.lstart[i]; j < N.lstart[i + 1]; ++j) dA += -F1[N.lidx[j]];
            for (int j = N.rstart[i]; j < N.rstart[i + 1]; ++j) dA += F1[N.ridx[j]];
            for (int j = N.lstart[i]; j < N.lstart[i + 1]; ++j) { int f = N.lidx[j]; dQ += -(F2[f] - pL[f]); }
            for (int j = N.rstart[i]; j < N.rstart[i + 1]; ++j) { int f = N.ridx[j]; dQ += F2[f] - pR[f]; }
            const int kd = N.kind[i];
            double A1 = Ag[i] + dt * dA / N.dx[i];
            double Q1 = Qg[i] + dt * dQ / N.dx[i];
            const double neg = clamp0(-A1);
            bsum[2] += neg * N.dx[i] * (kd >= 2 ? 0.0 : 1.0);
            A1 = A1 + neg;
            const double y1 = sec_depth(s, i, A1);
            const double Ac = fmax(A1, 1e-12);
            const double R = Ac / sec_perim(s, i, y1);
            const double nm = N.nman[i];
            const double denom = 1.0 + dt * g * (nm * nm) * fabs(Q1) / (Ac * pow(fmax(R, c.h_dry), 4.0 / 3.0));
            Q1 = Q1 / denom;
            if (!((y1 >= c.h_dry) && kd != 1)) Q1 = 0.0;
            if (kd >= 2) { A1 = Ag[i]; Q1 = Qg[i]; }
            A[i] = A1;
            Q[i] = Q1;
        }
        block_sum<3>(bsum, red);
        if (tid == 0) {
            tot_in += bsum[0] * dt;
            tot_out += bsum[1] * dt;
            tot_clip += bsum[2];
        }
    }
    __syncthreads();
    for (int i = tid; i < nc; i += nt) { N.A[i] = A[i]; N.Q[i] = Q[i]; }
    if (snap_eta) {                         // output: level z + depth and discharge (coupling.py:229-242)
        double v1 = 0.0;
        for (int i = tid; i < nc; i += nt) {
            snap_eta[i] = (float)(N.z[i] + sec_depth(s, i, A[i]));
            snap_q[i] = (float)Q[i];
            if (N.kind[i] <= 1) v1 += A[i] * N.dx[i];
        }
        if (snap_v1d) {                     // channel volume over the interior cells (swe1d.py:245-247)
            double vv[1] = {v1};
            block_sum<1>(vv, red);
            if (tid == 0) *snap_v1d = vv[0];
        }
    }
    if (tid == 0 && vols) {
        vols[0] = tot_in;
        vols[1] = tot_out;
        vols[2] = tot_clip;
    }
}


// ---------------------------------------------------------- float32 substeps
// The production form of the network step: section geometry, wave speeds, fluxes,
// the outflow limiter and friction in float32 arithmetic; the state (cross-section
// area A and discharge Q), its per-substep update, the clip and boundary tallies, and
// the depth of the junction level pools in float64.  GB300 runs float64 at a small
// fraction of its float32 rate, and the float64 network filled one SM's float64 pipe.
struct SecF {
    const float *b, *m, *yb, *ts;
};
__device__ __forceinline__ float secf_area(const SecF& s, int i, float y) {
    const float yt = fminf(y, s.yb[i]);
    return yt * (s.b[i] + s.m[i] * yt) + s.ts[i] * fmaxf(y - s.yb[i], 0.0f);
}
__device__ __forceinline__ float secf_top(const SecF& s, int i, float y) {
    return y <= s.yb[i] ? s.b[i] + 2.0f * s.m[i] * y : s.ts[i];
}
__device__ __forceinline__ float secf_i1(const SecF& s, int i, float y) {
    const float yt = fminf(y, s.yb[i]);
    const float above = fmaxf(y - s.yb[i], 0.0f);
    const float it = s.b[i] * yt * yt * 0.5f + s.m[i] * (yt * yt * yt) * (1.0f / 3.0f);
    const float at = yt * (s.b[i] + s.m[i] * yt);
    return it + at * above + s.ts[i] * above * above * 0.5f;
}
__device__ __forceinline__ float secf_perim(const SecF& s, int i, float y) {
    const float yt = fminf(y, s.yb[i]);
    return s.b[i] + 2.0f * yt * sqrtf(1.0f + s.m[i] * s.m[i]);
}
__device__ __forceinline__ float secf_depth(const SecF& s, int i, float A) {
    A = fmaxf(A, 0.0f);
    const float b = s.b[i], yb = s.yb[i];
    const float ab = yb * (b + s.m[i] * yb);
    return A <= ab ? 2.0f * A / (b + sqrtf(b * b + 4.0f * s.m[i] * A)) : yb + (A - ab) / s.ts[i];
}

__device__ __forceinline__ void hll_1d_f32(float AL, float QL, float pL, float cL, float AR, float QR, float pR,
                                           float cR, float uL, float uR, float& F1o, float& F2o) {
    const float tiny = 1e-14f;
    const bool dryL = AL <= tiny, dryR = AR <= tiny;
    float SL = fminf(uL - cL, uR - cR);
    float SR = fmaxf(uL + cL, uR + cR);
    if (dryL) { SL = uR - 2.0f * cR; SR = uR + cR; }
    if (dryR) { SL = uL - cL; SR = uL + 2.0f * cL; }
    const float FL2 = QL * uL + pL, FR2 = QR * uR + pR;
    float den = SR - SL;
    if (fabsf(den) < tiny) den = 1.0f;
    float F1, F2;
    if (SL >= 0.0f) { F1 = QL; F2 = FL2; }
    else if (SR <= 0.0f) { F1 = QR; F2 = FR2; }
    else {
        const float inv = 1.0f / den;
        F1 = (SR * QL - SL * QR + SL * SR * (AR - AL)) * inv;
        F2 = (SR * FL2 - SL * FR2 + SL * SR * (QR - QL)) * inv;
    }
    if (dryL && dryR) { F1 = 0.0f; F2 = 0.0f; }
    F1o = F1;
    F2o = F2;
}

// Shared memory of the float32 substeps: the state in float64 (A, Q and their
// ghost-filled copies), a reduction slot, the per-substep float32 work arrays, and the
// network's static geometry and connectivity staged once per launch, so that no phase
// waits on a global load (a lone CTA per network has no other warps to hide it).
__host__ __device__ inline size_t net_smem_bytes_f32(int n_cells, int n_faces) {
    const size_t nc = (size_t)n_cells, nf = (size_t)n_faces;
    return sizeof(double) * (4 * nc + 32 * 4) + sizeof(float) * (4 * nc + 4 * nf) +   // state, red; work
           sizeof(float) * (8 * nc + 4 * nf) +                                       // cell and face geometry
           sizeof(int) * (2 * nc + 2 * nf + 2 * (nc + 1) + 2 * nf) + 16;             // kinds, faces, CSR
}

// n_sub substeps of dt/n_sub each for the network N (the arguments of net_substeps_dev).
__device__ __forceinline__ void net_substeps_f32_dev(const Net& N, const Consts& c, double dt_total, int n_sub,
                                                     const double* __restrict__ forcing, double* vols, double* sm,
                                                     float* snap_eta = nullptr, float* snap_q = nullptr,
                                                     double* snap_v1d = nullptr) {
    const int nc = N.n_cells, nf = N.n_faces, tid = threadIdx.x, nt = blockDim.x;
    double *A = sm, *Q = A + nc, *Ag = Q + nc, *Qg = Ag + nc, *red = Qg + nc;      // red: 128 doubles
    float *Af = reinterpret_cast<float*>(red + 32 * 4), *yv = Af + nc, *uv = yv + nc, *th = uv + nc;
    float *F1 = th + nc, *F2 = F1 + nf, *pL = F2 + nf, *pR = pL + nf;
    // staged geometry
    float *zs = pR + nf, *dxs = zs + nc, *bs = dxs + nc, *ms = bs + nc, *ybs = ms + nc, *tss = ybs + nc,
          *nms = tss + nc, *gss = nms + nc;
    float *fbs = gss + nc, *fms = fbs + nf, *fybs = fms + nf, *ftss = fybs + nf;
    int *kind = reinterpret_cast<int*>(ftss + nf), *gsrc = kind + nc, *fl = gsrc + nc, *fr = fl + nf;
    int *lst = fr + nf, *rst = lst + nc + 1, *lix = rst + nc + 1, *rix = lix + nf;
    for (int i = tid; i < nc; i += nt) {
        A[i] = N.A[i]; Q[i] = N.Q[i];
        zs[i] = N.zf[i]; dxs[i] = N.dxf[i]; bs[i] = N.bf[i]; ms[i] = N.mf[i]; ybs[i] = N.ybf[i]; tss[i] = N.tsf[i];
        nms[i] = N.nmanf[i]; gss[i] = N.gsignf[i];
        kind[i] = N.kind[i]; gsrc[i] = N.gsrc[i];
    }
    for (int i = tid; i <= nc; i += nt) { lst[i] = N.lstart[i]; rst[i] = N.rstart[i]; }
    for (int f = tid; f < nf; f += nt) {
        fbs[f] = N.fbf[f]; fms[f] = N.fmf[f]; fybs[f] = N.fybf[f]; ftss[f] = N.ftsf[f];
        fl[f] = N.fl[f]; fr[f] = N.fr[f];
        lix[f] = N.lidx[f]; rix[f] = N.ridx[f];
    }
    const SecF s{bs, ms, ybs, tss}, fs{fbs, fms, fybs, ftss};
    const Sec sd{N.b, N.m, N.yb, N.ts};
    __shared__ float s_k[3];
    if (tid == 0) {
        s_k[0] = (float)c.g;
        s_k[1] = (float)c.h_dry;
        s_k[2] = (float)(dt_total / n_sub);
    }
    __syncthreads();
    const float g = s_k[0], h_dry = s_k[1], dt = s_k[2];
    double tot_in = 0.0, tot_out = 0.0, tot_clip = 0.0;
    for (int k = 0; k < n_sub; ++k) {
        const float q_in = (float)forcing[2 * k + 0];
        const float eta = (float)forcing[2 * k + 1];
        // ghost cells from the interior neighbour (swe1d.py:265-294)
        for (int i = tid; i < nc; i += nt) {
            const int kd = kind[i];
            if (kd < 2) {
                Ag[i] = A[i];
                Qg[i] = Q[i];
                Af[i] = (float)A[i];
                continue;
            }
            const int src = gsrc[i];
            const float As = (float)A[src], Qs = (float)Q[src], sg = gss[i];
            const float ys = secf_depth(s, i, As);
            const float un = sg * (ys >= h_dry ? Qs / fmaxf(As, 1e-12f) : 0.0f);
            const bool wet_i = ys >= h_dry;
            float An, Qn;
            if (kd == 3) {
                const float yst = fmaxf(eta - zs[i], 0.0f);
                float Ast = secf_area(s, i, yst);
                const float ci = sqrtf(g * As / secf_top(s, i, ys));
                const float cg = sqrtf(g * Ast / secf_top(s, i, yst));
                float un_st = wet_i ? un + 2.0f * (ci - cg) : 0.0f;
                if (wet_i && (un > ci)) { un_st = un; Ast = As; }
                if (!(secf_depth(s, i, Ast) >= h_dry)) un_st = 0.0f;
                An = Ast;
                Qn = sg * Ast * un_st;
            } else if (kd == 2) {
                const float b = bs[i];
                const float yc = fmaxf(cbrtf(q_in * q_in / (g * b * b)), h_dry);
                An = wet_i ? As : secf_area(s, i, yc);
                Qn = -sg * q_in;
            } else {
                An = As;
                Qn = -Qs;
            }
            Ag[i] = (double)An;
            Qg[i] = (double)Qn;
            Af[i] = An;
        }
        __syncthreads();
        // depth and velocity; a junction's level-pool depth in float64
        for (int i = tid; i < nc; i += nt) {
            const float y = kind[i] == 1 ? (float)sec_depth(sd, i, Ag[i]) : secf_depth(s, i, Af[i]);
            yv[i] = y;
            uv[i] = y >= h_dry ? (float)Qg[i] / fmaxf(Af[i], 1e-12f) : 0.0f;
        }
        __syncthreads();
        // face fluxes with hydrostatic reconstruction (swe1d.py:326-336)
        for (int f = tid; f < nf; f += nt) {
            const int l = fl[f], r = fr[f];
            const float zL = zs[l], zR = zs[r], zfc = fmaxf(zL, zR);
            const float yL = fmaxf(zL + yv[l] - zfc, 0.0f), yR = fmaxf(zR + yv[r] - zfc, 0.0f);
            const float AL = secf_area(fs, f, yL), AR = secf_area(fs, f, yR);
            const float uL = uv[l], uR = uv[r];
            const float pl = g * secf_i1(fs, f, yL), pr = g * secf_i1(fs, f, yR);
            pL[f] = pl;
            pR[f] = pr;
            const float cL = sqrtf(g * AL / secf_top(fs, f, yL));
            const float cR = sqrtf(g * AR / secf_top(fs, f, yR));
            hll_1d_f32(AL, AL * uL, pl, cL, AR, AR * uR, pr, cR, uL, uR, F1[f], F2[f]);
        }
        __syncthreads();
        // outflow limiter; ghosts unlimited (swe1d.py:337-344)
        for (int i = tid; i < nc; i += nt) {
            float out = 0.0f;
            for (int j = lst[i]; j < lst[i + 1]; ++j) out += fmaxf(F1[lix[j]], 0.0f);
            for (int j = rst[i]; j < rst[i + 1]; ++j) out += fmaxf(-F1[rix[j]], 0.0f);
            const float vol = Af[i] * dxs[i];
            const float need = out * dt;
            const float t = need > vol ? vol / (need > 0.0f ? need : 1.0f) : 1.0f;
            th[i] = kind[i] >= 2 ? 1.0f : t;
        }
        __syncthreads();
        double bsum[3] = {0.0, 0.0, 0.0};
        for (int f = tid; f < nf; f += nt) {
            const float sc = F1[f] > 0.0f ? th[fl[f]] : th[fr[f]];
            const float Fs = F1[f] * sc;
            F1[f] = Fs;
            if (kind[fl[f]] >= 2) { bsum[0] += fmaxf(Fs, 0.0f); bsum[1] += fmaxf(-Fs, 0.0f); }
            if (kind[fr[f]] >= 2) { bsum[0] += fmaxf(-Fs, 0.0f); bsum[1] += fmaxf(Fs, 0.0f); }
        }
        __syncthreads();
        // update in float64, clip, semi-implicit friction; ghosts keep their filled state
        // (swe1d.py:345-368)
        for (int i = tid; i < nc; i += nt) {
            float dA = 0.0f, dQ = 0.0f;
            for (int j = lst[i]; j < lst[i + 1]; ++j) { const int f = lix[j]; dA -= F1[f]; dQ -= F2[f] - pL[f]; }
            for (int j = rst[i]; j < rst[i + 1]; ++j) { const int f = rix[j]; dA += F1[f]; dQ += F2[f] - pR[f]; }
            const int kd = kind[i];
            const float rdx = 1.0f / dxs[i];
            double A1 = Ag[i] + (double)(dt * dA * rdx);
            double Q1 = Qg[i] + (double)(dt * dQ * rdx);
            const double neg = clamp0(-A1);
            if (neg > 0.0 && kd < 2) bsum[2] += neg * N.dx[i];
            A1 = A1 + neg;
            const float A1f = (float)A1;
            const float y1 = secf_depth(s, i, A1f);
            const float Ac = fmaxf(A1f, 1e-12f);
            const float R = Ac / secf_perim(s, i, y1);
            const float nm = nms[i];
            const float denom = 1.0f + dt * g * (nm * nm) * fabsf((float)Q1) / (Ac * powf(fmaxf(R, h_dry), 4.0f / 3.0f));
            Q1 = Q1 / (double)denom;
            if (!((y1 >= h_dry) && kd != 1)) Q1 = 0.0;
            if (kd >= 2) { A1 = Ag[i]; Q1 = Qg[i]; }
            A[i] = A1;
            Q[i] = Q1;
        }
        bsum[0] *= (double)dt;
        bsum[1] *= (double)dt;
        block_sum<3>(bsum, red);
        if (tid == 0) {
            tot_in += bsum[0];
            tot_out += bsum[1];
            tot_clip += bsum[2];
        }
    }
    __syncthreads();
    for (int i = tid; i < nc; i += nt) { N.A[i] = A[i]; N.Q[i] = Q[i]; }
    if (snap_eta) {                         // output: level z + depth and discharge (coupling.py:229-242)
        double v1 = 0.0;
        for (int i = tid; i < nc; i += nt) {
            snap_eta[i] = (float)(N.z[i] + sec_depth(sd, i, A[i]));
            snap_q[i] = (float)Q[i];
            if (kind[i] <= 1) v1 += A[i] * N.dx[i];
        }
        if (snap_v1d) {                     // channel volume over the interior cells (swe1d.py:245-247)
            double vv[1] = {v1};
            block_sum<1>(vv, red);
            if (tid == 0) *snap_v1d = vv[0];
        }
    }
    if (tid == 0 && vols) {
        vols[0] = tot_in;
        vols[1] = tot_out;
        vols[2] = tot_clip;
    }
}

// Shared memory the exchange of one member uses: volumes per link, depth and limit per
// unique 2-D cell, level (then limit) and storage per 1-D cell, and the reductions.
__host__ __device__ inline size_t exchange_smem_bytes(int n_links, int n_unique, int n_cells, size_t size) {
    return sizeof(double) * 96 + size * ((size_t)n_links + 2 * (size_t)n_unique + 2 * (size_t)n_cells);
}

// Barrier `id` among n threads (whole warps) of a CTA
__device__ __forceinline__ void bar_group(int id, int n) { asm volatile("barrier.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// What the exchange and the CFL reduction need of one 1-D cell: water level, plan area,
// volume above the bank, and the wave rate of a wet interior cell (0 otherwise).
template <class R>
struct CellLevel {
    R eta, plan, avail, rate;
    bool wet;
};

// Production form: float32 from float32 copies of the section tables.
__device__ __forceinline__ CellLevel<float> cell_level(const Net& N, int i, float g, float h_dry, bool rate) {
    CellLevel<float> o;
    const float A = fmaxf((float)N.A[i], 0.0f);
    const float b = N.bf[i], m = N.mf[i], yb = N.ybf[i], ts = N.tsf[i], dx = N.dxf[i];
    const float ab = yb * (b + m * yb);
    const float y = A <= ab ? 2.0f * A / (b + sqrtf(b * b + 4.0f * m * A)) : yb + (A - ab) / ts;
    const float top = y <= yb ? b + 2.0f * m * y : ts;
    o.eta = N.zf[i] + y;
    o.plan = top * dx;
    o.avail = fmaxf(A - ab, 0.0f) * dx;
    o.wet = rate && N.kind[i] <= 1 && y > h_dry;
    o.rate = o.wet ? (fabsf((float)N.Q[i] / fmaxf(A, 1e-12f)) + sqrtf(g * A / top)) / dx : 0.0f;
    return o;
}
__device__ __forceinline__ CellLevel<double> cell_level(const Net& N, int i, double g, double h_dry, bool rate) {
    CellLevel<double> o;
    const Sec s{N.b, N.m, N.yb, N.ts};
    const double A = N.A[i], dx = N.dx[i];
    const double y = sec_depth(s, i, A), top = sec_top(s, i, y);
    o.eta = N.z[i] + y;
    o.plan = top * dx;
    o.avail = clamp0(A - sec_bank_area(s, i)) * dx;
    o.wet = rate && N.kind[i] <= 1 && y > h_dry;
    o.rate = o.wet ? (fabs(N.Q[i] / fmax(A, 1e-12)) + sqrt(g * A / top)) / dx : 0.0;
    return o;
}

// Signed volume of one link over dt before the donor limits (coupling.py:78-97): positive
// from the 2-D to the 1-D side.  rp: 1 / (2-D cell area) + 1 / (1-D plan area).
__device__ __forceinline__ float link_volume(float eta1, float eta2, float zb, float len, float rp, float dt, float cw,
                                             float relax) {
    const float up = fmaxf(eta1, eta2), dn = fminf(eta1, eta2);
    const float d_up = fmaxf(up - zb, 0.0f), d_dn = fmaxf(dn - zb, 0.0f);
    const float ratio = d_up > 0.0f ? d_dn / d_up : 0.0f;
    const float sub = powf(fmaxf(1.0f - ratio * sqrtf(ratio), 0.0f), 0.385f);
    const float q = cw * len * (d_up * sqrtf(d_up)) * sub;
    const float v = fminf(q * dt, relax * ((up - dn) / rp));
    return eta2 > eta1 ? v : -v;
}
// float64: a link whose water stands below its bank moves nothing, so the powers of the
// weir formula (d^1.5 = d sqrt(d), and pow(., 0.385) only where the weir is submerged) are
// left to the few links that overtop.
__device__ __forceinline__ double link_volume(double eta1, double eta2, double zb, double len, double rp, double dt,
                                              double cw, double relax) {
    const double up = rmax(eta1, eta2), dn = rmin(eta1, eta2);
    const double d_up = f64_clamp0(up - zb);
    if (f64_bits(d_up) == 0) return 0.0;
    const double d_dn = f64_clamp0(dn - zb);
    double q = cw * len * (d_up * sqrt(d_up));
    if (f64_bits(d_dn) != 0) {
        const double ratio = d_dn / d_up;
        q = q * pow(f64_clamp0(1.0 - ratio * sqrt(ratio)), 0.385);
    }
    const double v = rmin(q * dt, relax * ((up - dn) / rp));
    return eta2 > eta1 ? v : -v;
}

__device__ __forceinline__ float pos_part(float x) { return fmaxf(x, 0.0f); }
__device__ __forceinline__ double pos_part(double x) { return f64_relu(x); }

// Constants of the exchange and the channel rate in the compute type, formed on the host
template <class R>
struct ExchK {
    R g, h_dry, cw, relax, limit;
};
template <class R>
inline ExchK<R> make_exch_k(const Consts& c) {
    return ExchK<R>{(R)c.g, (R)c.h_dry, (R)c.weir_cw, (R)c.exchange_relax, (R)c.exchange_limit};
}

// A member record copied to shared memory by the CTA (its pointers are read many times)
template <class T>
__device__ __forceinline__ void stage_record(T* dst, const T* src) {
    static_assert(sizeof(T) % 4 == 0, "copied as 32-bit words");
    for (int k = threadIdx.x; k < (int)(sizeof(T) / 4); k += blockDim.x)
        reinterpret_cast<unsigned*>(dst)[k] = reinterpret_cast<const unsigned*>(src)[k];
}

// Weir exchange of one member by nt threads (whole warps, this one tid) of a CTA
// (coupling.py:73-124), with the 1-D CFL rate of the same cells.  float64 plain method;
// float32 in the production form (GB300's float64 pipe runs at a small fraction of the
// float32 rate), with the 1-D area update and the tallies in float64.
//
// It is a chain of dependent phases on one SM, bound by the latency of their loads.  So
// every static table entry and 2-D depth a thread needs is fetched before the first
// barrier, for EXCH_SLOTS links and 2-D cells per thread at once (more in a loop), and the
// later phases run from registers and shared memory; links lie in the order of their 1-D
// cell, so a cell's sum walks contiguous shared memory.  Measured with the pre kernel
// below, a step of six served storms in float32 89 -> 78 us, one of a 400 x 325 storm in
// float64 444 -> 313 us.
//
// sync: barrier of the nt threads.  ready(): barrier with whoever chooses dt; returns it.
//  go(): barrier before the states are changed; false leaves them as they are.
// s_rate (optional): per warp the largest rate of a wet cell, -1 where none is wet.
constexpr int EXCH_SLOTS = 3;
template <class R, class Sync, class Ready, class Go>
__device__ __forceinline__ void exchange_dev(const Lnk& L, const Net& N, const Grid<R>& gd, const ExchK<R>& K,
                                             double* __restrict__ Vout, double* __restrict__ exch, int mb, double* sm,
                                             int tid, int nt, R* s_rate, Sync sync, Ready ready, Go go) {
    constexpr int S = EXCH_SLOTS;
    constexpr bool F32 = sizeof(R) == 4;
    const int nl = L.n_links, nu = L.n_unique, nc = N.n_cells;
    const R area = R(gd.area);
    double* red = sm;                                   // 64 doubles used
    R* V = reinterpret_cast<R*>(sm + 96);
    R *hq = V + nl, *f2 = hq + nu, *eta1 = f2 + nu, *rp = eta1 + nc, *f1 = eta1;
    auto zbank = [&](int l) -> R { if constexpr (F32) return L.zbank_f[l]; else return L.zbank[l]; };
    auto length = [&](int l) -> R { if constexpr (F32) return L.length_f[l]; else return L.length[l]; };
    auto z2 = [&](int l) -> R { if constexpr (F32) return L.z2_f[l]; else return L.z2[l]; };

    int c1[S], q2[S], cell[S], u0[S];
    R zb[S], len[S], zz[S];
#pragma unroll
    for (int j = 0; j < S; ++j) {
        const int k = tid + j * nt;
        cell[j] = u0[j] = 0;
        if (k < nu) { cell[j] = L.uniq[k]; u0[j] = L.ufirst[k]; }
        c1[j] = q2[j] = 0;
        zb[j] = len[j] = zz[j] = R(0);
        if (k < nl) { c1[j] = L.cell1d[k]; q2[j] = L.inv[k]; zb[j] = zbank(k); len[j] = length(k); zz[j] = z2(k); }
    }
#pragma unroll
    for (int j = 0; j < S; ++j) {
        const int k = tid + j * nt;
        if (k < nu) hq[k] = gd.h[cell[j]];
    }
    for (int k = tid + S * nt; k < nu; k += nt) hq[k] = gd.h[L.uniq[k]];
    R rate = R(-1);
    for (int i = tid; i < nc; i += nt) {
        const CellLevel<R> o = cell_level(N, i, K.g, K.h_dry, s_rate != nullptr);
        eta1[i] = o.eta;
        rp[i] = gd.rarea + R(1) / o.plan;
        if (o.wet) rate = rate > o.rate ? rate : o.rate;
    }
    if (s_rate) {
        for (int o = 16; o > 0; o >>= 1) {
            const R w = __shfl_xor_sync(0xffffffffu, rate, o);
            rate = w > rate ? w : rate;
        }
        if ((tid & 31) == 0) s_rate[tid >> 5] = rate;
    }
    const R dt = ready();
#pragma unroll
    for (int j = 0; j < S; ++j) {
        const int l = tid + j * nt;
        if (l < nl) V[l] = link_volume(eta1[c1[j]], zz[j] + hq[q2[j]], zb[j], len[j], rp[c1[j]], dt, K.cw, K.relax);
    }
    for (int l = tid + S * nt; l < nl; l += nt) {
        const int c = L.cell1d[l];
        V[l] = link_volume(eta1[c], z2(l) + hq[L.inv[l]], zbank(l), length(l), rp[c], dt, K.cw, K.relax);
    }
    sync();
    // donor limits, aggregated per donor in the caller's link order (coupling.py:98-107)
    auto limit2 = [&](int k, int one) {
        R tot = R(0);
        if (one >= 0) tot = pos_part(V[one]);
        else
            for (int j = L.ustart[k]; j < L.ustart[k + 1]; ++j) tot += pos_part(V[L.uidx[j]]);
        const R avail = K.limit * hq[k] * area;
        f2[k] = tot > avail ? avail / (tot > R(0) ? tot : R(1)) : R(1);
    };
#pragma unroll
    for (int j = 0; j < S; ++j)
        if (tid + j * nt < nu) limit2(tid + j * nt, u0[j]);
    for (int k = tid + S * nt; k < nu; k += nt) limit2(k, L.ufirst[k]);
    for (int i = tid; i < nc; i += nt) {
        R tot = R(0);
        for (int j = L.cstart[i]; j < L.cstart[i + 1]; ++j) tot += pos_part(-V[j]);
        const R avail = K.limit * (tot > R(0) ? cell_level(N, i, K.g, K.h_dry, false).avail : R(0));
        f1[i] = tot > avail ? avail / (tot > R(0) ? tot : R(1)) : R(1);
    }
    sync();
    R ex0 = R(0), ex1 = R(0);
    auto settle = [&](int l, int k, int c) {
        const R v0 = V[l], v = v0 > R(0) ? v0 * f2[k] : v0 * f1[c];
        V[l] = v;
        if (Vout) Vout[L.v_offset + L.orig[l]] = (double)v;
        ex0 += pos_part(v);
        ex1 += pos_part(-v);
    };
#pragma unroll
    for (int j = 0; j < S; ++j)
        if (tid + j * nt < nl) settle(tid + j * nt, q2[j], c1[j]);
    for (int l = tid + S * nt; l < nl; l += nt) settle(l, L.inv[l], L.cell1d[l]);
    if (!go()) return;
    // apply: 2-D through the unique cells, momentum kept only for water that stays (a cell
    // that gains and loses nothing keeps what it has)
    auto apply = [&](int k, int idx, int one) {
        R d = R(0);
        if (one >= 0) d = V[one];
        else
            for (int j = L.ustart[k]; j < L.ustart[k + 1]; ++j) d += V[L.uidx[j]];
        const R h0 = hq[k];
        if (d == R(0) && h0 > R(0)) return;
        R hn, keep;
        if constexpr (F32) {
            hn = h0 - d * gd.rarea;
            keep = h0 > 0.0f ? fminf(hn / h0, 1.0f) : 0.0f;
        } else {
            hn = h0 - d / area;
            keep = h0 > 0.0 ? fmin(hn / h0, 1.0) : 0.0;
        }
        gd.h[idx] = hn;
        gd.hu[idx] = gd.hu[idx] * keep;
        gd.hv[idx] = gd.hv[idx] * keep;
    };
#pragma unroll
    for (int j = 0; j < S; ++j)
        if (tid + j * nt < nu) apply(tid + j * nt, cell[j], u0[j]);
    for (int k = tid + S * nt; k < nu; k += nt) apply(k, L.uniq[k], L.ufirst[k]);
    for (int i = tid; i < nc; i += nt) {
        R d = R(0);
        for (int j = L.cstart[i]; j < L.cstart[i + 1]; ++j) d += V[j];
        if (d != R(0)) {
            if constexpr (F32) N.A[i] = N.A[i] + (double)(d / N.dxf[i]);
            else N.A[i] = N.A[i] + d / N.dx[i];
        }
    }
    if (!exch) return;
    // tallies in float64: lanes, then warps in order
    const double e0 = warp_sum_sparse((double)ex0), e1 = warp_sum_sparse((double)ex1);
    if ((tid & 31) == 0) {
        red[2 * (tid >> 5)] = e0;
        red[2 * (tid >> 5) + 1] = e1;
    }
    sync();
    if (tid < 2) {
        double a = red[tid];
        for (int w = 1; w < nt / 32; ++w) {
            const double b = red[2 * w + tid];
            if (f64_bits(b) << 1 != 0) a += b;
        }
        if (f64_bits(a) << 1 != 0) exch[mb * 2 + tid] += a;
    }
}

// One CTA of EXCHANGE_THREADS per member.  The drop-in step runs it alone between
// its CFL wait and the 2-D stages.
constexpr int EXCHANGE_THREADS = 512;

template <class R>
__global__ void __launch_bounds__(EXCHANGE_THREADS, sizeof(R) == 4 ? 2 : 1) exchange_kernel(const Lnk* __restrict__ links,
                                                                    const Net* __restrict__ nets,
                                                                    const Grid<R>* __restrict__ grids, ExchK<R> K, R dt,
                                                                    double* __restrict__ Vout,
                                                                    double* __restrict__ exch) {
    extern __shared__ double sm[];
    __shared__ Lnk L;
    __shared__ Net N;
    const int mb = blockIdx.x;
    stage_record(&L, links + mb);
    stage_record(&N, nets + mb);
    __syncthreads();
    exchange_dev<R>(L, N, grids[mb], K, Vout, exch, mb, sm, threadIdx.x, EXCHANGE_THREADS, nullptr,
                    [] { __syncthreads(); }, [&] { __syncthreads(); return dt; }, [] { __syncthreads(); return true; });
}

}  // namespace his
