// 1-D St. Venant network step (one CTA per member) and 1-D <-> 2-D weir exchange (one CTA per
// member, or a cluster of them).
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
    // products of the sections' constants: area at the bank, b^2, 4 m, sqrt(1 + m^2) and
    // 1 / dx of the cells; area and first moment at the bank, b / 2 and m / 3 of the faces
    const double *ab, *b2, *m4, *sp, *rdx;
    const double *fab, *fib, *fbh, *fm3;
    const int* ghosts;                             // the ghost cells (kinds 2 and up)
    int n_ghosts, pad;
    const float *zf, *dxf, *bf, *mf, *ybf, *tsf;   // float32 copies of z, dx and the cell sections
    const float *nmanf, *gsignf;                   // float32 roughness and ghost signs
    const float *fbf, *fmf, *fybf, *ftsf;          // float32 face sections
    double *A, *Q;
};

// CTAs that share the float64 exchange of one member
constexpr int EXCH_SLICES = 8;

struct Lnk {
    // Links in the order of their 1-D cell (within a cell in the caller's order), so that a
    // cell's links are contiguous; orig: the caller's index; cell2d: the 2-D cell
    int n_links, n_multi, v_offset, pad;
    const int *cell1d, *cell2d, *orig;
    const double *zbank, *length, *z2;
    const float *zbank_f, *length_f, *z2_f;        // float32 copies for the production form
    const int* cstart;                             // 1-D cell -> its links
    // Links that share their 2-D cell with others (n_multi of them): peer[l] is -1 for a link
    // alone on its cell, else the cell's entry in mstart, whose links midx lists in the caller's
    // order
    const int *peer, *mstart, *midx;
    // Slices of the 1-D cells (and with them of the links) for the CTAs of a cluster, of about
    // equal numbers of links
    int slice[EXCH_SLICES + 1], pad2;
};

// ---------------------------------------------------------------- sections (swe1d.py:51-84)
// Float64 geometry in few FP64 instructions (f64_ops.cuh): the products of a section's
// constants come from tables, and the wall above the bank is a branch that water below the
// bank does not take.  (Every quantity is >= 0, so comparisons are on the bit patterns.)
__device__ __forceinline__ bool f64_le(double a, double b) { return f64_bits(a) <= f64_bits(b); }   // a, b >= +0

__device__ __forceinline__ double cell_depth(const Net& N, int i, double A) {
    A = f64_clamp0(A);
    if (f64_bits(A) == 0) return 0.0;
    const double ab = N.ab[i];
    if (f64_le(A, ab)) return 2.0 * A / (N.b[i] + sqrt(fma(N.m4[i], A, N.b2[i])));
    return N.yb[i] + (A - ab) / N.ts[i];
}
__device__ __forceinline__ double cell_area(const Net& N, int i, double y) {
    const double yb = N.yb[i];
    return f64_le(y, yb) ? y * fma(N.m[i], y, N.b[i]) : fma(N.ts[i], y - yb, N.ab[i]);
}
__device__ __forceinline__ double cell_top(const Net& N, int i, double y) {
    return f64_le(y, N.yb[i]) ? fma(2.0 * N.m[i], y, N.b[i]) : N.ts[i];
}
__device__ __forceinline__ double cell_velocity(const Consts& c, double y, double A, double Q) {
    return f64_ge_pos(y, c.h_dry) ? Q / (f64_ge_pos(A, 1e-12) ? A : 1e-12) : 0.0;
}

// One side of a face: area, hydrostatic force and wave speed at depth y of its section
struct FaceSide {
    double A, p, c;
};
__device__ __forceinline__ FaceSide face_side(const Net& N, int f, double g, double y) {
    if (f64_bits(y) == 0) return FaceSide{0.0, 0.0, 0.0};
    const double yb = N.fyb[f], b = N.fb[f], m = N.fm[f];
    double A, I, top;
    if (f64_le(y, yb)) {
        A = y * fma(m, y, b);
        I = y * y * fma(N.fm3[f], y, N.fbh[f]);
        top = fma(2.0 * m, y, b);
    } else {
        const double above = y - yb, ts = N.fts[f], ab = N.fab[f];
        A = fma(ts, above, ab);
        I = N.fib[f] + above * fma(0.5 * ts, above, ab);
        top = ts;
    }
    return FaceSide{A, g * I, sqrt(g * A / top)};
}

// HLL flux of the 1-D equations (swe1d.py:87-107)
__device__ __forceinline__ void hll_1d(const FaceSide& L, double uL, const FaceSide& R, double uR, double& F1,
                                       double& F2) {
    const double tiny = 1e-14;
    const bool dryL = f64_le(L.A, tiny), dryR = f64_le(R.A, tiny);
    F1 = F2 = 0.0;
    if (dryL && dryR) return;
    double SL, SR;
    if (dryL) { SL = fma(-2.0, R.c, uR); SR = uR + R.c; }
    else if (dryR) { SL = uL - L.c; SR = fma(2.0, L.c, uL); }
    else {
        SL = f64_min(uL - L.c, uR - R.c);
        SR = f64_max(uL + L.c, uR + R.c);
    }
    const double QL = L.A * uL, QR = R.A * uR;
    if (f64_plus(SL)) {
        F1 = QL;
        F2 = fma(QL, uL, L.p);
    } else if (f64_minus(SR)) {
        F1 = QR;
        F2 = fma(QR, uR, R.p);
    } else {
        double den = SR - SL;
        if (f64_mag_lt(den, tiny)) den = 1.0;
        const double r = __drcp_rn(den), SS = SL * SR;
        const double mL = fma(QL, uL, L.p), mR = fma(QR, uR, R.p);
        F1 = fma(SS, R.A - L.A, fma(-SL, QR, SR * QL)) * r;
        F2 = fma(SS, QR - QL, fma(-SL, mR, SR * mL)) * r;
    }
}

// Largest wave rate (|u| + c) / dx of a wet interior cell, or -1 (swe1d.py:253-262)
__device__ __forceinline__ double cell_rate_1d(const Net& N, const Consts& c, int i, double y, double A, double Q) {
    if (N.kind[i] > 1 || !f64_ge_pos(y, c.h_dry) || f64_bits(y) == f64_bits(c.h_dry)) return -1.0;
    const double cc = sqrt(c.g * A / cell_top(N, i, y));
    return f64_div(fabs(cell_velocity(c, y, A, Q)) + cc, N.dx[i], N.rdx[i]);
}

// Deterministic block sum of NV doubles; result valid in thread 0.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = warp_sum_sparse(v[j]);
    if (lane == 0)
        for (int j = 0; j < NV; ++j) red[warp * NV + j] = v[j];
    __syncthreads();
    if (threadIdx.x == 0)
        for (int j = 0; j < NV; ++j) {
            double a = red[j];
            for (int w = 1; w < nw; ++w) {
                const double b = red[w * NV + j];
                if (f64_bits(b) << 1 != 0) a += b;
            }
            v[j] = a;
        }
    __syncthreads();
}

__host__ __device__ inline size_t net_smem_bytes(int n_cells, int n_faces) {
    return sizeof(double) * (5 * (size_t)n_cells + 4 * (size_t)n_faces + 32 * 4);
}

// Threads of a float64 network CTA: a warp for the ghosts beside those of the cells
constexpr int NET64_THREADS = 256;

// n_sub substeps of dt/n_sub each for the network N, run by the whole CTA (NET64_THREADS).
// forcing: per substep (inflow, stage).  vols (thread 0, if non-NULL): bnd_in,
// bnd_out, clip summed over the substeps.  sm: net_smem_bytes() of shared memory.
//
// Bound by one SM's FP64 pipe and by the length of the per-substep chain: ghosts, faces,
// limiter, update, with a barrier between.  The depth a cell's update needs for its
// friction is kept as the next substep's, the limiter's factors are applied where the
// fluxes are summed, and the tallies are summed once per call.  3170 -> 950 FP64 warp
// instructions per substep of 161 cells (two substeps with their CFL reduction through
// the solver class 299 -> 173 us).
__device__ __forceinline__ void net_substeps_dev(const Net& N, const Consts& c, double dt_total, int n_sub,
                                                 const double* __restrict__ forcing, double* vols, double* sm,
                                                 float* snap_eta = nullptr, float* snap_q = nullptr,
                                                 double* snap_v1d = nullptr) {
    const int nc = N.n_cells, nf = N.n_faces, tid = threadIdx.x, nt = blockDim.x;
    // A, Q: state, with the ghosts filled at the start of a substep; y, u: depth and velocity
    double *A = sm, *Q = A + nc, *yv = Q + nc, *uv = yv + nc, *th = uv + nc;
    double *F1 = th + nc, *F2 = F1 + nf, *pL = F2 + nf, *pR = pL + nf, *red = pR + nf;
    const double g = c.g, dt = dt_total / n_sub;
    for (int i = tid; i < nc; i += nt) {
        const double a = N.A[i], q = N.Q[i];
        A[i] = a;
        Q[i] = q;
        if (N.kind[i] < 2) {
            const double y = cell_depth(N, i, a);
            yv[i] = y;
            uv[i] = cell_velocity(c, y, a, q);
        }
    }
    __syncthreads();
    double bsum[3] = {0.0, 0.0, 0.0};
    for (int k = 0; k < n_sub; ++k) {
        const double q_in = forcing[2 * k + 0];
        const double eta = forcing[2 * k + 1];
        // ghost cells from the interior neighbour (swe1d.py:265-294)
        for (int j = tid; j < N.n_ghosts; j += nt) {
            const int i = N.ghosts[j], kd = N.kind[i], src = N.gsrc[i];
            const double As = A[src], Qs = Q[src], sg = N.gsign[i];
            const double ys = cell_depth(N, i, As);
            const bool wet_i = f64_ge_pos(ys, c.h_dry);
            double An, Qn, y;
            if (kd == 3) {
                const double un = sg * cell_velocity(c, ys, As, Qs);
                const double yst = f64_clamp0(eta - N.z[i]);
                double Ast = cell_area(N, i, yst), un_st = 0.0;
                y = cell_depth(N, i, Ast);
                if (wet_i) {
                    const double ci = sqrt(g * As / cell_top(N, i, ys));
                    const double cg = f64_bits(Ast) == 0 ? 0.0 : sqrt(g * Ast / cell_top(N, i, yst));
                    un_st = fma(2.0, ci - cg, un);
                    if (un > ci) {
                        un_st = un;
                        Ast = As;
                        y = ys;
                    }
                }
                if (!f64_ge_pos(y, c.h_dry)) un_st = 0.0;
                An = Ast;
                Qn = sg * Ast * un_st;
            } else if (kd == 2) {
                An = As;
                y = ys;
                if (!wet_i) {
                    const double yc = fmax(cbrt(q_in * q_in / (g * N.b[i] * N.b[i])), c.h_dry);
                    An = cell_area(N, i, yc);
                    y = cell_depth(N, i, An);
                }
                Qn = -sg * q_in;
            } else {
                An = As;
                y = ys;
                Qn = -Qs;
            }
            A[i] = An;
            Q[i] = Qn;
            yv[i] = y;
            uv[i] = cell_velocity(c, y, An, Qn);
        }
        __syncthreads();
        // face fluxes with hydrostatic reconstruction (swe1d.py:326-336)
        for (int f = tid; f < nf; f += nt) {
            const int l = N.fl[f], r = N.fr[f];
            const double zL = N.z[l], zR = N.z[r], zf = f64_max(zL, zR);
            const FaceSide L = face_side(N, f, g, f64_clamp0(zL + yv[l] - zf));
            const FaceSide R = face_side(N, f, g, f64_clamp0(zR + yv[r] - zf));
            pL[f] = L.p;
            pR[f] = R.p;
            hll_1d(L, uv[l], R, uv[r], F1[f], F2[f]);
        }
        __syncthreads();
        // outflow limiter; ghosts unlimited (swe1d.py:337-344)
        for (int i = tid; i < nc; i += nt) {
            double out = 0.0, t = 1.0;
            if (N.kind[i] < 2) {
                for (int j = N.lstart[i]; j < N.lstart[i + 1]; ++j) out += f64_relu(F1[N.lidx[j]]);
                for (int j = N.rstart[i]; j < N.rstart[i + 1]; ++j) out += f64_relu(-F1[N.ridx[j]]);
                const double vol = A[i] * N.dx[i], need = out * dt;
                if (need > vol) t = vol / (need > 0.0 ? need : 1.0);
            }
            th[i] = t;
        }
        __syncthreads();
        // update with the limited fluxes, clip, semi-implicit friction; ghosts keep their filled
        // state, and their faces carry the boundary volumes (swe1d.py:345-368)
        for (int i = tid; i < nc; i += nt) {
            const bool ghost = N.kind[i] >= 2;
            double dA = 0.0, dQ = 0.0;
            auto limited = [&](int f) {
                const double F = F1[f], t = th[f64_pos(F) ? N.fl[f] : N.fr[f]];
                return f64_bits(t) == f64_bits(1.0) ? F : F * t;
            };
            for (int j = N.lstart[i]; j < N.lstart[i + 1]; ++j) {
                const int f = N.lidx[j];
                const double F = limited(f);
                if (ghost) { bsum[0] += f64_relu(F); bsum[1] += f64_relu(-F); continue; }
                dA -= F;
                dQ -= F2[f] - pL[f];
            }
            for (int j = N.rstart[i]; j < N.rstart[i + 1]; ++j) {
                const int f = N.ridx[j];
                const double F = limited(f);
                if (ghost) { bsum[0] += f64_relu(-F); bsum[1] += f64_relu(F); continue; }
                dA += F;
                dQ += F2[f] - pR[f];
            }
            if (ghost) continue;
            const double dx = N.dx[i], rdx = N.rdx[i];
            double A1 = A[i] + f64_div(dt * dA, dx, rdx);
            double Q1 = Q[i] + f64_div(dt * dQ, dx, rdx);
            if (f64_neg(A1)) {
                bsum[2] -= A1 * dx;
                A1 = 0.0;
            }
            const double y1 = cell_depth(N, i, A1);
            if (f64_ge_pos(y1, c.h_dry) && N.kind[i] != 1) {
                if (f64_bits(Q1) << 1 != 0) {
                    // Q / (1 + dt g n^2 |Q| / (A R^(4/3))), as one quotient
                    const double yb = N.yb[i], Ac = f64_ge_pos(A1, 1e-12) ? A1 : 1e-12;
                    const double R = Ac / fma(2.0 * (f64_le(y1, yb) ? y1 : yb), N.sp[i], N.b[i]);
                    const double nm = N.nman[i], X = Ac * f64_pow43(f64_ge_pos(R, c.h_dry) ? R : c.h_dry);
                    Q1 = Q1 * (X / fma(dt * g * (nm * nm), fabs(Q1), X));
                }
            } else {
                Q1 = 0.0;
            }
            A[i] = A1;
            Q[i] = Q1;
            yv[i] = y1;
            uv[i] = cell_velocity(c, y1, A1, Q1);
        }
        __syncthreads();
    }
    bsum[0] *= dt;
    bsum[1] *= dt;
    block_sum<3>(bsum, red);
    for (int i = tid; i < nc; i += nt) { N.A[i] = A[i]; N.Q[i] = Q[i]; }
    if (snap_eta) {                         // output: level z + depth and discharge (coupling.py:229-242)
        double v1 = 0.0;
        for (int i = tid; i < nc; i += nt) {
            snap_eta[i] = (float)(N.z[i] + yv[i]);
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
        vols[0] = bsum[0];
        vols[1] = bsum[1];
        vols[2] = bsum[2];
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
            const float y = kind[i] == 1 ? (float)cell_depth(N, i, Ag[i]) : secf_depth(s, i, Af[i]);
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
            snap_eta[i] = (float)(N.z[i] + cell_depth(N, i, A[i]));
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

// Shared memory of the exchange of one slice: volumes per link, level (then limit) and
// storage per 1-D cell.
__host__ __device__ inline size_t exchange_smem_bytes(int n_links, int n_cells, size_t size) {
    return size * ((size_t)n_links + 2 * (size_t)n_cells);
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
    const double A = N.A[i], dx = N.dx[i];
    const double y = cell_depth(N, i, A), top = cell_top(N, i, y);
    o.eta = N.z[i] + y;
    o.plan = top * dx;
    o.avail = f64_clamp0(A - N.ab[i]) * dx;
    o.wet = rate && N.kind[i] <= 1 && f64_ge_pos(y, h_dry) && f64_bits(y) != f64_bits(h_dry);
    o.rate = o.wet ? f64_div(fabs(N.Q[i] / (f64_ge_pos(A, 1e-12) ? A : 1e-12)) + sqrt(g * A / top), dx, N.rdx[i]) : 0.0;
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

// Weir exchange of one member by nt threads (whole warps, this one tid) of a CTA, or of a
// slice of its 1-D cells and their links by one CTA of a cluster (coupling.py:73-124), with
// the 1-D CFL rate of the same cells.  float64 plain method; float32 in the production form
// (GB300's float64 pipe runs at a small fraction of the float32 rate), with the 1-D area
// update and the tallies in float64.
//
// In float32 it is a chain of dependent phases bound by the latency of their loads: what a
// thread needs of its links is fetched before the first barrier, for SLOTS links at
// once (more in a loop), a link alone on its 2-D cell limits and moves that cell's water
// itself, and a 1-D cell's sums walk its contiguous links in shared memory.  In float64 it is
// bound by FP64 instructions (powers, roots and quotients of every link that overtops; 4800
// per 400 x 325 member, 47 us of one SM's pipe), so EXCH_SLICES CTAs share a member: the
// pre-step of such a member 73 -> 25 us, a resident step of it 296 -> 253 us.
//
// sync: barrier of the nt threads.  wide: barrier of every thread of the member's CTAs.
// ready(): barrier with whoever chooses dt; returns it.  go(): barrier before the states are
// changed; false leaves them as they are.  Vg: volumes by position in global memory.
// put_rate (optional): takes each warp's largest rate of a wet cell, -1 where none is wet.
// SLOTS: links per thread fetched ahead (each costs registers).  s0, ns: the first of this CTA's
// slices and their number; tally: 2 values of its first slice.
template <class R, int SLOTS, class Sync, class Wide, class Ready, class Go, class Rate>
__device__ __forceinline__ void exchange_dev(const Lnk& L, const Net& N, const Grid<R>& gd, const ExchK<R>& K,
                                             double* __restrict__ Vout, double* Vg, double* __restrict__ tally,
                                             int s0, int ns, double* sm, int tid, int nt, bool rates, Sync sync,
                                             Wide wide, Ready ready, Go go, Rate put_rate) {
    constexpr int S = SLOTS;
    constexpr bool F32 = sizeof(R) == 4;
    const bool whole = ns == EXCH_SLICES;               // (a constant: this CTA has the whole member)
    const int c0 = whole ? 0 : L.slice[s0], l0 = whole ? 0 : L.cstart[c0];
    const int nc = whole ? N.n_cells : L.slice[s0 + ns] - c0, nl = whole ? L.n_links : L.cstart[c0 + nc] - l0;
    const R area = R(gd.area);
    R* V = reinterpret_cast<R*>(sm);
    R *eta1 = V + nl, *rp = eta1 + nc, *f1 = eta1;
    auto zbank = [&](int l) -> R { if constexpr (F32) return L.zbank_f[l]; else return L.zbank[l]; };
    auto length = [&](int l) -> R { if constexpr (F32) return L.length_f[l]; else return L.length[l]; };
    auto z2 = [&](int l) -> R { if constexpr (F32) return L.z2_f[l]; else return L.z2[l]; };

    const bool multi = L.n_multi > 0;
    int cell[S], at[S], peer[S];
    R zb[S], len[S], zz[S], hq[S];
#pragma unroll
    for (int j = 0; j < S; ++j) {
        const int k = tid + j * nt, l = l0 + k;
        cell[j] = at[j] = 0;
        peer[j] = -1;
        zb[j] = len[j] = zz[j] = hq[j] = R(0);
        if (k < nl) {
            cell[j] = L.cell1d[l] - c0;
            at[j] = L.cell2d[l];
            if (multi) peer[j] = L.peer[l];
            zb[j] = zbank(l);
            len[j] = length(l);
            zz[j] = z2(l);
        }
    }
#pragma unroll
    for (int j = 0; j < S; ++j)
        if (tid + j * nt < nl) hq[j] = gd.h[at[j]];
    R rate = R(-1);
    for (int i = tid; i < nc; i += nt) {
        const CellLevel<R> o = cell_level(N, c0 + i, K.g, K.h_dry, rates);
        eta1[i] = o.eta;
        rp[i] = gd.rarea + R(1) / o.plan;
        if (o.wet) rate = o.rate > rate ? o.rate : rate;
    }
    if (rates) {
        for (int o = 16; o > 0; o >>= 1) {
            const R w = __shfl_xor_sync(0xffffffffu, rate, o);
            rate = w > rate ? w : rate;
        }
        put_rate(rate);
    }
    const R dt = ready();
    // volumes before the limits
    auto volume = [&](int k, int c, R h, R zbk, R ln, R zk, int p) {
        const R v = link_volume(eta1[c], zk + h, zbk, ln, rp[c], dt, K.cw, K.relax);
        V[k] = v;
        if (p >= 0) Vg[l0 + k] = (double)v;
    };
#pragma unroll
    for (int j = 0; j < S; ++j)
        if (tid + j * nt < nl) volume(tid + j * nt, cell[j], hq[j], zb[j], len[j], zz[j], peer[j]);
    for (int k = tid + S * nt; k < nl; k += nt) {
        const int l = l0 + k;
        volume(k, L.cell1d[l] - c0, gd.h[L.cell2d[l]], zbank(l), length(l), z2(l), L.peer[l]);
    }
    if (multi) wide();
    sync();
    // donor limits, aggregated per donor in the caller's link order (coupling.py:98-107); a
    // 2-D donor's limit is formed by each of its links
    for (int i = tid; i < nc; i += nt) {
        R tot = R(0);
        for (int j = L.cstart[c0 + i] - l0; j < L.cstart[c0 + i + 1] - l0; ++j) tot += pos_part(-V[j]);
        const R avail = K.limit * (tot > R(0) ? cell_level(N, c0 + i, K.g, K.h_dry, false).avail : R(0));
        f1[i] = tot > avail ? avail / (tot > R(0) ? tot : R(1)) : R(1);
    }
    auto limit2 = [&](R v, R h, int p) -> R {
        R tot = pos_part(v);
        if (p >= 0) {
            tot = R(0);
            for (int j = L.mstart[p]; j < L.mstart[p + 1]; ++j) tot += pos_part((R)Vg[L.midx[j]]);
        }
        const R avail = K.limit * h * area;
        return tot > avail ? v * (avail / (tot > R(0) ? tot : R(1))) : v;
    };
    sync();
    auto settle = [&](int k, int c, R h, int p) {
        R v = V[k];
        v = v > R(0) ? limit2(v, h, p) : v * f1[c];
        return v;
    };
    auto keep_v = [&](int k, R v, int p) {
        V[k] = v;
        if (p >= 0) Vg[l0 + k] = (double)v;
        if (Vout) Vout[L.v_offset + L.orig[l0 + k]] = (double)v;
    };
    R vs[S];
#pragma unroll
    for (int j = 0; j < S; ++j)
        if (tid + j * nt < nl) vs[j] = settle(tid + j * nt, cell[j], hq[j], peer[j]);
    for (int k = tid + S * nt; k < nl; k += nt) V[k] = settle(k, L.cell1d[l0 + k] - c0, gd.h[L.cell2d[l0 + k]], L.peer[l0 + k]);
    if (multi) wide();                                  // shared volumes are read before they change
#pragma unroll
    for (int j = 0; j < S; ++j)
        if (tid + j * nt < nl) keep_v(tid + j * nt, vs[j], peer[j]);
    for (int k = tid + S * nt; k < nl; k += nt) keep_v(k, V[k], L.peer[l0 + k]);
    if (multi) wide();
    if (!go()) return;
    // apply: 2-D cells, momentum kept only for water that stays (a cell that gains and loses
    // nothing keeps what it has); a shared cell by the first of its links
    auto mine = [&](int k, int p) { return p < 0 || L.midx[L.mstart[p]] == l0 + k; };
    auto apply = [&](int k, int idx, int p, R h0) {
        R d = V[k];
        if (p >= 0) {
            d = R(0);
            for (int j = L.mstart[p]; j < L.mstart[p + 1]; ++j) d += (R)Vg[L.midx[j]];
        }
        if (d == R(0) && h0 > R(0)) return;
        R hn, keep;
        if constexpr (F32) {
            hn = h0 - d * gd.rarea;
            keep = h0 > 0.0f ? fminf(hn / h0, 1.0f) : 0.0f;
        } else {
            hn = h0 - f64_div(d, area, gd.rarea);
            keep = h0 > 0.0 ? f64_min(hn / h0, 1.0) : 0.0;
        }
        gd.h[idx] = hn;
        gd.hu[idx] = gd.hu[idx] * keep;
        gd.hv[idx] = gd.hv[idx] * keep;
    };
#pragma unroll
    for (int j = 0; j < S; ++j)
        if (tid + j * nt < nl && mine(tid + j * nt, peer[j])) apply(tid + j * nt, at[j], peer[j], hq[j]);
    for (int k = tid + S * nt; k < nl; k += nt) {
        const int p = L.peer[l0 + k], idx = L.cell2d[l0 + k];
        if (mine(k, p)) apply(k, idx, p, gd.h[idx]);
    }
    for (int i = tid; i < nc; i += nt) {
        const int c = c0 + i;
        R d = R(0);
        for (int j = L.cstart[c] - l0; j < L.cstart[c + 1] - l0; ++j) d += V[j];
        if (d != R(0)) {
            if constexpr (F32) N.A[c] = N.A[c] + (double)(d / N.dxf[c]);
            else N.A[c] = N.A[c] + f64_div(d, N.dx[c], N.rdx[c]);
        }
    }
    // Tallies, a warp to a slice: lane l takes the slice's links l, l + 32, ..., four at a time in R,
    // then in float64, and the lanes by a shuffle tree, so that a member's totals do not depend
    // on how many CTAs share it.
    const int w = tid >> 5, lane = tid & 31;
    if (w >= ns) return;
    const int a = L.cstart[L.slice[s0 + w]] - l0, b = L.cstart[L.slice[s0 + w + 1]] - l0;
    double e0 = 0.0, e1 = 0.0;
    for (int k = a; k < b; k += 128) {
        R x0 = R(0), x1 = R(0);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int q = k + 32 * j + lane;
            const R v = q < b ? V[q] : R(0);
            // (float64: a sum that gets nothing costs a vote)
            if (F32 || __any_sync(0xffffffffu, pos_part(v) != R(0))) x0 += pos_part(v);
            if (F32 || __any_sync(0xffffffffu, pos_part(-v) != R(0))) x1 += pos_part(-v);
        }
        if (__any_sync(0xffffffffu, x0 != R(0))) e0 += (double)x0;
        if (__any_sync(0xffffffffu, x1 != R(0))) e1 += (double)x1;
    }
    e0 = warp_sum_sparse(e0);
    e1 = warp_sum_sparse(e1);
    if (lane == 0) {
        if (f64_bits(e0) << 1 != 0) tally[2 * w] += e0;
        if (f64_bits(e1) << 1 != 0) tally[2 * w + 1] += e1;
    }
}

// Barrier of every thread of a member's CTAs
template <int G>
__device__ __forceinline__ void member_sync(int threads) {
    if constexpr (G > 1) {
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    } else {
        bar_group(1, threads);
    }
}

// The drop-in step runs the exchange alone between its CFL wait and the 2-D stages.
constexpr int EXCHANGE_THREADS = 512;

template <class R, int G>
__global__ void __cluster_dims__(G, 1, 1) __launch_bounds__(EXCHANGE_THREADS, sizeof(R) == 4 ? 2 : 1)
exchange_kernel(const Lnk* __restrict__ links, const Net* __restrict__ nets, const Grid<R>* __restrict__ grids,
                ExchK<R> K, R dt, double* __restrict__ Vout, double* Vg, double* __restrict__ exch) {
    extern __shared__ double sm[];
    __shared__ Lnk L;
    __shared__ Net N;
    const int mb = blockIdx.x / G, rank = blockIdx.x % G;
    stage_record(&L, links + mb);
    stage_record(&N, nets + mb);
    __syncthreads();
    constexpr int NS = EXCH_SLICES / G;             // slices of this CTA
    static_assert(NS * G == EXCH_SLICES && EXCHANGE_THREADS / 32 >= NS, "whole slices, a warp to each");
    auto sync = [] { __syncthreads(); };
    exchange_dev<R, G == 1 ? 3 : 1>(L, N, grids[mb], K, Vout, Vg + L.v_offset,
                    exch + (size_t)(mb * EXCH_SLICES + rank * NS) * 2, rank * NS, NS, sm, threadIdx.x,
                    EXCHANGE_THREADS, false, sync, [] { member_sync<G>(EXCHANGE_THREADS); },
                    [&] { __syncthreads(); return dt; }, [] { __syncthreads(); return true; }, [](R) {});
}

}  // namespace his
