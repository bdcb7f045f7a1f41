// 2-D finite-volume step kernels of the float32 production form: row-marching strips
// (the float64 method's are in swe2d_tile64.cuh), and the per-strip-chunk reductions of
// both precisions.
//
// A CTA of NT threads owns a strip of W <= NT - 6 columns of one member and marches
// up a chunk of rows [y0, y1).  Thread t works on column cx = x0 - 3 + t.  Per new
// row r, with two barriers (StripPipe::row below):
//   A  builds row r of (h, u, v, z) into a four-row shared ring (ghost cells at the
//      domain edges, boundaries.py:81-128), prefetches row r+1 and the update inputs
//      of row r-3, forms the y-reconstruction of row r-1 and the x-reconstruction of
//      row r-2 (swe2d.py:205-219) and publishes the latter's plus side;
//   B  forms the y-face between rows r-2 and r-1 and the x-face west of its cell in
//      row r-2 (swe2d.py:61-101, 226-234), two independent chains side by side;
//   C  forms the positivity-limiter theta of row r-2 (swe2d.py:259-264);
//   D  updates row r-3: divergence of the donor-scaled fluxes, bed source, RK stage,
//      then in the last stage rain, infiltration, retention, friction, CFL rate and
//      peaks (swe2d.py:305-371).
// Every cell is loaded once (plus a 3-column halo each side) and every face flux,
// reconstruction and theta is computed once.  Per-thread partial sums (clip,
// boundary flux, infiltration, rain, rate, volumes) are reduced once per strip-chunk
// into one float64 slot set, summed in a fixed order per member by the finalize
// kernel: states and rates do not depend on the batch a member runs in, its totals only
// through the decomposition, where that is left to the library (default_tile).
#pragma once
#include "his_device.cuh"

namespace his {

struct StripRef {
    int member, x0, w, y0, y1;
    short sub_w, sub_h;              // float64: largest sub-tile (swe2d_tile64.cuh)
};

// Four values of one cell or face kept together in shared memory, so that one
// vector access moves them: cells {h, u, v, z}, faces {F1, F2L, F2R, F3}, and the
// plus side of the x-reconstruction.
template <class R>
struct alignas(4 * sizeof(R)) Q4 {
    R a, b, c, d;
};

// Shared-memory layout of one CTA.  Rings of the last rows' cells, x- and y-faces and
// thetas: a thread publishes each value once and reads both its neighbours' entries
// and its own earlier rows from them, so no row-to-row state is shifted through
// registers.  Every row of entries has one padding slot on each side: thread t's
// entry is at t + 1, so the neighbours of the first and last thread are in bounds
// (their values are never used).
template <class R, int NT>
struct StripGeom {
    static constexpr int RING = 4;                 // rows kept per ring (slot = row & 3)
    static constexpr int P = NT + 2;               // padded row of entries
    static constexpr int NRED = 11;                // reduced values (the reduction reuses the cell ring)
    // cells [RING][P], x-recon plus side [P], x-faces [2][P], y-faces [RING][P]; then
    // the plus-side surface slope [P], theta [RING][P] and two old peaks [2][P]
    static constexpr size_t quads = (size_t)(RING + 1 + 2 + RING) * P;
    static constexpr size_t scalars = (size_t)(1 + RING + 2) * P;
    static_assert((size_t)4 * RING * P >= (size_t)(NT / 32) * NRED, "reduction scratch must fit in the cell ring");
    static constexpr size_t smem_bytes = sizeof(Q4<R>) * quads + sizeof(R) * scalars;
    // resident CTAs per SM the kernels are register-capped for (a chunk marched in segments:
    // few of them share an SM)
    static constexpr int min_ctas(int stage, int seg) {
        const int threads = seg > 1 ? 512 : stage == 1 ? 768 : 640;
        return threads / (NT * seg) > 0 ? threads / (NT * seg) : 1;
    }
    // a chunk marched in segments: each segment's rings, then every row's sums per thread
    // (SegSums) and every segment's maxima
    static constexpr int NSUM = 9, NMAX = 2;
    static constexpr size_t seg_stride = (smem_bytes + 31) / 32 * 32;
    static constexpr size_t seg_smem(int seg, int rows) {
        return seg * seg_stride + sizeof(R) * NT * ((size_t)rows * NSUM + (size_t)seg * NMAX);
    }
};

// Centred bed source of one cell along one axis (swe2d.py:220): -g/2 (H- + H+)(Z+ - Z-)
// with Z+ - Z- replaced by the in-cell surface slope (the hydrostatic part of the face
// momentum fluxes is carried by riemann_wb) and H- + H+ = 2 h.  The row loop computes it
// where the reconstruction is formed and carries it in registers to the update of that
// cell.
__device__ __forceinline__ float bed_term(const KC<float>& c, const Recon& r) { return -2.0f * c.g * r.h0 * r.sE; }

// One halo position: an interior cell, or the ghost that the x-sweep (outside in x)
// or the y-sweep (outside in y) would see (boundaries.py:81-128), in two parts for
// software pipelining: halo_fetch issues the loads of the source cell (the cell
// itself, or the layer a ghost copies) rows ahead; halo_build turns the fetched raw
// values into (h, u, v, z) when the row is due.
template <class R>
struct HaloRaw {
    R h, hu, hv, z;
};

template <class R>
__device__ __forceinline__ HaloRaw<R> halo_fetch(const KC<R>& c, const Grid<R>& gd, const R* __restrict__ H,
                                                 const R* __restrict__ HU, const R* __restrict__ HV, int gx, int gy) {
    const int nx = gd.nx, ny = gd.ny;
    const bool inx = (unsigned)gx < (unsigned)nx, iny = (unsigned)gy < (unsigned)ny;
    HaloRaw<R> a;
    if (!inx && !iny) { a.h = a.hu = a.hv = a.z = R(0); return a; }
    // 32-bit cell indices (a grid holds at most 2^30 cells): one wide multiply-add forms
    // each address
    unsigned i;
    if (inx && iny) {
        i = (unsigned)gy * (unsigned)nx + (unsigned)gx;
    } else {
        const int ng = c.order == 1 ? 1 : 2;
        const bool alongx = !inx;
        const int n = alongx ? nx : ny;
        const int gpos = alongx ? gx : gy;
        const bool lo = gpos < 0;
        const int side = alongx ? (lo ? EDGE_W : EDGE_E) : (lo ? EDGE_S : EDGE_N);
        const int k = lo ? (-gpos - 1) : (gpos - n);
        const int kind = gd.bc[side];
        int layer;
        if (kind == BC_CLOSED || kind == BC_TRANSMISSIVE) {
            if (n < ng) layer = lo ? 0 : n - 1;
            else layer = lo ? k : n - 1 - k;
        } else {
            layer = lo ? 0 : n - 1;
        }
        layer = layer < 0 ? 0 : (layer > n - 1 ? n - 1 : layer);
        i = alongx ? (unsigned)gy * (unsigned)nx + (unsigned)layer : (unsigned)layer * (unsigned)nx + (unsigned)gx;
    }
    a.h = H[i];
    a.hu = HU[i];
    a.hv = HV[i];
    a.z = gd.z[i];
    return a;
}

template <class R>
__device__ __forceinline__ void halo_build(const KC<R>& c, const Grid<R>& gd, const R* bcv, const HaloRaw<R>& a,
                                           int gx, int gy, R& hh, R& uu, R& vv, R& zz) {
    const int nx = gd.nx, ny = gd.ny;
    const bool inx = (unsigned)gx < (unsigned)nx, iny = (unsigned)gy < (unsigned)ny;
    if (!inx && !iny) { hh = uu = vv = zz = R(0); return; }
    R u0, v0;
    kp_velocity(c, a.h, a.hu, a.hv, u0, v0);
    zz = a.z;
    if (inx && iny) { hh = a.h; uu = u0; vv = v0; return; }
    const bool alongx = !inx;
    const int n = alongx ? nx : ny;
    const int gpos = alongx ? gx : gy;
    const bool lo = gpos < 0;
    const int side = alongx ? (lo ? EDGE_W : EDGE_E) : (lo ? EDGE_S : EDGE_N);
    const int kind = gd.bc[side];
    (void)n;
    const R sgn = lo ? R(-1) : R(1);
    R un = sgn * (alongx ? u0 : v0);
    R ut = alongx ? v0 : u0;
    R hg, ung, utg;
    if (kind == BC_CLOSED) { hg = a.h; ung = -un; utg = ut; }
    else if (kind == BC_TRANSMISSIVE) { hg = a.h; ung = un; utg = ut; }
    else if (kind == BC_STAGE) stage_ghost(c, bcv[side], a.h, un, ut, a.z, hg, ung, utg);
    else discharge_ghost(c, bcv[side], a.h, hg, ung, utg);
    hh = hg;
    if (alongx) { uu = sgn * ung; vv = utg; }
    else { vv = sgn * ung; uu = utg; }
}

// Per-cell inputs of the update (row orow), fetched one row ahead.
template <class R>
struct CellIn {
    R h0, hu0, hv0, hu1, hv1, sf, ic, f0, fc, k, S, n, rw;
};

// Optional fields of a member, tested once per CTA: the row loop reads a bit of a
// register instead of re-reading a 64-bit pointer from the shared record and
// comparing it with null.
enum : unsigned { FEAT_STORE = 1u, FEAT_HORTON = 2u, FEAT_RAINW = 4u, FEAT_PEAK = 8u, FEAT_PSPEED = 16u, FEAT_SNAP = 32u,
                  FEAT_PEAKS = FEAT_PEAK | FEAT_PSPEED };
template <class R>
__device__ __forceinline__ unsigned grid_features(const Grid<R>& gd) {
    return (gd.S ? FEAT_STORE : 0u) | (gd.f0 ? FEAT_HORTON : 0u) | (gd.rw ? FEAT_RAINW : 0u) |
           (gd.pk ? FEAT_PEAK : 0u) | (gd.ps ? FEAT_PSPEED : 0u);
}

template <class R, int STAGE>
__device__ __forceinline__ CellIn<R> cell_fetch(const Grid<R>& gd, unsigned i, unsigned feat) {
    CellIn<R> a;
    a.hu0 = gd.hu[i];
    a.hv0 = gd.hv[i];
    if (STAGE == 2) {
        a.h0 = gd.h[i];
        a.hu1 = gd.hu1[i];
        a.hv1 = gd.hv1[i];
    } else {
        a.h0 = a.hu1 = a.hv1 = R(0);
    }
    if (STAGE != 1) {
        const bool hs = feat & FEAT_STORE, hf = feat & FEAT_HORTON;
        a.sf = hs ? gd.sf[i] : R(0);
        a.S = hs ? gd.S[i] : R(0);
        a.ic = hf ? gd.ic[i] : R(0);
        a.f0 = hf ? gd.f0[i] : R(0);
        a.fc = hf ? gd.fc[i] : R(0);
        a.k = hf ? gd.k[i] : R(0);
        a.n = gd.n[i];
        a.rw = (feat & FEAT_RAINW) ? gd.rw[i] : R(0);
    } else {
        a.sf = a.S = a.ic = a.f0 = a.fc = a.k = a.n = a.rw = R(0);
    }
    return a;
}

template <class T>
__device__ __forceinline__ T warp_sum_t(T v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
template <class T>
__device__ __forceinline__ T warp_max_t(T v) {
    for (int o = 16; o > 0; o >>= 1) {
        T w = __shfl_down_sync(0xffffffffu, v, o);
        v = w > v ? w : v;
    }
    return v;
}

// Block reduction of NV per-thread values in the compute type T (warps by shuffles,
// then lane j of warp 0 over the warps in order), one float64 store per value.
template <int NV, class T>
__device__ __forceinline__ void block_reduce_store(T (&v)[NV], const bool* is_max, T* red, double* out,
                                                   const int* slots, int nthreads) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = nthreads >> 5;
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = is_max[j] ? warp_max_t(v[j]) : warp_sum_t(v[j]);
    if (lane == 0 && warp < nw) {
#pragma unroll
        for (int j = 0; j < NV; ++j) red[warp * NV + j] = v[j];
    }
    __syncthreads();
    if (warp == 0 && lane < NV) {
        const bool mx = is_max[lane];
        T a = red[lane];
        for (int w = 1; w < nw; ++w) {
            const T b = red[w * NV + lane];
            a = mx ? (b > a ? b : a) : a + b;
        }
        out[slots[lane]] = (double)a;
    }
}

// A running peak's old value on its way to shared memory, and the wait for it
__device__ __forceinline__ void peak_fetch(float* s, const float* p) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(p)
                 : "memory");
}
__device__ __forceinline__ void peak_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One side of a reconstructed cell as a face sees it: depth, normal and tangential
// velocity, X = the in-cell bed slope d and S = the in-cell surface slope sE.  The cell's
// own bed z and depth h0 (the flux's difference form) come with the cell record.
struct Side {
    float H, U, V, X, S;
};
__device__ __forceinline__ Side side_plus(const Recon& r) { return Side{r.Hp, r.Up, r.Vp, r.d, r.sE}; }
__device__ __forceinline__ Side side_minus(const Recon& r) { return Side{r.Hm, r.Um, r.Vm, r.d, r.sE}; }

// Face flux from the plus side of the cell below / west of the face (bed zl, depth hl)
// and the minus side of the cell above / east of it: face_flux's arithmetic exactly.
__device__ __forceinline__ Q4<float> side_flux(const KC<float>& c, const Side& L, float zl, float hl, const Side& Rt,
                                               float zr, float hr) {
    Recon a, b;
    a.Hp = L.H; a.Up = L.U; a.Vp = L.V;
    b.Hm = Rt.H; b.Um = Rt.U; b.Vm = Rt.V;
    a.d = L.X; a.sE = L.S; a.z = zl; a.h0 = hl;
    b.d = Rt.X; b.sE = Rt.S; b.z = zr; b.h0 = hr;
    Q4<float> f;
    face_flux(c, a, b, f.a, f.b, f.c, f.d);
    return f;
}

// The row-marching pipeline of one strip chunk (see the head of this file).  Row r is
// the newest row built; per row two barriers separate the phases:
//   A  build row r into the cell ring, prefetch row r+1 and the update inputs of row
//      r-3; y-reconstruction of row r-1 and the y-face between rows r-2 and r-1;
//      x-reconstruction of row r-2 from its neighbours' cells, plus side published
//   -- barrier --
//   B  x-face between columns cx-1 and cx of row r-2, published
//   -- barrier --
//   C  theta of row r-2, published
//   D  update of row r-3 from the rings' entries of rows r-4 .. r-2
// row<true> is the steady state: every row touched lies inside the grid, so the
// range tests, y-ghosts and domain-edge terms drop out; row<false> handles the
// pipeline fill at the chunk's start, the drain at its end and the grid's edges.
//
// SEG > 1: the chunk's rows are dealt to SEG groups of NT threads, which march side by side,
// each with its own rings and barrier; the rows' contributions to the partial sums are kept
// per row and thread and added up in row order at the end, so that the sums are those of one
// march over all rows, bit for bit.  (But where a thread adds twice to a sum in a row, the terms
// of a column that is both the west and the east edge: strip_segments marches sets with such
// members in one.)
//
// PEAKS: some member of the set has running peaks (a kernel without their code takes 5251 us for
// 16 steps of 64 storms of 400 x 325 cells, one that tests for them in every row 5285).
template <class R, int NT, int STAGE, int SEG, bool PEAKS>
struct StripPipe {
    static_assert(sizeof(R) == 4, "the float64 step is tile64_kernel's");
    using G = StripGeom<R, NT>;
    static constexpr int P = G::P;
    static constexpr int RM = G::RING - 1;
    Q4<R>* s_cell;
    Q4<R>* s_rp;
    Q4<R>* s_xf;
    Q4<R>* s_yf;
    R* s_rs;
    R* s_th;
    const Grid<R>& gd;
    const KC<R>& c;
    const R* bcv;
    float* const* s_snap;
    const R* __restrict__ H;
    const R* __restrict__ HU;
    const R* __restrict__ HV;
    int ts, cx, cxc, nx, ny, cy0, y0, y1, scol, xside, xkind;      // cy0: the chunk's first row; [y0, y1) this march
    unsigned feat;                     // FEAT_* bits of the member's optional fields
    bool col_in, do_out, west, east;
    R dt, hdt, idx, idy, rdt, tt;
    // carried state of this thread's column
    HaloRaw<R> ra;                     // raw row r (prefetched one row ahead)
    Side ylow;                      // plus side of the y-reconstruction of row r-2
    R by1, by2, bx1;                   // bed terms: y of rows r-2, r-3; x of row r-3
    CellIn<R> cin;
    R old_pk, old_ps;                  // PEAKS: row r-3's running peaks
    R acc_clip, xin, xout, yin, yout, infil, rainw, rate, hsum, ssum, hmax;
    R* sums;                           // SEG > 1: this thread's entry of the chunk's first row
    int bar;                           // and its segment's barrier

    // Barrier among the NT threads of one march
    __device__ __forceinline__ void sync() const {
        if (SEG == 1) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(NT) : "memory");
    }
    // Row's contributions to the sums, put aside (SEG > 1)
    __device__ __forceinline__ void put_sums(int row) {
        R* s = sums + (size_t)row * (G::NSUM * NT);
        R* const v[G::NSUM] = {&acc_clip, &xin, &xout, &yin, &yout, &infil, &rainw, &hsum, &ssum};
#pragma unroll
        for (int k = 0; k < (STAGE == 1 ? 5 : G::NSUM); ++k) {
            s[k * NT] = *v[k];
            *v[k] = R(0);
        }
    }
    // All rows' contributions added in row order
    __device__ __forceinline__ void take_sums(int rows) {
        R* const v[G::NSUM] = {&acc_clip, &xin, &xout, &yin, &yout, &infil, &rainw, &hsum, &ssum};
        for (int j = 0; j < rows; ++j) {
            const R* s = sums + (size_t)j * (G::NSUM * NT);
#pragma unroll
            for (int k = 0; k < (STAGE == 1 ? 5 : G::NSUM); ++k) *v[k] += s[k * NT];
        }
    }

    // The running peaks of cell i before this step, fetched with the row's other inputs: into
    // registers where segments, few warps to an SM, have some to spare, else into shared memory
    // (16 steps of 64 storms with both peaks 5470 us; loaded by the update 6450; an integer
    // maximum in L2, which keeps a NaN for good, 5340.  Six served storms: 850
    // and 850 us by either).
    __device__ __forceinline__ void peaks_fetch(unsigned i) {
        if (SEG > 1) {
            if (feat & FEAT_PEAK) old_pk = gd.pk[i];
            if (feat & FEAT_PSPEED) old_ps = gd.ps[i];
        } else {
            R* s = s_th + G::RING * P + ts;
            if (feat & FEAT_PEAK) peak_fetch(s, gd.pk + i);
            if (feat & FEAT_PSPEED) peak_fetch(s + P, gd.ps + i);
        }
    }
    // Raised, from any start (fmaxf: NaN on either side gives way)
    __device__ __forceinline__ void peaks_raise(unsigned i, R h, R speed) {
        const R* s = s_th + G::RING * P + ts;
        if (SEG == 1) peak_wait();
        if (feat & FEAT_PEAK) gd.pk[i] = fmaxf(SEG > 1 ? old_pk : s[0], h);
        if (feat & FEAT_PSPEED) gd.ps[i] = fmaxf(SEG > 1 ? old_ps : s[P], speed);
    }
    // Raw values of an interior row at this thread's source column (its own column, or
    // the layer an x-ghost copies)
    __device__ __forceinline__ HaloRaw<R> fetch_in(int gy) const {
        const unsigned i = (unsigned)gy * (unsigned)nx + (unsigned)scol;
        return HaloRaw<R>{H[i], HU[i], HV[i], gd.z[i]};
    }
    // halo_build for a row inside the grid: an interior cell, or the x-ghost that the
    // x-sweep would see (boundaries.py:81-128)
    __device__ __forceinline__ Q4<R> build_in(const HaloRaw<R>& a) const {
        R u0, v0;
        kp_velocity(c, a.h, a.hu, a.hv, u0, v0);
        if (xkind < 0) return Q4<R>{a.h, u0, v0, a.z};
        const R sgn = xside == EDGE_W ? R(-1) : R(1);
        const R un = sgn * u0, ut = v0;
        R hg, ung, utg;
        if (xkind == BC_CLOSED) { hg = a.h; ung = -un; utg = ut; }
        else if (xkind == BC_TRANSMISSIVE) { hg = a.h; ung = un; utg = ut; }
        else if (xkind == BC_STAGE) stage_ghost(c, bcv[xside], a.h, un, ut, a.z, hg, ung, utg);
        else discharge_ghost(c, bcv[xside], a.h, hg, ung, utg);
        return Q4<R>{hg, sgn * ung, utg, a.z};
    }

    template <bool FULL>
    __device__ __forceinline__ void row(const int r) {
        const int k0 = (r & RM) * P, k1 = ((r - 1) & RM) * P, k2 = ((r - 2) & RM) * P, k3 = ((r - 3) & RM) * P,
                  k4 = ((r - 4) & RM) * P;
        const int xo = ((r - 2) & 1) * P, xp = ((r - 3) & 1) * P;
        const int orow = r - 3, row = r - 2;
        const bool upd = FULL || (orow >= y0 && orow < y1);
        // ---- A: row r, prefetches, y-face r-1, x-reconstruction of row r-2
        Q4<R> c0;
        if (FULL) {
            c0 = build_in(ra);
        } else {
            halo_build(c, gd, bcv, ra, cx, r, c0.a, c0.b, c0.c, c0.d);
        }
        s_cell[k0 + ts] = c0;
        ra = FULL ? fetch_in(r + 1) : halo_fetch(c, gd, H, HU, HV, cx, r + 1);
        if (upd) {
            const unsigned i = (unsigned)orow * (unsigned)nx + (unsigned)cxc;
            cin = cell_fetch<R, STAGE>(gd, i, feat);
            if (PEAKS && (feat & FEAT_PEAKS)) peaks_fetch(i);
        }
        R by0 = R(0), bx0 = R(0);
        const Q4<R> c2 = s_cell[k2 + ts];           // own cells of rows r-2 and r-1
        const Q4<R> c1 = s_cell[k1 + ts];
        // y-reconstruction of row r-1 (normal velocity v, tangential u); its face with
        // row r-2 is formed in phase B beside the x-face, two independent chains
        const bool yact = FULL || r >= y0 - 1;
        Side ylo = ylow, yum;
        if (yact) {
            const Recon yup = reconstruct(c, c2.a, c1.a, c0.a, c2.c, c1.c, c0.c, c2.b, c1.b, c0.b, c2.d, c1.d, c0.d);
            yum = side_minus(yup);
            ylow = side_plus(yup);
            if (c.order == 2) by0 = bed_term(c, yup);
        }
        const bool xact = FULL || (r >= y0 + 1 && (unsigned)row < (unsigned)ny);
        Q4<R> cl;
        Side xm;
        if (xact) {
            cl = s_cell[k2 + ts - 1];
            const Q4<R> cr = s_cell[k2 + ts + 1];
            const Recon xr = reconstruct(c, cl.a, c2.a, cr.a, cl.b, c2.b, cr.b, cl.c, c2.c, cr.c, cl.d, c2.d, cr.d);
            const Side xp_ = side_plus(xr);
            s_rp[ts] = Q4<R>{xp_.H, xp_.U, xp_.V, xp_.X};
            s_rs[ts] = xp_.S;
            xm = side_minus(xr);
            if (c.order == 2) bx0 = bed_term(c, xr);
        }
        sync();
        // ---- B: y-face between rows r-2 and r-1; x-face between columns cx-1 and cx of row r-2
        Q4<R> yf0{R(0), R(0), R(0), R(0)};
        if (yact) {
            const int fy = r - 1;
            if (FULL || (r >= y0 && fy >= 0 && fy <= ny)) yf0 = side_flux(c, ylo, c2.d, c2.a, yum, c1.d, c1.a);
            if (FULL || r >= y0) s_yf[k1 + ts] = yf0;
        }
        Q4<R> xf0{R(0), R(0), R(0), R(0)};
        if (xact) {
            const Q4<R> lp = s_rp[ts - 1];
            const Side L{lp.a, lp.b, lp.c, lp.d, s_rs[ts - 1]};
            xf0 = side_flux(c, L, cl.d, cl.a, xm, c2.d, c2.a);
            s_xf[xo + ts] = xf0;
        }
        sync();
        // ---- C: theta of row r-2 (swe2d.py:259-264); 1 outside the grid
        R th0 = R(1);
        Q4<R> yn{R(0), R(0), R(0), R(0)};          // y-face r-2: south of row r-2, north of row r-3
        if (FULL || r >= y0 + 1) {
            yn = s_yf[k2 + ts];
            if (FULL || (unsigned)row < (unsigned)ny) {
                const R Fw = xf0.a, Fe = s_xf[xo + ts + 1].a, Gs = yn.a, Gn = yf0.a;
                const R out = fmaf((Gn + fabsf(Gn)) + (fabsf(Gs) - Gs), idy,
                                   __fmul_rn((Fe + fabsf(Fe)) + (fabsf(Fw) - Fw), idx));      // twice the outflow
                const R need = __fmul_rn(out, hdt);
                const R hh = c2.a;
                const R th = need > hh ? hh / (need > R(0) ? need : R(1)) : R(1);
                th0 = col_in ? th : R(1);
            }
            s_th[k2 + ts] = th0;
        }
        // ---- D: update of row r-3
        if (upd) {
            update<FULL>(orow, xp, k3, k4, th0, yn);
            if (SEG > 1) put_sums(orow - cy0);
        }
        by2 = by1;
        by1 = by0;
        bx1 = bx0;
    }

    template <bool FULL>
    __device__ __forceinline__ void update(const int orow, const int xp, const int k3, const int k4, const R thN,
                                           const Q4<R>& yn) {
        const R thC = s_th[k3 + ts], thS = s_th[k4 + ts];
        const R thW = s_th[k3 + ts - 1], thE = s_th[k3 + ts + 1];
        const Q4<R> xw = s_xf[xp + ts], xe = s_xf[xp + ts + 1], ys = s_yf[k3 + ts];
        const R h3 = s_cell[k3 + ts].a;
        R Fw = xw.a, Fe = xe.a, Gs = ys.a, Gn = yn.a, Tw = xw.d, Te = xe.d, Ts = ys.d, Tn = yn.d;
        // donor scaling, where any cell near this warp's is limited
        if (__any_sync(0xffffffffu, fminf(fminf(fminf(thC, thW), fminf(thE, thS)), thN) < 1.0f)) {
            const R sw = Fw > R(0) ? thW : thC, se = Fe > R(0) ? thC : thE;
            const R ss = Gs > R(0) ? thS : thC, sn = Gn > R(0) ? thC : thN;
            Fw = __fmul_rn(Fw, sw); Tw = __fmul_rn(Tw, sw); Fe = __fmul_rn(Fe, se); Te = __fmul_rn(Te, se);
            Gs = __fmul_rn(Gs, ss); Ts = __fmul_rn(Ts, ss); Gn = __fmul_rn(Gn, sn); Tn = __fmul_rn(Tn, sn);
        }
        // which product of a sum is fused is written out: a cell's bits must not depend on the
        // instantiation that updates it
        const R dh = fmaf(Gs - Gn, idy, __fmul_rn(Fw - Fe, idx));
        R dhu = __fmul_rn(xw.c - xe.b, idx), dhv = __fmul_rn(ys.c - yn.b, idy);
        if (c.order == 2) {
            dhu = fmaf(bx1, idx, dhu);
            dhv = fmaf(by2, idy, dhv);
        }
        dhu = fmaf(Ts - Tn, idy, dhu);
        dhv = fmaf(Tw - Te, idx, dhv);
        if (!do_out) return;
        if (west) { xin += relu(Fw); xout += relu(-Fw); }
        if (east) { xin += relu(-Fe); xout += relu(Fe); }
        if (!FULL) {
            if (orow == 0) { yin += relu(Gs); yout += relu(-Gs); }
            if (orow == ny - 1) { yin += relu(-Gn); yout += relu(Gn); }
        }
        const unsigned i = (unsigned)orow * (unsigned)nx + (unsigned)cx;
        R hn, hun, hvn;
        if (STAGE == 2) {
            hn = R(0.5) * fmaf(dt, dh, cin.h0 + h3);
            hun = R(0.5) * fmaf(dt, dhu, cin.hu0 + cin.hu1);
            hvn = R(0.5) * fmaf(dt, dhv, cin.hv0 + cin.hv1);
        } else {
            hn = fmaf(dt, dh, h3);
            hun = fmaf(dt, dhu, cin.hu0);
            hvn = fmaf(dt, dhv, cin.hv0);
        }
        const R neg = clamp0(-hn);
        acc_clip += neg;
        hn = hn + neg;
        if (STAGE == 1) {
            gd.h1[i] = hn; gd.hu1[i] = hun; gd.hv1[i] = hvn;
            return;
        }
        // ---- rain, Horton infiltration, retention store (swe2d.py:330-360)
        R sf = cin.sf;
        if (feat & FEAT_RAINW) {
            const R add = __fmul_rn(rdt, cin.rw);
            hn = hn + add;
            rainw += add;
        } else {
            hn = hn + rdt;
        }
        const R hp = hn;                   // depth the momentum belongs to
        if (feat & FEAT_HORTON) {
            const R rate_f = fmaf(cin.f0 - cin.fc, expf(-cin.k * tt), cin.fc);
            const R pot = __fmul_rn(rate_f, dt);
            const R take = rmin(pot, hn);
            hn = hn - take;
            R taken = take;
            if (feat & FEAT_STORE) {
                const R tks = rmin(pot - take, sf);
                sf = sf - tks;
                taken = taken + tks;
            }
            infil += taken;
            gd.ic[i] = cin.ic + taken;
        }
        if (feat & FEAT_STORE) {
            const R room = clamp0(cin.S - sf);
            const R fill = rmin(room, hn);
            hn = hn - fill;
            sf = sf + fill;
            gd.sf[i] = sf;
        }
        if (feat & (FEAT_HORTON | FEAT_STORE)) {       // water lost takes its momentum along
            const R keep = hp > R(0) ? hn / hp : R(0);
            hun = hun * keep;
            hvn = hvn * keep;
        }
        // ---- semi-implicit Manning friction (swe2d.py:362-370)
        // KP factor of the new depth, kept for the CFL velocity below
        const R h2 = hn * hn, h4 = __fmul_rn(h2, h2);
        const R ks = hn >= c.h_dry ? 1.4142135623730951f * hn * rsqrtf(h4 + fmaxf(h4, c.kp_eps)) : 0.0f;
        R u = hun * ks, v = hvn * ks;
        const R speed = dsqrt(fmaf(u, u, __fmul_rn(v, v)));
        const R nm = cin.n;
        const R slow = 1.0f / __fadd_rn(1.0f, dt * c.g * nm * nm * speed * powf(hn, -4.0f / 3.0f));
        u = u * slow;
        v = v * slow;
        const bool wet = hn >= c.h_dry;
        hun = wet ? hn * u : R(0);
        hvn = wet ? hn * v : R(0);
        if (STAGE == 2) {
            gd.h[i] = hn; gd.hu[i] = hun; gd.hv[i] = hvn;
        } else {
            gd.h1[i] = hn; gd.hu1[i] = hun; gd.hv1[i] = hvn;
        }
        // ---- CFL rate of the new state for the next step (swe2d.py:179-184)
        const R u2 = hun * ks, v2 = hvn * ks;
        // running peak speed and output use the KP velocities of the new state, as the
        // reference's snapshots do (swe2d.py:161-167, coupling.py:229-242)
        if (PEAKS && (feat & FEAT_PEAKS)) peaks_raise(i, hn, dsqrt(fmaf(u2, u2, __fmul_rn(v2, v2))));
        if (feat & FEAT_SNAP) {
            s_snap[0][i] = (float)hn;
            s_snap[1][i] = (float)u2;
            s_snap[2][i] = (float)v2;
        }
        const R cw = dsqrt(c.g * hn);
        const R rr = hn > c.h_dry ? fmaf(__fadd_rn(fabsf(v2), cw), idy, __fmul_rn(__fadd_rn(fabsf(u2), cw), idx)) : R(0);
        rate = rmax(rate, rr);
        hsum += hn;
        ssum += sf;
        hmax = rmax(hmax, hn);
    }
};

// Source column of an x-ghost: the layer of the grid it copies (boundaries.py:104-116),
// as halo_fetch picks it; the column itself inside the grid.
template <class R>
__device__ __forceinline__ int ghost_source_column(const KC<R>& c, const Grid<R>& gd, int cx) {
    const int nx = gd.nx;
    if ((unsigned)cx < (unsigned)nx) return cx;
    const int ng = c.order == 1 ? 1 : 2;
    const bool lo = cx < 0;
    const int k = lo ? (-cx - 1) : (cx - nx);
    const int kind = gd.bc[lo ? EDGE_W : EDGE_E];
    int layer;
    if (kind == BC_CLOSED || kind == BC_TRANSMISSIVE) layer = nx < ng ? (lo ? 0 : nx - 1) : (lo ? k : nx - 1 - k);
    else layer = lo ? 0 : nx - 1;
    return layer < 0 ? 0 : (layer > nx - 1 ? nx - 1 : layer);
}

// STAGE: 0 = first-order full step, 1 = RK stage 1, 2 = RK stage 2 + sources.
// Stage 1 writes the stage buffers; stage 2 reads them in its halo and writes the
// state.  The first-order step reads the state in its halo, so it writes its result
// to the stage buffers and stage_copy_kernel moves it back (no CTA overwrites cells
// that another CTA may still read).
//
// With few chunks a march is bound by its latency: 1.6 us a row, rows + 6 of them, two warps
// on an SM.  SEG = 2 and 4 march parts of the chunk side by side (strip_segments): one served
// storm of 400 x 325 cells in 58 x 16 took 71.5 us a step in one march, 59.7 in four.
template <class R, int NT, int STAGE, int SEG, bool PEAKS>
__global__ void __launch_bounds__(NT * SEG, StripGeom<R, NT>::min_ctas(STAGE, SEG)) strip_kernel(const Grid<R>* __restrict__ grids,
                                                    const StripRef* __restrict__ strips,
                                                    const StepParams* __restrict__ params, const KC<R> kc,
                                                    double* __restrict__ partials) {
    using G = StripGeom<R, NT>;
    // the stages of the second-order method (1, 2) and the first-order step (0) are
    // launched for their order only, so the order is a constant of the instantiation
    KC<R> c = kc;
    c.order = STAGE == 0 ? 1 : 2;
    constexpr int P = G::P;
    extern __shared__ __align__(32) unsigned char smem_raw[];
    __shared__ R bcv[4];
    __shared__ float* s_snap[3];                      // output slots of this step (stage 0 / 2)
    // the member's record, staged once: its field pointers are re-read every row, and
    // from global memory those reads stall the row loop
    __shared__ __align__(16) Grid<R> s_gd;

    const StripRef sr = strips[blockIdx.x];
    const StepParams& pr = params[sr.member];
    if (!pr.active) return;
    const int t = SEG == 1 ? threadIdx.x : threadIdx.x % NT, seg = SEG == 1 ? 0 : threadIdx.x / NT;
    {
        static_assert(sizeof(Grid<R>) % 4 == 0, "record copied as 32-bit words");
        const unsigned* src = reinterpret_cast<const unsigned*>(grids + sr.member);
        unsigned* dst = reinterpret_cast<unsigned*>(&s_gd);
        for (int k = threadIdx.x; k < (int)(sizeof(Grid<R>) / 4); k += NT * SEG) dst[k] = src[k];
    }
    if (threadIdx.x < 4) bcv[t] = par_bc<R>(pr, STAGE == 2, t);
    if (threadIdx.x == 0) {
        s_snap[0] = STAGE != 1 ? pr.snap_h : nullptr;
        s_snap[1] = pr.snap_u;
        s_snap[2] = pr.snap_v;
    }
    __syncthreads();
    const Grid<R>& gd = s_gd;
    Q4<R>* s_cell = reinterpret_cast<Q4<R>*>(smem_raw + seg * G::seg_stride);
    Q4<R>* s_rp = s_cell + G::RING * P;
    Q4<R>* s_xf = s_rp + P;
    Q4<R>* s_yf = s_xf + 2 * P;
    R* s_rs = reinterpret_cast<R*>(s_yf + G::RING * P);
    R* s_th = s_rs + P;
    StripPipe<R, NT, STAGE, SEG, PEAKS> pp{s_cell, s_rp, s_xf, s_yf, s_rs, s_th, gd, c, bcv, s_snap,
                               STAGE == 2 ? gd.h1 : gd.h, STAGE == 2 ? gd.hu1 : gd.hu, STAGE == 2 ? gd.hv1 : gd.hv};
    const int nx = gd.nx, ny = gd.ny;
    const int x0 = sr.x0, W = sr.w, rows = (sr.y1 - sr.y0 + SEG - 1) / SEG;
    const int y0 = SEG == 1 ? sr.y0 : min(sr.y0 + seg * rows, sr.y1), y1 = SEG == 1 ? sr.y1 : min(y0 + rows, sr.y1);
    const int cx = x0 - 3 + t;                        // this thread's column
    const int q = cx - x0;                            // column relative to the strip
    pp.ts = t + 1;
    pp.feat = grid_features(gd) | (s_snap[0] ? FEAT_SNAP : 0u);      // FEAT_SNAP: outputs due this step
    pp.cx = cx;
    pp.cxc = cx < 0 ? 0 : (cx > nx - 1 ? nx - 1 : cx);
    pp.nx = nx;
    pp.ny = ny;
    pp.cy0 = sr.y0;
    pp.y0 = y0;
    pp.y1 = y1;
    R* const s_sum = reinterpret_cast<R*>(smem_raw + SEG * G::seg_stride);
    R* const s_max = s_sum + (sr.y1 - sr.y0) * (G::NSUM * NT);
    pp.sums = s_sum + t;
    pp.bar = seg + 1;
    pp.col_in = (unsigned)cx < (unsigned)nx;
    pp.do_out = q >= 0 && q < W && pp.col_in;
    if (!pp.do_out) pp.feat &= ~FEAT_PEAKS;           // a halo column's peaks are another strip's
    pp.west = cx == 0;
    pp.east = cx == nx - 1;
    pp.scol = ghost_source_column(c, gd, cx);
    pp.xside = cx < 0 ? EDGE_W : EDGE_E;
    pp.xkind = pp.col_in ? -1 : gd.bc[pp.xside];
    pp.dt = par_dt<R>(pr);
    pp.hdt = R(0.5) * pp.dt;
    pp.idx = gd.idx;
    pp.idy = gd.idy;
    pp.rdt = __fmul_rn(par_rain<R>(pr), pp.dt);
    pp.tt = clamp0(par_t<R>(pr) - gd.rt0);
    pp.acc_clip = pp.xin = pp.xout = pp.yin = pp.yout = pp.infil = pp.rainw = pp.rate = pp.hsum = pp.ssum = R(0);
    pp.hmax = R(0);
    pp.by1 = pp.by2 = pp.bx1 = R(0);
    pp.old_pk = pp.old_ps = R(0);
    // software pipeline: raw rows are fetched one row ahead
    if (SEG == 1 || y0 < y1) pp.ra = halo_fetch(c, gd, pp.H, pp.HU, pp.HV, cx, y0 - 3);
    static_assert((G::RING & (G::RING - 1)) == 0, "ring slots are row & (RING - 1)");
    // steady-state rows: every row touched (r-4 .. r+1) inside the grid, the update row
    // neither the first nor the last row of the grid
    const int r_lo = max(y0 + 3, 4), r_hi = min(y1 + 2, ny - 2);
    int r = SEG == 1 || y0 < y1 ? y0 - 3 : y1 + 3;     // a segment without rows marches none
    for (; r <= y1 + 2 && r < r_lo; ++r) pp.template row<false>(r);
    // (not unrolled: four copies of the row body ran 1.75x slower, the hot loop no
    // longer fitting the instruction cache beside the other member chains' kernels)
    for (; r <= r_hi; ++r) pp.template row<true>(r);
    for (; r <= y1 + 2; ++r) pp.template row<false>(r);
    if (SEG > 1 && STAGE != 1) {
        s_max[(seg * G::NMAX + 0) * NT + t] = pp.rate;
        s_max[(seg * G::NMAX + 1) * NT + t] = pp.hmax;
    }
    __syncthreads();
    if (SEG > 1 && seg == 0) {
        pp.take_sums(sr.y1 - sr.y0);
        if (STAGE != 1) {
#pragma unroll
            for (int k = 1; k < SEG; ++k) {
                pp.rate = rmax(pp.rate, s_max[(k * G::NMAX + 0) * NT + t]);
                pp.hmax = rmax(pp.hmax, s_max[(k * G::NMAX + 1) * NT + t]);
            }
        }
    }
    R* red = reinterpret_cast<R*>(smem_raw);
    double* out = partials + (size_t)blockIdx.x * NPART;
    if (STAGE == 1) {
        R v[5] = {pp.acc_clip, pp.xin, pp.xout, pp.yin, pp.yout};
        const bool mx[5] = {false, false, false, false, false};
        const int sl[5] = {P_CLIP1, P_XIN1, P_XOUT1, P_YIN1, P_YOUT1};
        block_reduce_store<5>(v, mx, red, out, sl, NT);
    } else {
        const int b = STAGE == 2 ? P_CLIP2 : P_CLIP1;
        R v[11] = {pp.acc_clip, pp.xin, pp.xout, pp.yin, pp.yout, pp.infil, pp.rainw, pp.rate, pp.hsum, pp.ssum,
                   pp.hmax};
        const bool mx[11] = {false, false, false, false, false, false, false, true, false, false, true};
        const int sl[11] = {b, b + 1, b + 2, b + 3, b + 4, P_INFIL, P_RAINW, P_RATE, P_HSUM, P_SSUM, P_HMAX};
        block_reduce_store<11>(v, mx, red, out, sl, NT);
    }
}

// Cells of a strip-chunk in row order, spread over the threads of a CTA: consecutive
// threads take consecutive cells, and a chunk of any shape keeps every thread busy (one
// column per thread left most of a GPU idle behind a march of up to 48 rows).
constexpr int CHUNK_THREADS = 256;
template <class F>
__device__ __forceinline__ void for_chunk_cells(const StripRef& sr, int nx, F f) {
    const int n = sr.w * (sr.y1 - sr.y0);
    for (int i = threadIdx.x; i < n; i += CHUNK_THREADS) {
        const int y = i / sr.w;
        f((size_t)(sr.y0 + y) * nx + (sr.x0 + (i - y * sr.w)));
    }
}

// First-order step: move the result from the stage buffers back to the state.
template <class R>
__global__ void __launch_bounds__(CHUNK_THREADS) stage_copy_kernel(const Grid<R>* __restrict__ grids,
                                                                   const StripRef* __restrict__ strips,
                                                                   const StepParams* __restrict__ params) {
    const StripRef sr = strips[blockIdx.x];
    const Grid<R>& gd = grids[sr.member];
    if (!params[sr.member].active) return;
    R *__restrict__ h = gd.h, *__restrict__ hu = gd.hu, *__restrict__ hv = gd.hv;
    const R *__restrict__ h1 = gd.h1, *__restrict__ hu1 = gd.hu1, *__restrict__ hv1 = gd.hv1;
    for_chunk_cells(sr, gd.nx, [&](size_t i) {
        h[i] = h1[i];
        hu[i] = hu1[i];
        hv[i] = hv1[i];
    });
}

// CFL rate of one cell's state (swe2d.py:179-184); float64: rate64, as in the step.
__device__ __forceinline__ float cell_rate(const KC<float>& c, float h, float hu, float hv, const Grid<float>& gd) {
    float u, v;
    kp_velocity(c, h, hu, hv, u, v);
    const float cw = sqrtf(c.g * h);
    return h > c.h_dry ? fmaf(__fadd_rn(fabsf(v), cw), gd.idy, __fmul_rn(__fadd_rn(fabsf(u), cw), gd.idx)) : 0.0f;
}
__device__ __forceinline__ double rate64(const KC<double>& c, double h, double u, double v, double dx, double dy,
                                         double idx, double idy) {
    const double cw = sqrt(c.g * h);
    return f64_div(fabs(u) + cw, dx, idx) + f64_div(fabs(v) + cw, dy, idy);
}
__device__ __forceinline__ double cell_rate(const KC<double>& c, double h, double hu, double hv,
                                            const Grid<double>& gd) {
    if (!f64_ge_pos(h, c.h_dry) || f64_bits(h) == f64_bits(c.h_dry)) return 0.0;
    double u, v;
    kp_velocity(c, h, hu, hv, u, v);
    return rate64(c, h, u, v, gd.rdx, gd.rdy, gd.idx, gd.idy);
}

// Per strip-chunk CFL rate, surface and retained water of the current state (float64 sums).
template <class R>
__global__ void __launch_bounds__(CHUNK_THREADS) strip_reduce_kernel(const Grid<R>* __restrict__ grids,
                                                                     const StripRef* __restrict__ strips, const KC<R> c,
                                                                     double* __restrict__ partials) {
    __shared__ double red[32 * 3];
    const StripRef sr = strips[blockIdx.x];
    const Grid<R>& gd = grids[sr.member];
    R rate = R(0);
    double hs = 0, ss = 0;
    for_chunk_cells(sr, gd.nx, [&](size_t i) {
        const R h = gd.h[i];
        rate = rmax(rate, cell_rate(c, h, gd.hu[i], gd.hv[i], gd));
        hs += (double)h;
        ss += (double)gd.sf[i];
    });
    double v[3] = {(double)rate, hs, ss};
    const bool mx[3] = {true, false, false};
    const int sl[3] = {P_RATE, P_HSUM, P_SSUM};
    block_reduce_store<3>(v, mx, red, partials + (size_t)blockIdx.x * NPART, sl, CHUNK_THREADS);
}

// Per strip-chunk CFL rate alone (swe2d.py:179-184), for the step's dt: the maximum
// is exact in the compute type, so the result equals strip_reduce_kernel's.  Writes only
// the P_RATE partial.
template <class R>
__global__ void __launch_bounds__(CHUNK_THREADS) strip_rate_kernel(const Grid<R>* __restrict__ grids,
                                                                   const StripRef* __restrict__ strips, const KC<R> c,
                                                                   double* __restrict__ partials) {
    __shared__ R red[32];
    const StripRef sr = strips[blockIdx.x];
    const Grid<R>& gd = grids[sr.member];
    const R *__restrict__ h = gd.h, *__restrict__ hu = gd.hu, *__restrict__ hv = gd.hv;
    R rate = R(0);
    for_chunk_cells(sr, gd.nx, [&](size_t i) { rate = rmax(rate, cell_rate(c, h[i], hu[i], hv[i], gd)); });
    R v[1] = {rate};
    const bool mx[1] = {true};
    const int sl[1] = {P_RATE};
    block_reduce_store<1>(v, mx, red, partials + (size_t)blockIdx.x * NPART, sl, CHUNK_THREADS);
}

// N quantities j[] of a member's strip-chunk partials over its tiles, each summed (the rate
// and the depth: their maximum) in a fixed order by one warp: lane l takes the tiles l,
// l + 32, ..., then the lanes by a shuffle tree; valid in lane 0.
template <int N>
__device__ __forceinline__ void sum_columns(const double* __restrict__ partials, int tile0, int n_tiles,
                                            const int (&j)[N], double (&s)[N]) {
    const int lane = threadIdx.x & 31;
    bool mx[N];
#pragma unroll
    for (int q = 0; q < N; ++q) {
        mx[q] = j[q] == P_RATE || j[q] == P_HMAX;
        s[q] = 0.0;
    }
    // four tiles' loads in flight; a quantity that is zero in every lane's tile (edges, clips,
    // options that are off) costs a vote instead of an add
    const double* p = partials + (size_t)tile0 * NPART;
    for (int t0 = 0; t0 < n_tiles; t0 += 128) {
        double v[4][N];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int t = t0 + 32 * k + lane;
#pragma unroll
            for (int q = 0; q < N; ++q) v[k][q] = t < n_tiles ? p[(size_t)t * NPART + j[q]] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int q = 0; q < N; ++q) {
                if (!__any_sync(0xffffffffu, f64_bits(v[k][q]) << 1 != 0)) continue;
                s[q] = mx[q] ? fmax(s[q], v[k][q]) : s[q] + v[k][q];
            }
    }
#pragma unroll
    for (int q = 0; q < N; ++q) s[q] = mx[q] ? warp_max(s[q]) : warp_sum_sparse(s[q]);
}

// All of them into S[NPART] by a CTA: warp w the quantities w and w + FIN_WARPS.  Eight warps
// instead of one: a float64 add costs a warp 64 cycles, and one warp spent 16 quantities x
// (tiles / 32 + 5) of them in a row (1601 x 1301 float32 step with its reduction 261 -> 244 us,
// 225 -> 212 with four loads in flight and votes instead of adds of zeros; six served
// storms 94.7 -> 89.1 us per step).
constexpr int FIN_THREADS = 256, FIN_WARPS = FIN_THREADS / 32;
__device__ __forceinline__ void sum_partials(const double* __restrict__ partials, int tile0, int n_tiles, double* S) {
    const int warp = threadIdx.x >> 5;
    static_assert(NPART == 2 * FIN_WARPS, "two quantities per warp");
    const int j[2] = {warp, warp + FIN_WARPS};
    double s[2];
    sum_columns<2>(partials, tile0, n_tiles, j, s);
    if ((threadIdx.x & 31) == 0) {
        S[j[0]] = s[0];
        S[j[1]] = s[1];
    }
    __syncthreads();
}

// Volume terms of a step from its partial sums (m^3): one thread per term, in different
// warps, so that their float64 chains run side by side.  term: 0 boundary in, 1 boundary
// out, 2 rain, 3 infiltration, 4 clip.
template <class R>
__device__ __forceinline__ double step_term(int term, const Grid<R>& gd, double dt_, double rain, int order,
                                            const double* S) {
    const double dt = (double)R(dt_);
    if (term <= 1) {
        double q = S[term ? P_XOUT1 : P_XIN1] * gd.dy + S[term ? P_YOUT1 : P_YIN1] * gd.dx;
        if (order == 2) q = 0.5 * (q + (S[term ? P_XOUT2 : P_XIN2] * gd.dy + S[term ? P_YOUT2 : P_YIN2] * gd.dx));
        return q * dt;
    }
    if (term == 2)
        return gd.rw ? S[P_RAINW] * gd.area
                     : (double)(R(rain) * R(dt_)) * ((double)((long long)gd.nx * gd.ny) * gd.area);
    if (term == 3) return S[P_INFIL] * gd.area;
    const double clip = S[P_CLIP1] * gd.area;
    return order == 2 ? clip + S[P_CLIP2] * gd.area : clip;
}

// Per-member totals from the strip-chunk partials, in a fixed order.  out: 8 per
// member = bnd_in, bnd_out, rain, infil, clip (m^3), rate (1/s), surface and retained
// volume.  mode 0: after a step; mode 1: rate and volumes only; mode 2: rate only
// (after strip_rate_kernel).  For the caller (device-writable, optional): mode 0 the 5 volumes
// at StepParams::vols, modes 1 and 2 the rates at ext.  ledger (optional, mode 0): an 8 x n_members
// float64 ledger (rows LG_*) the step's rain, infiltration, boundary and clip volumes
// are added into.
//
// SPLIT: a CTA of FIN_COLUMNS warps for each of a member's FIN_OUT outputs instead of one for all
// (modes 0 and 1).  One SM takes an FP64 instruction per 19 cycles and a column's loads touch
// a line per tile, so one CTA takes 18 us for the 16 columns of 1148 tiles, eight 12 (a
// 1601 x 1301 float32 step with its CFL rate 186 -> 180 us).  From FIN_SPLIT tiles per member on:
// with 42 for each of 64 members, 512 CTAs cost more than they save (a coupled step 480 us in
// one CTA per member, 487 in eight).  Same order of summation, same bits.
constexpr int FIN_OUT = 8, FIN_COLUMNS = 4, FIN_SPLIT = 512;
template <class R, bool SPLIT>
__global__ void __launch_bounds__(FIN_THREADS) finalize_kernel(const Grid<R>* __restrict__ grids,
                                                               const StepParams* __restrict__ params, Consts c,
                                                               const double* __restrict__ partials,
                                                               double* __restrict__ out, int mode,
                                                               double* __restrict__ ext = nullptr,
                                                               double* __restrict__ ledger = nullptr) {
    __shared__ double S[NPART];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m = SPLIT ? blockIdx.x / FIN_OUT : blockIdx.x, k = SPLIT ? blockIdx.x % FIN_OUT : warp;
    const Grid<R>& gd = grids[m];
    if (mode == 0 && !params[m].active) return;
    double* o = out + (size_t)m * 8;
    if (mode == 2) {
        // the rates of 8 groups of tiles, then of the groups (a maximum has no order)
        double r = 0.0;
        for (int t = threadIdx.x; t < gd.n_tiles; t += FIN_THREADS)
            r = fmax(r, partials[(size_t)(gd.tile0 + t) * NPART + P_RATE]);
        r = warp_max(r);
        if (lane == 0) S[warp] = r;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < FIN_WARPS; ++w) r = fmax(r, S[w]);
            o[5] = r;
            if (ext) ext[m] = r;
        }
        return;
    }
    if constexpr (SPLIT) {
        // a warp per column that the CTA's output needs
        constexpr int COLUMNS[FIN_OUT][FIN_COLUMNS] = {{P_XIN1, P_YIN1, P_XIN2, P_YIN2},
                                                       {P_XOUT1, P_YOUT1, P_XOUT2, P_YOUT2},
                                                       {P_RAINW, -1, -1, -1}, {P_INFIL, -1, -1, -1},
                                                       {P_CLIP1, P_CLIP2, -1, -1}, {P_RATE, -1, -1, -1},
                                                       {P_HSUM, -1, -1, -1}, {P_SSUM, -1, -1, -1}};
        if (mode == 1 && k < 5) return;
        const int j[1] = {COLUMNS[k][warp]};
        if (j[0] >= 0) {
            double s[1];
            sum_columns<1>(partials, gd.tile0, gd.n_tiles, j, s);
            if (lane == 0) S[j[0]] = s[0];
        }
        __syncthreads();
        if (threadIdx.x != 0) return;
    } else {
        sum_partials(partials, gd.tile0, gd.n_tiles, S);
        if (lane != 0) return;
    }
    if (k == 5) {
        o[5] = S[P_RATE];
        if (mode != 0 && ext) ext[m] = S[P_RATE];
    } else if (k == 6) {
        o[6] = S[P_HSUM] * gd.area;
    } else if (k == 7) {
        o[7] = S[P_SSUM] * gd.area;
    } else if (mode == 0) {
        const double v = step_term(k, gd, params[m].dt, params[m].rain, c.order, S);
        o[k] = v;
        if (params[m].vols) params[m].vols[k] = v;
        if (ledger) {
            const int row = k == 0 ? LG_BND2_IN : k == 1 ? LG_BND2_OUT : k == 2 ? LG_RAIN : k == 3 ? LG_INFIL : LG_CLIP2;
            ledger[row * (size_t)(SPLIT ? gridDim.x / FIN_OUT : gridDim.x) + m] += v;
        }
    }
}

}  // namespace his
