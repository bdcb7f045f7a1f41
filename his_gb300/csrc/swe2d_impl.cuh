// Precision-templated host launchers of the 2-D strip kernels, the weir exchange and
// the device-resident engine.  Included once per precision by swe2d_f64.cu and
// swe2d_f32.cu.
#pragma once
#include <algorithm>
#include <climits>
#include <vector>

#include "engine_kernels.cuh"
#include "face_rule.h"
#include "his_internal.h"
#include "net1d_kernels.cuh"
#include "swe2d_strip.cuh"
#include "swe2d_tile64.cuh"

namespace his {

// How a grid's stages are launched: dynamic shared memory of the stage kernel, and for
// float64 sets with room for their faces the faces' table and the cell kernel's shared
// memory (NULL faces: the fused kernel); for float32 sets the segments a chunk is marched in.
struct StagePlan {
    size_t smem;
    const void* faces;
    size_t smem_cell;
    int seg;
    bool peaks;                      // some member has running peaks
};

// Segments (1, 2 or 4) the rows of a float32 strip-chunk are marched in side by side: the
// least estimated time for `tiles` chunks of at most `rows` rows, by default_tile's model of
// the march ((rows + 6) row times, a row 1.6 us while an SM holds few marches and 0.4 + 0.28 us
// x marches per SM beyond), where all of an SM's chunks stay resident.  Strips of up to 58
// columns only.  Measured, us per step in 1, 2 and 4 segments, second order with sources:
// 400 x 325 in 58 x 16, 147 chunks 57, 45 and 37; 294 58, 46 and 45; 441 58, 52 and 70; 588
// 62, 69 and 69; in 58 x 48 (49 chunks) 107, 70 and 57; 1601 x 1301 in 58 x 48 (784) 146,
// 330 and 235.
//
// A set with a member of one column is marched in one, for its totals' sake (StripPipe).
inline int strip_segments(int nt, int tiles, int rows, int narrowest) {
    if (nt != 64 || narrowest < 2) return 1;
    using G = StripGeom<float, 64>;
    const double per_sm = tiles / 152.0;
    int best = 1;
    double least = INFINITY;
    for (int seg = 1; seg <= 4; seg *= 2) {
        const int part = (rows + seg - 1) / seg;
        if (seg > 1 && std::ceil(per_sm) * (double)(G::seg_smem(seg, rows) + 2048) > 227 * 1024.0) break;
        const double t = (part + 6) * std::max(1.6, 0.4 + 0.28 * seg * per_sm);
        if (t < 0.9 * least) {
            least = t;
            best = seg;
        }
    }
    return best;
}

template <class R, int NT, int STAGE, bool PEAKS>
void launch_strips(const Grid<R>* grids, const StripRef* strips, const StepParams* params, const KC<R>& kc, double* part,
                   int count, const StagePlan& plan, cudaStream_t s) {
    if constexpr (NT == 64) {
        if (plan.seg == 4) {
            strip_kernel<R, NT, STAGE, 4, PEAKS><<<count, 4 * NT, plan.smem, s>>>(grids, strips, params, kc, part);
            return;
        }
        if (plan.seg == 2) {
            strip_kernel<R, NT, STAGE, 2, PEAKS><<<count, 2 * NT, plan.smem, s>>>(grids, strips, params, kc, part);
            return;
        }
    }
    strip_kernel<R, NT, STAGE, 1, PEAKS><<<count, NT, plan.smem, s>>>(grids, strips, params, kc, part);
}

// Launch of one stage over `count` strip-chunks: float32 marches strips with NT threads,
// float64 works off sub-tiles, faces and cells in two kernels or fused.
template <class R, int NT, int STAGE>
void launch_stage(const Grid<R>* grids, const StripRef* strips, const StepParams* params, const KC<R>& kc, double* part,
                  int count, const StagePlan& plan, cudaStream_t s) {
    if constexpr (sizeof(R) == 8) {
        if (plan.faces) {
            auto* faces = reinterpret_cast<const Faces64*>(plan.faces);
            face64_kernel<STAGE><<<count, TILE64_THREADS, plan.smem, s>>>(grids, faces, strips, params, kc);
            cell64_kernel<STAGE><<<count, TILE64_THREADS, plan.smem_cell, s>>>(grids, faces, strips, params, kc, part);
        } else {
            tile64_kernel<STAGE><<<count, TILE64_THREADS, plan.smem, s>>>(grids, strips, params, kc, part);
        }
    } else {
        if (STAGE != 1 && plan.peaks) launch_strips<R, NT, STAGE, STAGE != 1>(grids, strips, params, kc, part, count, plan, s);
        else launch_strips<R, NT, STAGE, false>(grids, strips, params, kc, part, count, plan, s);
    }
}

// Strip-chunk of a member whose full chunks are w x rows cells.
inline StripRef strip_ref(int member, int x0, int wc, int y0, int y1, int w, int rows) {
    return StripRef{member, x0, wc, y0, y1, (short)tile64_part(w, TILE64_W), (short)tile64_part(rows, TILE64_H)};
}

// Dynamic shared memory of a stage CTA over strip-chunks of at most w x rows cells
// (float32: marched in seg segments).
template <class R, int NT>
size_t stage_smem(int w, int rows, int order, int seg) {
    if constexpr (sizeof(R) == 8) return tile64_smem(tile64_part(w, TILE64_W), tile64_part(rows, TILE64_H), order == 2);
    else return seg > 1 ? StripGeom<R, NT>::seg_smem(seg, rows) : StripGeom<R, NT>::smem_bytes;
}

// Shared memory limits of one stage's strip kernels.
template <class R, int NT, int STAGE, bool PEAKS>
int set_strip_attrs() {
    constexpr int MOST = 227 * 1024;
    HIS_CK(cudaFuncSetAttribute(strip_kernel<R, NT, STAGE, 1, PEAKS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)StripGeom<R, NT>::smem_bytes));
    if constexpr (NT == 64) {
        HIS_CK(cudaFuncSetAttribute(strip_kernel<R, NT, STAGE, 2, PEAKS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    MOST - 1024));
        HIS_CK(cudaFuncSetAttribute(strip_kernel<R, NT, STAGE, 4, PEAKS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    MOST - 1024));
    }
    if constexpr (STAGE != 1 && !PEAKS) return set_strip_attrs<R, NT, STAGE, true>();
    return HIS_OK;
}

template <class R, int NT>
int set_stage_attrs() {
    if constexpr (sizeof(R) == 8) {
        const int bytes = (int)tile64_smem(TILE64_W, TILE64_H, true);
        HIS_CK(cudaFuncSetAttribute(tile64_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        HIS_CK(cudaFuncSetAttribute(tile64_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        HIS_CK(cudaFuncSetAttribute(tile64_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        const int face = (int)face64_smem(TILE64_W, TILE64_H, true);
        HIS_CK(cudaFuncSetAttribute(face64_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, face));
        HIS_CK(cudaFuncSetAttribute(face64_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, face));
        HIS_CK(cudaFuncSetAttribute(face64_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, face));
    } else {
        int rc;
        if ((rc = set_strip_attrs<R, NT, 0, false>()) || (rc = set_strip_attrs<R, NT, 1, false>()) ||
            (rc = set_strip_attrs<R, NT, 2, false>()))
            return rc;
    }
    return HIS_OK;
}

inline StagePlan stage_plan(const his_grid* g) { return StagePlan{g->stage_smem, g->d_faces, g->cell_smem, g->seg, g->peaks}; }

// The 2-D stages of one step on stream s (no finalize), over tiles [t0, t0 + count)
// (default: all); a tile's partials sit at its global index.
template <class R, int NT>
int launch_stages(his_grid* g, cudaStream_t s, int t0 = 0, int count = -1) {
    if (count < 0) count = g->n_tiles - t0;
    if (count == 0) return HIS_OK;
    auto* grids = reinterpret_cast<const Grid<R>*>(g->d_grids);
    const KC<R> kc = make_kc<R>(g->c);
    auto* strips = reinterpret_cast<const StripRef*>(g->d_tiles) + t0;
    double* part = g->d_partials + (size_t)t0 * NPART;
    if (g->c.order == 2) {
        launch_stage<R, NT, 1>(grids, strips, g->d_params, kc, part, count, stage_plan(g), s);
        launch_stage<R, NT, 2>(grids, strips, g->d_params, kc, part, count, stage_plan(g), s);
    } else {
        launch_stage<R, NT, 0>(grids, strips, g->d_params, kc, part, count, stage_plan(g), s);
        stage_copy_kernel<R><<<count, CHUNK_THREADS, 0, s>>>(grids, strips, g->d_params);
    }
    HIS_CK(cudaGetLastError());
    return HIS_OK;
}

// The stages over all tiles in g->n_parts parts side by side (part 0 on s), joined
// back into s.
template <class R, int NT>
int launch_stages_parted(his_grid* g, cudaStream_t s) {
    const int np = g->n_parts;
    if (np <= 1) return launch_stages<R, NT>(g, s);
    HIS_CK(cudaEventRecord(g->pev_fork, s));
    for (int k = 1; k < np; ++k) {
        HIS_CK(cudaStreamWaitEvent(g->ps[k - 1], g->pev_fork, 0));
        int rc = launch_stages<R, NT>(g, g->ps[k - 1], g->part_t[k], g->part_t[k + 1] - g->part_t[k]);
        if (rc) return rc;
        HIS_CK(cudaEventRecord(g->pev_join[k - 1], g->ps[k - 1]));
    }
    int rc = launch_stages<R, NT>(g, s, g->part_t[0], g->part_t[1] - g->part_t[0]);
    if (rc) return rc;
    for (int k = 1; k < np; ++k) HIS_CK(cudaStreamWaitEvent(s, g->pev_join[k - 1], 0));
    return HIS_OK;
}

// finalize_kernel over n members of n_tiles tiles in all
template <class R>
void finalize_launch(const Grid<R>* grids, const StepParams* params, const Consts& c, const double* partials, double* out,
                     int mode, double* ext, double* ledger, int n, int n_tiles, cudaStream_t s) {
    if (mode != 2 && n_tiles / n >= FIN_SPLIT)
        finalize_kernel<R, true><<<n * FIN_OUT, 32 * FIN_COLUMNS, 0, s>>>(grids, params, c, partials, out, mode, ext, ledger);
    else
        finalize_kernel<R, false><<<n, FIN_THREADS, 0, s>>>(grids, params, c, partials, out, mode, ext, ledger);
}

template <class R, int NT>
int launch_step_nt(his_grid* g, cudaStream_t s, double* ledger) {
    int rc = launch_stages_parted<R, NT>(g, s);
    if (rc) return rc;
    finalize_launch(reinterpret_cast<const Grid<R>*>(g->d_grids), g->d_params, g->c, g->d_partials, g->d_out, 0, nullptr,
                    ledger, g->n, g->n_tiles, s);
    HIS_CK(cudaGetLastError());
    return HIS_OK;
}

template <class R>
int launch_reduce(his_grid* g, cudaStream_t s, double* ext, bool rate_only) {
    auto* grids = reinterpret_cast<const Grid<R>*>(g->d_grids);
    auto* strips = reinterpret_cast<const StripRef*>(g->d_tiles);
    if (rate_only)
        strip_rate_kernel<R><<<g->n_tiles, CHUNK_THREADS, 0, s>>>(grids, strips, make_kc<R>(g->c), g->d_partials);
    else
        strip_reduce_kernel<R><<<g->n_tiles, CHUNK_THREADS, 0, s>>>(grids, strips, make_kc<R>(g->c), g->d_partials);
    finalize_launch(grids, g->d_params, g->c, g->d_partials, g->d_out, rate_only ? 2 : 1, ext, nullptr, g->n, g->n_tiles, s);
    HIS_CK(cudaGetLastError());
    return HIS_OK;
}

// float64 has one CTA size, whatever the strip width
#define HIS_NT_DISPATCH(FN, R, g, ...)                           \
    do {                                                         \
        if constexpr (sizeof(R) == 8) return FN<R, 0>(g, __VA_ARGS__); \
        else if (g->nt == 64) return FN<R, 64>(g, __VA_ARGS__);       \
        else if (g->nt == 128) return FN<R, 128>(g, __VA_ARGS__); \
        else if (g->nt == 224) return FN<R, 224>(g, __VA_ARGS__); \
        else if (g->nt == 352) return FN<R, 352>(g, __VA_ARGS__); \
        set_error("unsupported strip width (threads per CTA)");  \
        return HIS_ERR_BAD_ARG;                                  \
    } while (0)

// Face planes and bed terms of a float64 set's members and their table, where the set takes them
// (faces_taken) and the device can give them; else the fused kernel runs.
inline int faces_alloc(his_grid* g) {
    size_t total = 0, cells = 0;
    std::vector<size_t> off(g->n);
    auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
    for (int m = 0; m < g->n; ++m) {
        const size_t ny = g->desc[m].ny, nx = g->desc[m].nx;
        off[m] = total;
        total += up(32 * ny * (nx + 1)) + up(32 * (ny + 1) * nx) + up(16 * ny * nx);
        cells += ny * nx;
    }
    size_t free_bytes = 0, all_bytes = 0;
    HIS_CK(cudaMemGetInfo(&free_bytes, &all_bytes));
    if (!faces_taken(total, cells, free_bytes)) return HIS_OK;
    if (cudaMalloc(&g->d_face_planes, total) != cudaSuccess) {
        cudaGetLastError();
        g->d_face_planes = nullptr;
        return HIS_OK;
    }
    std::vector<Faces64> F(g->n);
    for (int m = 0; m < g->n; ++m) {
        const size_t ny = g->desc[m].ny, nx = g->desc[m].nx;
        char* p = (char*)g->d_face_planes + off[m];
        F[m].fx = (Q4<double>*)p;
        p += up(32 * ny * (nx + 1));
        F[m].fy = (Q4<double>*)p;
        p += up(32 * (ny + 1) * nx);
        F[m].bed = (double2*)p;
    }
    HIS_CK(cudaMalloc(&g->d_faces, sizeof(Faces64) * g->n));
    HIS_CK(cudaMemcpy(g->d_faces, F.data(), sizeof(Faces64) * g->n, cudaMemcpyHostToDevice));
    g->scratch_bytes += total;
    return HIS_OK;
}

// Strip decomposition of every member: columns in ceil(nx / (NT - 6)) strips of equal
// width, rows in chunks of `ty` rows; the work units are listed member by member.
template <class R>
int grid_init_impl(his_grid* g) {
    int rc;
    if constexpr (sizeof(R) == 8) {
        if ((rc = set_stage_attrs<R, 0>()) != HIS_OK) return rc;
    } else {
        if ((rc = set_stage_attrs<R, 64>()) != HIS_OK) return rc;
        if ((rc = set_stage_attrs<R, 128>()) != HIS_OK) return rc;
        if ((rc = set_stage_attrs<R, 224>()) != HIS_OK) return rc;
        if ((rc = set_stage_attrs<R, 352>()) != HIS_OK) return rc;
    }
    const int n = g->n;
    std::vector<Grid<R>> H(n);
    std::vector<StripRef> strips;
    g->tile0.assign(n, 0);
    g->ntile.assign(n, 0);
    std::vector<size_t> off(n);
    size_t total = 0;
    for (int m = 0; m < n; ++m) {
        const his_grid_desc& d = g->desc[m];
        size_t plane = ((size_t)d.ny * d.nx * sizeof(R) + 255) & ~size_t(255);
        off[m] = total;
        total += 3 * plane;
    }
    g->scratch_bytes = total;
    HIS_CK(cudaMalloc(&g->d_scratch, total > 0 ? total : 256));
    const int wmax = g->tx;
    int sub_w = 1, sub_h = 1, rows = 1, narrowest = INT_MAX;
    for (int m = 0; m < n; ++m) {
        const his_grid_desc& d = g->desc[m];
        Grid<R>& G = H[m];
        G.ny = d.ny;
        G.nx = d.nx;
        for (int e = 0; e < 4; ++e) G.bc[e] = d.bc[e];
        G.dx = d.dx;
        G.dy = d.dy;
        G.area = d.dx * d.dy;
        G.t0 = d.horton_t0;
        G.rdx = R(d.dx);
        G.rdy = R(d.dy);
        G.rt0 = R(d.horton_t0);
        G.idx = R(1.0 / d.dx);
        G.idy = R(1.0 / d.dy);
        G.rarea = R(1.0 / G.area);
        const int ns = (d.nx + wmax - 1) / wmax;
        const int w = (d.nx + ns - 1) / ns;
        const int nch = (d.ny + g->ty - 1) / g->ty;
        const int hch = (d.ny + nch - 1) / nch;          // balanced chunk height <= ty
        G.tiles_x = ns;
        G.tiles_y = nch;
        G.n_tiles = ns * nch;
        rows = std::max(rows, hch);
        narrowest = std::min(narrowest, d.nx);
        if constexpr (sizeof(R) == 8) {
            sub_w = std::max(sub_w, tile64_part(w, TILE64_W));
            sub_h = std::max(sub_h, tile64_part(hch, TILE64_H));
        }
        G.tile0 = (int)strips.size();
        g->tile0[m] = G.tile0;
        g->ntile[m] = G.n_tiles;
        for (int cy = 0; cy < nch; ++cy)
            for (int sx = 0; sx < ns; ++sx) {
                const int x0 = sx * w, y0 = cy * hch;
                strips.push_back(strip_ref(m, x0, std::min(w, d.nx - x0), y0, std::min(y0 + hch, d.ny), w, hch));
            }
        G.h = (R*)d.h; G.hu = (R*)d.hu; G.hv = (R*)d.hv; G.sf = (R*)d.s_filled; G.ic = (R*)d.infil_cum;
        size_t plane = ((size_t)d.ny * d.nx * sizeof(R) + 255) & ~size_t(255);
        char* base = (char*)g->d_scratch + off[m];
        G.h1 = (R*)base; G.hu1 = (R*)(base + plane); G.hv1 = (R*)(base + 2 * plane);
        G.z = (const R*)d.z; G.n = (const R*)d.manning; G.S = (const R*)d.storage;
        G.f0 = (const R*)d.f0; G.fc = (const R*)d.fc; G.k = (const R*)d.k; G.rw = (const R*)d.rain_weight;
        G.pk = (R*)d.peak_h; G.ps = (R*)d.peak_speed;
        g->peaks = g->peaks || G.pk || G.ps;
    }
    g->n_tiles = (int)strips.size();
    if constexpr (sizeof(R) == 8) {
        if ((rc = faces_alloc(g)) != HIS_OK) return rc;
        const bool second = g->c.order == 2;
        g->stage_smem = g->d_faces ? face64_smem(sub_w, sub_h, second) : tile64_smem(sub_w, sub_h, second);
        g->cell_smem = cell64_smem(sub_w, sub_h);
    } else {
        g->seg = strip_segments(g->nt, g->n_tiles, rows, narrowest);
        g->stage_smem = g->nt == 64 ? stage_smem<R, 64>(0, rows, 0, g->seg) : g->nt == 128 ? stage_smem<R, 128>(0, 0, 0, 1)
                      : g->nt == 224 ? stage_smem<R, 224>(0, 0, 0, 1) : stage_smem<R, 352>(0, 0, 0, 1);
    }
    HIS_CK(cudaMalloc(&g->d_grids, sizeof(Grid<R>) * n));
    HIS_CK(cudaMemcpy(g->d_grids, H.data(), sizeof(Grid<R>) * n, cudaMemcpyHostToDevice));
    HIS_CK(cudaMalloc(&g->d_tiles, sizeof(StripRef) * strips.size()));
    HIS_CK(cudaMemcpy(g->d_tiles, strips.data(), sizeof(StripRef) * strips.size(), cudaMemcpyHostToDevice));
    HIS_CK(cudaMalloc(&g->d_partials, sizeof(double) * NPART * (size_t)g->n_tiles));
    HIS_CK(cudaMemset(g->d_partials, 0, sizeof(double) * NPART * (size_t)g->n_tiles));
    g->table_bytes = sizeof(Grid<R>) * n + sizeof(StripRef) * strips.size() + sizeof(double) * NPART * g->n_tiles;
    return HIS_OK;
}

template <class R>
int grid_step_impl(his_grid* g, cudaStream_t s, double* ledger) {
    HIS_NT_DISPATCH(launch_step_nt, R, g, s, ledger);
}

template <class R>
int grid_reduce_impl(his_grid* g, cudaStream_t s, double* ext, bool rate_only) {
    return launch_reduce<R>(g, s, ext, rate_only);
}

template <class R>
int exchange_impl(his_links* l, const Consts& c, double dt, double* V, cudaStream_t s) {
    constexpr int G = sizeof(R) == 8 ? EXCH_SLICES : 1;
    const size_t smem = l->smem_of(sizeof(R));
    if (smem > 48 * 1024)
        HIS_CK(cudaFuncSetAttribute(exchange_kernel<R, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    exchange_kernel<R, G><<<l->n * G, EXCHANGE_THREADS, smem, s>>>(l->d_links, l->net->d_nets,
                                                                   reinterpret_cast<const Grid<R>*>(l->grid->d_grids),
                                                                   make_exch_k<R>(c), (R)dt, V, l->d_Vpos, l->d_exch);
    HIS_CK(cudaGetLastError());
    return HIS_OK;
}

// CTAs per member of a set's pre-steps (see eng_pre_kernel).
template <class R>
int pre_ctas(const his_engine* E) { return sizeof(R) == 8 ? EXCH_SLICES : E->n <= PRE_MEMBERS_F32 ? 4 : 1; }

// The pre-step of members [m0, m0 + mc), with the set's number of CTAs per member; turn: behind
// the accounting of the step before it (pre_ctas > 1).
template <class R>
void launch_pre(his_engine* E, const Grid<R>* grids, int m0, int mc, cudaStream_t s, bool turn = false) {
    his_grid* g = E->grid;
    const Net* nets = E->net ? E->net->d_nets : nullptr;
    const Lnk* links = E->links ? E->links->d_links : nullptr;
    double* exch = E->links ? E->links->d_exch : nullptr;
    double* vpos = E->links ? E->links->d_Vpos : nullptr;
    auto launch = [&](auto kernel, int ctas) {
        kernel<<<mc * ctas, ENG_PRE_THREADS, E->pre_smem, s>>>(E->d_em, g->d_params, grids, nets, links, g->c,
                                                               make_exch_k<R>(g->c), E->d_netf, E->max_sub, vpos, exch,
                                                               m0, g->d_partials, E->net ? E->d_vol1d : nullptr,
                                                               g->d_out);
    };
    constexpr int G = sizeof(R) == 8 ? EXCH_SLICES : 4;
    if (sizeof(R) == 4 && pre_ctas<R>(E) == 1) launch(eng_pre_kernel<R, sizeof(R) == 4 ? 1 : G, false>, 1);
    else if (turn) launch(eng_pre_kernel<R, G, true>, G);
    else launch(eng_pre_kernel<R, G, false>, G);
}

// One device-resident step for every member of one chain (see engine_kernels.cuh)
// on the chain's main stream; the 1-D substeps run on its side stream between a
// fork and a join event, concurrently with the 2-D stages.
template <class R, int NT>
int eng_enqueue_nt(his_grid* g, his_engine* E, int chain, int n_steps) {
    auto* grids = reinterpret_cast<const Grid<R>*>(g->d_grids);
    const int m0 = E->chain_m[chain], mc = E->chain_m[chain + 1] - m0;
    const int t0 = E->chain_t[chain], tc = E->chain_t[chain + 1] - t0;
    cudaStream_t s_main = E->main_of(chain), s_side = E->side_of(chain);
    cudaEvent_t fork = E->fork_of(chain), join = E->join_of(chain);
    if (mc == 0) return HIS_OK;
    const bool turns = pre_ctas<R>(E) > 1;
    for (int k = 0; k < n_steps; ++k) {
        if (k == 0 || !turns) launch_pre<R>(E, grids, m0, mc, s_main);
        if (E->net) {
            HIS_CK(cudaEventRecord(fork, s_main));
            HIS_CK(cudaStreamWaitEvent(s_side, fork, 0));
            int rc = net_engine_launch(E, s_side, m0, mc);
            if (rc) return rc;
            HIS_CK(cudaEventRecord(join, s_side));
        }
        int rc = launch_stages<R, NT>(g, s_main, t0, tc);
        if (rc) return rc;
        if (E->net) HIS_CK(cudaStreamWaitEvent(s_main, join, 0));
        if (turns && k + 1 < n_steps) launch_pre<R>(E, grids, m0, mc, s_main, true);
        else eng_post_kernel<R><<<mc, FIN_THREADS, 0, s_main>>>(E->d_em, g->d_params, grids, g->c, g->d_partials,
                                                  E->net ? E->d_vol1d : nullptr, g->d_out, m0);
        HIS_CK(cudaGetLastError());
    }
    return HIS_OK;
}

template <class R>
int engine_enqueue_impl(his_engine* E, int chain, int n_steps) {
    his_grid* g = E->grid;
    HIS_NT_DISPATCH(eng_enqueue_nt, R, g, E, chain, n_steps);
}

template <class R>
int engine_take_rate_impl(his_engine* E) {
    // kernel attributes are set here, outside any stream capture
    if (E->pre_smem > 48 * 1024) {
        constexpr int G = sizeof(R) == 8 ? EXCH_SLICES : 4;
        for (auto kernel : {eng_pre_kernel<R, sizeof(R) == 4 ? 1 : G, false>, eng_pre_kernel<R, G, false>, eng_pre_kernel<R, G, true>})
            HIS_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)E->pre_smem));
    }
    int rc = grid_reduce_impl<R>(E->grid, E->s0, nullptr, false);
    if (rc) return rc;
    eng_take_rate_kernel<<<(E->n + 127) / 128, 128, 0, E->s0>>>(E->d_em, E->grid->d_out, E->n);
    HIS_CK(cudaGetLastError());
    return HIS_OK;
}

// Same step sequence as eng_enqueue_nt, uncaptured, with CUDA events around each
// kernel class on its own stream; accumulates device milliseconds into ms[6].
template <class R, int NT>
int eng_profile_nt(his_grid* g, his_engine* E, int n_steps, double* ms) {
    auto* grids = reinterpret_cast<const Grid<R>*>(g->d_grids);
    const KC<R> kc = make_kc<R>(g->c);
    auto* strips = reinterpret_cast<const StripRef*>(g->d_tiles);
    cudaEvent_t ev[7];
    for (auto& e : ev) HIS_CK(cudaEventCreate(&e));
    int rc = HIS_OK;
    for (int k = 0; k < n_steps && rc == HIS_OK; ++k) {
        cudaEventRecord(ev[0], E->s0);
        launch_pre<R>(E, grids, 0, E->n, E->s0);
        cudaEventRecord(ev[1], E->s0);
        if (E->net) {
            cudaStreamWaitEvent(E->s1, ev[1], 0);
            cudaEventRecord(ev[4], E->s1);
            rc = net_engine_launch(E, E->s1, 0, E->n);
            cudaEventRecord(ev[5], E->s1);
        }
        if (g->c.order == 2) {
            launch_stage<R, NT, 1>(grids, strips, g->d_params, kc, g->d_partials, g->n_tiles, stage_plan(g), E->s0);
            cudaEventRecord(ev[2], E->s0);
            launch_stage<R, NT, 2>(grids, strips, g->d_params, kc, g->d_partials, g->n_tiles, stage_plan(g), E->s0);
        } else {
            cudaEventRecord(ev[2], E->s0);
            launch_stage<R, NT, 0>(grids, strips, g->d_params, kc, g->d_partials, g->n_tiles, stage_plan(g), E->s0);
            stage_copy_kernel<R><<<g->n_tiles, CHUNK_THREADS, 0, E->s0>>>(grids, strips, g->d_params);
        }
        cudaEventRecord(ev[3], E->s0);
        if (E->net) cudaStreamWaitEvent(E->s0, ev[5], 0);
        eng_post_kernel<R><<<E->n, FIN_THREADS, 0, E->s0>>>(E->d_em, g->d_params, grids, g->c, g->d_partials,
                                                   E->net ? E->d_vol1d : nullptr, g->d_out, 0);
        cudaEventRecord(ev[6], E->s0);
        cudaError_t ce = cudaEventSynchronize(ev[6]);
        if (ce != cudaSuccess) { rc = cuda_fail(ce, "his_engine_profile"); break; }
        float t;
        cudaEventElapsedTime(&t, ev[0], ev[1]); ms[0] += t;
        cudaEventElapsedTime(&t, ev[1], ev[2]); ms[1] += t;
        cudaEventElapsedTime(&t, ev[2], ev[3]); ms[2] += t;
        if (E->net) { cudaEventElapsedTime(&t, ev[4], ev[5]); ms[3] += t; }
        cudaEventElapsedTime(&t, ev[3], ev[6]); ms[4] += t;
        cudaEventElapsedTime(&t, ev[0], ev[6]); ms[5] += t;
    }
    for (auto& e : ev) cudaEventDestroy(e);
    if (rc == HIS_OK) HIS_CK(cudaGetLastError());
    return rc;
}

template <class R>
int engine_profile_impl(his_engine* E, int n_steps, double* ms) {
    his_grid* g = E->grid;
    HIS_NT_DISPATCH(eng_profile_nt, R, g, E, n_steps, ms);
}

// ---------------------------------------------------------------- no-allocation step
// Writes the grid record, the step parameters and the strip table of one grid into
// the caller's scratch and clears its partial sums and totals.  The records arrive
// as kernel arguments, so no host buffer has to outlive the call.
template <class R>
__global__ void noalloc_setup_kernel(Grid<R> G, StepParams P, NoallocPlan L, unsigned char* __restrict__ base) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int stride = gridDim.x * blockDim.x;
    auto* strips = reinterpret_cast<StripRef*>(base + L.o_strips);
    auto* part = reinterpret_cast<double*>(base + L.o_part);
    for (int b = i; b < L.n_strips; b += stride) {
        const int sx = b % L.ns, cy = b / L.ns;
        const int x0 = sx * L.w, y0 = cy * L.hch;
        strips[b] = StripRef{0, x0, min(L.w, G.nx - x0), y0, min(y0 + L.hch, G.ny),
                             (short)tile64_part(L.w, TILE64_W), (short)tile64_part(L.hch, TILE64_H)};
    }
    for (int j = i; j < NPART * L.n_strips; j += stride) part[j] = 0.0;
    if (i < 8) reinterpret_cast<double*>(base + L.o_out)[i] = 0.0;
    if (i == 0) {
        *reinterpret_cast<Grid<R>*>(base + L.o_grid) = G;
        *reinterpret_cast<StepParams*>(base + L.o_params) = P;
    }
}

// One step of one grid with every table and stage buffer in the scratch at `base`
// (laid out by L): the same stage kernels, decomposition and fixed-order totals as a
// one-member set created with default tiles.
template <class R>
int noalloc_step_impl(const Consts& c, const his_grid_desc& d, const his_step_params& p, const NoallocPlan& L,
                      unsigned char* base, cudaStream_t s) {
    constexpr int NT = sizeof(R) == 8 ? 0 : 64;
    static_assert(sizeof(Grid<R>) <= 256 && sizeof(StepParams) <= 256, "records exceed their scratch slots");
    int rc = set_stage_attrs<R, NT>();
    if (rc) return rc;
    Grid<R> G{};
    G.ny = d.ny;
    G.nx = d.nx;
    for (int e = 0; e < 4; ++e) G.bc[e] = d.bc[e];
    G.dx = d.dx;
    G.dy = d.dy;
    G.area = d.dx * d.dy;
    G.t0 = d.horton_t0;
    G.rdx = R(d.dx);
    G.rdy = R(d.dy);
    G.rt0 = R(d.horton_t0);
    G.idx = R(1.0 / d.dx);
    G.idy = R(1.0 / d.dy);
    G.rarea = R(1.0 / G.area);
    G.tile0 = 0;
    G.tiles_x = L.ns;
    G.tiles_y = L.nch;
    G.n_tiles = L.n_strips;
    G.h = (R*)d.h; G.hu = (R*)d.hu; G.hv = (R*)d.hv; G.sf = (R*)d.s_filled; G.ic = (R*)d.infil_cum;
    unsigned char* st = base + L.o_stage;
    G.h1 = (R*)st; G.hu1 = (R*)(st + L.plane); G.hv1 = (R*)(st + 2 * L.plane);
    G.z = (const R*)d.z; G.n = (const R*)d.manning; G.S = (const R*)d.storage;
    G.f0 = (const R*)d.f0; G.fc = (const R*)d.fc; G.k = (const R*)d.k; G.rw = (const R*)d.rain_weight;
    G.pk = (R*)d.peak_h; G.ps = (R*)d.peak_speed;
    const StepParams P = step_params_from(p);
    const int work = std::max(L.n_strips * (int)NPART, 8);
    noalloc_setup_kernel<R><<<(work + 255) / 256, 256, 0, s>>>(G, P, L, base);
    auto* grid = reinterpret_cast<const Grid<R>*>(base + L.o_grid);
    auto* params = reinterpret_cast<const StepParams*>(base + L.o_params);
    auto* strips = reinterpret_cast<const StripRef*>(base + L.o_strips);
    auto* part = reinterpret_cast<double*>(base + L.o_part);
    auto* out = reinterpret_cast<double*>(base + L.o_out);
    const KC<R> kc = make_kc<R>(c);
    const int seg = sizeof(R) == 8 ? 1 : strip_segments(NT, L.n_strips, L.hch, G.nx);
    const StagePlan smem{stage_smem<R, NT>(L.w, L.hch, c.order, seg), nullptr, 0, seg, G.pk || G.ps};
    if (c.order == 2) {
        launch_stage<R, NT, 1>(grid, strips, params, kc, part, L.n_strips, smem, s);
        launch_stage<R, NT, 2>(grid, strips, params, kc, part, L.n_strips, smem, s);
    } else {
        launch_stage<R, NT, 0>(grid, strips, params, kc, part, L.n_strips, smem, s);
        stage_copy_kernel<R><<<L.n_strips, CHUNK_THREADS, 0, s>>>(grid, strips, params);
    }
    finalize_launch<R>(grid, params, c, part, out, 0, nullptr, nullptr, 1, L.n_strips, s);
    HIS_CK(cudaGetLastError());
    return HIS_OK;
}

}  // namespace his
