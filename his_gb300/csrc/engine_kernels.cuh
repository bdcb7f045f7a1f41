// Device-resident coupled time loop: every member advances with its own dt, chosen,
// forced and accounted for on the GPU, so K steps run as one CUDA graph with no
// host round trip.  The per-member kernels take the first member m0 of the chain
// they serve (block b works on member m0 + b).  One step is
//
//   eng_pre   (a CTA, or a cluster of four or eight, per member)  2-D CFL dt from the rate
//             of the current state, 1-D CFL and substep count, weir exchange, forcing at
//             t, t+dt and the 1-D substep starts          (coupling.py:201-212)
//   stage 1, stage 2 (tiles of every member)              (swe2d.py:305-371)
//   net substeps (one CTA per member, concurrent with the 2-D stages)
//                                                         (coupling.py:216-221)
//   eng_post  (one CTA per member)  step volumes summed in tile order into the
//             float64 accumulators, t += dt, plausibility (coupling.py:213-227, :169-192)
//
// Where a member's pre-step has several CTAs, a step's eng_post and the next one's eng_pre
// are one kernel (TURN below).
#pragma once
#include "net1d_kernels.cuh"
#include "swe2d_strip.cuh"

namespace his {

// The per-member pre-step CTAs (one, or a cluster of them, pre_ctas): warps 0 .. 13
// exchange water with the channel, each CTA a slice of it; warp 14 chooses dt and the
// substep count (every CTA the same) and evaluates the substep forcing, warp 15 the step's
// parameters, side by side (a float64 cosine or division is a chain of hundreds to
// thousands of cycles, and the exchange is a chain of load latencies).
//
// CTAs per member: float64 8, the exchange being bound by FP64 instructions; float32 4 while
// the set is small (32 members and fewer; no member's bits depend on it), where spare SMs
// shorten the chain, else 1.  16 steps in us with one CTA and with four (and TURN): 400 x 325
// cells in 58 x 48, 8 members 1904 and 1752, 24 2894 and 2802, 32 3238 and 3320, 48 4116 and 4430,
// 64 5253 and 5635; in 58 x 16, 8 1322 and 1181, 32 3368 and 3298, 64 6253 and 6227; 100 x 81
// cells, 8 644 and 571, 32 974 and 898, 48 983 and 976, 64 1064 and 1099.
constexpr int PRE_MEMBERS_F32 = 32;
constexpr int ENG_PRE_THREADS = 512, ENG_EXCH_THREADS = 448, ENG_EXCH_WARPS = ENG_EXCH_THREADS / 32;

//
// TURN: the last step's eng_post in front, spread over warps 14 and 15 of the member's CTAs:
// every CTA's take the clock, the rate and the status they need, side by side with the
// exchange's loads and water levels; rank 0's write them, and those of ranks 1 to 3 add up the
// volumes.  eng_post's chain (partial sums, then a division) and one launch leave the step:
// six served storms 60 -> 57 us a step, one float64 storm of 400 x 325 cells 252 -> 248.
// A member that ended or failed leaves at the substep count (s_nsub), as one that needs too
// many substeps does: after the barriers, before any state is written.
template <class R, int G, bool TURN>
__global__ void __cluster_dims__(G, 1, 1) __launch_bounds__(ENG_PRE_THREADS, sizeof(R) == 4 && G == 1 ? 2 : 1)
eng_pre_kernel(EngMember* __restrict__ em, StepParams* __restrict__ params, const Grid<R>* __restrict__ grids,
               const Net* __restrict__ nets, const Lnk* __restrict__ links, Consts c, ExchK<R> K,
               double* __restrict__ netf, int max_sub, double* Vg, double* __restrict__ exch, int m0,
               const double* __restrict__ partials, const double* __restrict__ vol1d, double* __restrict__ out) {
    static_assert(!TURN || G >= 4, "the volumes are added up by three CTAs beside the first");
    extern __shared__ double sm[];
    __shared__ Lnk s_L;
    __shared__ Net s_N;
    __shared__ int s_nsub, s_snap, s_status;
    __shared__ double s_dt, s_t;
    __shared__ R s_dtr, s_rate[G * ENG_EXCH_WARPS];     // every CTA's rates
    const int m = m0 + blockIdx.x / G, rank = blockIdx.x % G, tid = threadIdx.x, lane = tid & 31;
    EngMember& E = em[m];
    StepParams& P = params[m];
    if (E.status != ST_RUNNING) {              // (every thread reads it before any barrier)
        if (rank == 0 && tid == 0) P.active = 0;
        return;
    }
    // what the last step left, the clock and the output counter one step on (volatile: every
    // CTA reads it before the first barrier, behind which another CTA writes it)
    struct { double t, dt, rate, rain; int k_out, snap, n_sub; double* ledger; } last{};
    if (tid >= ENG_EXCH_THREADS) {
        const volatile EngMember& Ev = E;
        const volatile StepParams& Pv = P;
        last.t = Ev.t;
        last.rate = Ev.rate;
        last.k_out = Ev.k_out;
        if (TURN) {
            last.dt = Ev.dt;
            last.t += last.dt;
            last.rain = Pv.rain;
            last.snap = Pv.snap_k;
            last.n_sub = Ev.n_sub;
            if (last.snap >= 0) {
                last.k_out = last.snap + 1;
                last.ledger = Pv.snap_ledger;
            }
        }
    }
    // TURN: step volumes into the accumulators, by warp 14 (w = 0) and 15 (w = 1) of ranks 1 to 3
    auto add_volumes = [&](int w) {
        if (rank > 3) return;
        const Grid<R>& gd = grids[m];
        double* o = out + (size_t)m * 8;
        double* L = last.ledger;
        const bool net = vol1d && last.n_sub > 0;
        double S[NPART];
        auto take = [&](auto... q) {
            const int j[sizeof...(q)] = {(int)q...};
            double s[sizeof...(q)];
            sum_columns<sizeof...(q)>(partials, gd.tile0, gd.n_tiles, j, s);
            int k = 0;
            ((S[q] = s[k++]), ...);
        };
        auto account = [&](int term, int a, double more) {
            const double v = step_term(term, gd, last.dt, last.rain, c.order, S);
            if (lane != 0) return;
            o[term] = v;
            double acc = E.acc[a] + v;
            if (term == 4 && net) acc += more;
            E.acc[a] = acc;
            if (L) L[L_RAIN + a] = acc;
        };
        if (rank == 1 && w == 0) {
            take(P_XIN1, P_YIN1, P_XIN2, P_YIN2);
            account(0, 2, 0.0);
        } else if (rank == 1) {
            take(P_XOUT1, P_YOUT1, P_XOUT2, P_YOUT2);
            account(1, 3, 0.0);
        } else if (rank == 2 && w == 0) {
            take(P_RAINW, P_INFIL);
            account(2, 0, 0.0);
            account(3, 1, 0.0);
        } else if (rank == 2) {
            take(P_CLIP1, P_CLIP2);
            account(4, 6, net ? vol1d[m * 3 + 2] : 0.0);
        } else if (w == 0) {
            take(P_HSUM, P_SSUM);
            if (lane == 0) {
                const double v2 = S[P_HSUM] * gd.area, vs = S[P_SSUM] * gd.area;
                o[6] = v2;
                o[7] = vs;
                if (L) {
                    L[L_V2D] = v2;
                    L[L_STORE] = vs;
                }
            }
        } else if (lane < 2) {
            const double acc = net ? E.acc[4 + lane] + vol1d[m * 3 + lane] : E.acc[4 + lane];
            E.acc[4 + lane] = acc;
            if (L) L[L_BND1_IN + lane] = acc;
        }
    };
    if (nets) stage_record(&s_N, nets + m);
    if (links) stage_record(&s_L, links + m);
    // barriers of the CTA and of the member's CTAs, reached from the roles' own code
    auto all = [] { bar_group(1, ENG_PRE_THREADS); };
    auto wide = [] { member_sync<G>(ENG_PRE_THREADS); };
    wide();                                      // records are staged, every CTA has started
    const bool multi = links && s_L.n_multi > 0;
    if (tid < ENG_EXCH_THREADS) {
        auto put_rate = [&](R r) {
            if constexpr (G > 1) {
                if (lane < G) {
                    const unsigned here = (unsigned)__cvta_generic_to_shared(&s_rate[rank * ENG_EXCH_WARPS + (tid >> 5)]);
                    unsigned there;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(here), "r"(lane));
                    if constexpr (sizeof(R) == 8)
                        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(there), "d"(r) : "memory");
                    else
                        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(there), "f"(r) : "memory");
                }
            } else {
                if (lane == 0) s_rate[tid >> 5] = r;
            }
        };
        auto ready = [&] { wide(); return s_dtr; };
        auto go = [&] { all(); return s_nsub <= max_sub; };
        if (links) {
            constexpr int NS = EXCH_SLICES / G;      // slices of this CTA
            static_assert(NS * G == EXCH_SLICES && ENG_EXCH_WARPS >= NS, "whole slices, a warp to each");
            exchange_dev<R, 1>(s_L, s_N, grids[m], K, nullptr, Vg + s_L.v_offset,
                            exch + (size_t)(m * EXCH_SLICES + rank * NS) * 2, rank * NS, NS, sm, tid,
                            ENG_EXCH_THREADS, true,
                            [] { bar_group(2, ENG_EXCH_THREADS); }, wide, ready, go, put_rate);
        } else {
            R rate = R(-1);
            if (nets)
                for (int i = rank * ENG_EXCH_THREADS + tid; i < s_N.n_cells; i += G * ENG_EXCH_THREADS) {
                    const CellLevel<R> o = cell_level(s_N, i, K.g, K.h_dry, true);
                    if (o.wet) rate = o.rate > rate ? o.rate : rate;
                }
            for (int o = 16; o > 0; o >>= 1) {
                const R w = __shfl_xor_sync(0xffffffffu, rate, o);
                rate = w > rate ? w : rate;
            }
            put_rate(rate);
            ready();
            go();
        }
        return;
    }
    const Grid<R>& gd = grids[m];
    if (tid < ENG_EXCH_THREADS + 32) {
        double rate = last.rate;
        if (TURN) {
            const int j[1] = {P_RATE};
            double s[1];
            sum_columns<1>(partials, gd.tile0, gd.n_tiles, j, s);
            rate = s[0];
        }
        const double t = last.t;
        bool clamped = false;
        if (lane == 0) {
            double dt = rate > 0.0 ? c.cfl / rate : c.dt_max;
            if (dt < c.dt_min || dt > c.dt_max) {
                clamped = dt < c.dt_min;
                dt = fmin(fmax(dt, c.dt_min), c.dt_max);
            }
            // the step ends at the member's end or its next output time (coupling.py:255-262)
            double limit = E.t_end;
            const bool out_on = E.n_out > 0 && last.k_out < E.n_out;
            const double t_next = out_on ? E.out_dt * last.k_out : 0.0;
            if (out_on) limit = fmin(limit, t_next);
            dt = fmin(dt, limit - t);
            s_dt = dt;
            s_dtr = (R)dt;
            s_t = t;
            s_snap = out_on && t + dt >= t_next - 1e-9 ? last.k_out : -1;
        }
        __syncwarp();
        wide();                                  // dt is chosen, the channel rates are in s_rate
        if (lane == 0) {
            int n = 0;
            if (nets) {
                R r1 = s_rate[0];
                for (int w = 1; w < G * ENG_EXCH_WARPS; ++w) r1 = s_rate[w] > r1 ? s_rate[w] : r1;
                const double dt1 = r1 >= R(0) ? fmin(c.cfl_1d / (double)r1, c.dt_max) : c.dt_max;
                const double ns = ceil(s_dt / dt1 - 1e-9);
                n = ns < 1.0 ? 1 : (ns > (double)max_sub ? max_sub + 1 : (int)ns);
            }
            const bool run = !TURN || s_status == ST_RUNNING;
            s_nsub = run ? n : max_sub + 1;
            if (rank == 0) {
                if (run && clamped) E.n_clamped++;
                if (TURN) {
                    out[(size_t)m * 8 + 5] = rate;
                    E.rate = rate;
                    E.t = t;
                    if (last.snap >= 0) {
                        E.snap_t[last.snap] = t;
                        E.k_out = last.k_out;
                    }
                    E.steps += 1;
                    E.n_sub_max = max(E.n_sub_max, last.n_sub);
                    E.dt_min = fmin(E.dt_min, last.dt);
                    E.dt_max = fmax(E.dt_max, last.dt);
                }
            }
        }
        __syncwarp();
        if (multi)                               // (the exchange's own barriers)
            for (int k = 0; k < 3; ++k) wide();
        all();                                   // the substep count is known
        if (rank != 0) {
            if (TURN) add_volumes(0);
            return;
        }
        const int n = s_nsub;
        if (n > max_sub) {
            if (lane == 0) {
                if (!TURN || s_status == ST_RUNNING) E.status = ST_SUBSTEPS;
                P.active = 0;
            }
            return;
        }
        const double sub = s_dt / n;
        for (int k = lane; k < n; k += 32) {
            const double tk = s_t + k * sub;
            netf[((size_t)m * max_sub + k) * 2 + 0] = eng_inflow(E, tk);
            netf[((size_t)m * max_sub + k) * 2 + 1] = eng_tide(E, tk);
        }
        return;
    }
    if (TURN) {
        const int j[3] = {P_HSUM, P_RATE, P_HMAX};
        double s[3];
        sum_columns<3>(partials, gd.tile0, gd.n_tiles, j, s);
        if (lane == 0) {
            int st = ST_RUNNING;
            if (!isfinite(s[0]) || !isfinite(s[1])) st = ST_NONFINITE;
            else if (s[2] > MAX_PLAUSIBLE_DEPTH_2D) st = ST_IMPLAUSIBLE;
            else if (last.t >= E.t_end - 1e-9) st = ST_DONE;
            s_status = st;
            if (rank == 0) E.status = st;
        }
    }
    wide();
    const double dt = s_dt;
    // edge values at t by lanes 0..3 and at t + dt by lanes 4..7, rain by lane 8
    double v = 0.0;
    if (rank != 0) v = 0.0;
    else if (lane < 8) v = eng_edge(E, lane & 3, lane < 4 ? s_t : s_t + dt);
    else if (lane == 8) v = eng_rain(E, s_t);
    __syncwarp();
    if (multi)
        for (int k = 0; k < 3; ++k) wide();
    all();
    if (rank != 0) {
        if (TURN) add_volumes(1);
        return;
    }
    if (s_nsub > max_sub) return;
    if (lane < 4) {
        P.bc0[lane] = v;
        P.bc0_f[lane] = (float)v;
    } else if (lane < 8) {
        P.bc1[lane & 3] = v;
        P.bc1_f[lane & 3] = (float)v;
    } else if (lane == 8) {
        P.rain = v;
        P.rain_f = (float)v;
    } else if (lane == 9) {
        P.dt = dt;
        P.t = s_t;
        P.dt_f = (float)dt;
        P.t_f = (float)s_t;
        E.dt = dt;
        E.n_sub = s_nsub;
        P.active = 1;
        const int k = s_snap;
        P.snap_k = k;
        P.snap_h = k >= 0 ? E.snap_h + (size_t)k * E.cells : nullptr;
        P.snap_u = k >= 0 ? E.snap_u + (size_t)k * E.cells : nullptr;
        P.snap_v = k >= 0 ? E.snap_v + (size_t)k * E.cells : nullptr;
        P.snap_eta = k >= 0 && E.snap_eta ? E.snap_eta + (size_t)k * E.n1d : nullptr;
        P.snap_q = k >= 0 && E.snap_q ? E.snap_q + (size_t)k * E.n1d : nullptr;
        P.snap_ledger = k >= 0 && E.snap_ledger ? E.snap_ledger + (size_t)k * LEDGER_N : nullptr;
    }
}

template <class R>
__global__ void __launch_bounds__(FIN_THREADS) eng_post_kernel(EngMember* __restrict__ em,
                                                               const StepParams* __restrict__ params,
                                                               const Grid<R>* __restrict__ grids, Consts c,
                                                               const double* __restrict__ partials,
                                                               const double* __restrict__ vol1d,
                                                               double* __restrict__ out, int m0) {
    __shared__ double S[NPART];
    const int m = m0 + blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (!params[m].active) return;
    const Grid<R>& gd = grids[m];
    sum_partials(partials, gd.tile0, gd.n_tiles, S);
    if (lane != 0) return;
    // one thread per accumulated term, clock and status on another: each in its own warp
    EngMember& E = em[m];
    const StepParams& pr = params[m];
    double* o = out + (size_t)m * 8;
    double* L = pr.snap_k >= 0 ? pr.snap_ledger : nullptr;      // the 1-D kernel writes L[L_V1D]
    const bool net = vol1d && E.n_sub > 0;
    if (warp <= 4) {
        const double v = step_term(warp, gd, pr.dt, pr.rain, c.order, S);
        o[warp] = v;
        const int a = warp == 0 ? 2 : warp == 1 ? 3 : warp == 2 ? 0 : warp == 3 ? 1 : 6;
        double acc = E.acc[a] + v;
        if (warp == 4 && net) acc += vol1d[m * 3 + 2];
        E.acc[a] = acc;
        if (L) L[L_RAIN + a] = acc;
    } else if (warp == 5) {
        for (int k = 0; k < 2; ++k) {
            const double acc = net ? E.acc[4 + k] + vol1d[m * 3 + k] : E.acc[4 + k];
            E.acc[4 + k] = acc;
            if (L) L[L_BND1_IN + k] = acc;
        }
    } else if (warp == 6) {
        const double v2 = S[P_HSUM] * gd.area, vs = S[P_SSUM] * gd.area;
        o[6] = v2;
        o[7] = vs;
        if (L) {
            L[L_V2D] = v2;
            L[L_STORE] = vs;
        }
        E.dt_min = fmin(E.dt_min, E.dt);
        E.dt_max = fmax(E.dt_max, E.dt);
    } else {
        o[5] = S[P_RATE];
        E.rate = S[P_RATE];
        const double t = E.t + E.dt;
        E.t = t;
        if (pr.snap_k >= 0) {
            E.snap_t[pr.snap_k] = t;
            E.k_out = pr.snap_k + 1;
        }
        E.steps += 1;
        E.n_sub_max = max(E.n_sub_max, E.n_sub);
        if (!isfinite(S[P_HSUM]) || !isfinite(S[P_RATE])) E.status = ST_NONFINITE;
        else if (S[P_HMAX] > MAX_PLAUSIBLE_DEPTH_2D) E.status = ST_IMPLAUSIBLE;
        else if (t >= E.t_end - 1e-9) E.status = ST_DONE;
    }
}

// Copy the rate of the current state (finalize output, mode 1) into the engine records.
static __global__ void eng_take_rate_kernel(EngMember* __restrict__ em, const double* __restrict__ out, int n) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < n) em[m].rate = out[(size_t)m * 8 + 5];
}

}  // namespace his
