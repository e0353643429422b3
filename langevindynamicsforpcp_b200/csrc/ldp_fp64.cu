// ldp_fp64.cu -- plain FP64 trajectory kernels: one trajectory per thread, and
// group mode (few trajectories), whose stepping lanes other warps draw the
// noise for.
//
// Device restatement of LangevinEquationSIMDMultiple and its overdamped
// subclass (src/langevinDynamicsSingleBarrier.h:823-2888) and of the
// double-barrier engine (src/langevinDynamicsDoubleBarrier.h:933-3507): the
// per-lane SIMD loop becomes one CUDA thread stepping each trajectory, the
// lane's __m512d registers become this thread's registers, and the lazily grown
// per-cell barrier table (src/DataLocator.h:100-188) becomes a tagged ring
// of visited cells in HBM whose never-visited entries are a pure function of
// (trajectory, cell).
//
// Compiled with -fmad=false: every a*b+c is two roundings unless written as
// fma(), as in the reference's intrinsics (the only fused step is the
// overdamped drift, _mmSIMD_fmadd_pd at S.h:2868).
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include "ldp_device.cuh"
#include "ldp_engine.h"

namespace ldp {

struct T64 {
    double x, v, F, E, rprev, barrier;
    int64_t cell, well;
    int lb, state;
    uint32_t bits;
    double fpt_last, fpt2_last, tpt_last, tpt2_last;
    int64_t init_idx0, init_idx1, idx2_0, idx2_1, tpt2_well, wt_tick;
};

template <bool DBL>
__device__ __forceinline__ int64_t cell_key(int64_t cell, int lb) {
    return DBL ? cell * 2 + lb : cell;
}

// State of a cell never entered: BarrierStatus::Initialize (S.h:78-96),
// drawn from the trajectory's TAG_CELL stream; with UNIFORMINITALSTATES the
// value the reference hands over (S.h:1377-1380, D.h:1576-1578).
template <bool DBL>
__device__ int default_state(const KConst& k, uint32_t g, int64_t ck) {
    if (k.us) {
        if (DBL) return k.init_state;
        const int64_t trial = ((int64_t)g / k.lanes) % k.nruns;
        if (trial == 0) return 0;
        if (!k.rs) return k.init_state;
        const Words w = philox_at(0, g - (uint32_t)k.lanes, TAG_INIT, k.key0, k.key1);
        return ((double)w.w0 * 0x1p-32 <= k.p_first) ? 0 : 1;
    }
    const Words w = philox_at((uint64_t)ck, g, TAG_CELL, k.key0, k.key1);
    return ((double)w.w0 * 0x1p-32 < k.p_cell0) ? 0 : 1;
}

template <bool DBL>
// A cell-table entry: the barrier's state when it was left and its pending
// flip step; *found false for a cell never visited (state as drawn at its
// creation, step 0).
__device__ __forceinline__ void ring_load(const KConst& k, const TrajState& st, int64_t i, uint32_t g, int64_t ck,
                                          int* state, int64_t* nflip, bool* found) {
    const int64_t slot = ck & (int64_t)(k.slots - 1);
    const int64_t o = slot * st.n + i;
    if (st.ring_tag[o] == ck) {
        const int64_t d = st.ring_data[o];
        *state = (int)(d & 1);
        *nflip = d >> 1;
        *found = true;
    } else {
        *state = default_state<DBL>(k, g, ck);
        *nflip = 0;
        *found = false;
    }
}

__device__ __forceinline__ void ring_store(const KConst& k, const TrajState& st, int64_t i, int64_t ck, int state,
                                           int64_t nflip) {
    const int64_t slot = ck & (int64_t)(k.slots - 1);
    const int64_t o = slot * st.n + i;
    const int64_t old = st.ring_tag[o];
    if (old != ck && old != INT64_MIN) st.counts[(int64_t)LDP_C_EVICT * st.n + i] += 1;
    st.ring_tag[o] = ck;
    st.ring_data[o] = (nflip << 1) | (int64_t)state;
}

// ring_store of the barrier left, then ring_load of the one entered, with all
// their loads issued together: one memory latency instead of three in a row.
template <bool DBL>
__device__ __forceinline__ void ring_swap(const KConst& k, const TrajState& st, int64_t i, uint32_t g, int64_t left,
                                          int state, int64_t nflip, int64_t ck, int* ps, int64_t* nb, bool* found) {
    const int64_t mask = (int64_t)(k.slots - 1);
    const int64_t o = (left & mask) * st.n + i, e = (ck & mask) * st.n + i;
    const int64_t old = st.ring_tag[o], tag = st.ring_tag[e], d = st.ring_data[e];
    if (old != left && old != INT64_MIN) st.counts[(int64_t)LDP_C_EVICT * st.n + i] += 1;
    st.ring_tag[o] = left;
    st.ring_data[o] = (nflip << 1) | (int64_t)state;
    *found = tag == ck && o != e;   // o == e: the entry stored just now, of another barrier
    *ps = *found ? (int)(d & 1) : default_state<DBL>(k, g, ck);
    *nb = *found ? d >> 1 : 0;
}

// EnergyAndForce, S.h:1292-1324 / D.h:1464-1522.
template <bool DBL>
__device__ __forceinline__ void energy_force(const KConst& k, T64& t) {
    const int s = t.state;
    const double xp = t.x - (double)t.cell * k.L;
    if (!DBL) {
        const double sp = k.slope[s], sn = 0.0 - sp, H = k.Hs[s];
        const bool onN = (xp < 0.0) && (xp > -k.w);
        const bool onP = (xp < k.w) && (xp > 0.0);
        double E = 0.0, F = 0.0;
        if (onN) { E = H - xp * sn; F = sn; }
        if (onP) { E = H - xp * sp; F = sp; }
        t.E = E;
        t.F = F;
        t.barrier = H;
    } else {
        const bool onN0 = (xp < k.xb[0]) && (xp > k.lo0);
        const bool onP0 = (xp < k.xc) && (xp > k.xb[0]);
        const bool onN1 = (xp < k.xb[1]) && (xp > k.xc);
        const bool onP1 = (xp < k.hi1) && (xp > k.xb[1]);
        double E = 0.0, f = 0.0, B = 0.0;
        if (onN0) { E = xp * k.sN[0][s] + k.iN[0][s]; f = k.sN[0][s]; B = k.Hd[0][s]; }
        if (onP0) { E = xp * k.sP[0][s] + k.iP[0][s]; f = k.sP[0][s]; B = k.Hd[0][s]; }
        if (onN1) { E = xp * k.sN[1][s] + k.iN[1][s]; f = k.sN[1][s]; B = k.Hd[1][s]; }
        if (onP1) { E = xp * k.sP[1][s] + k.iP[1][s]; f = k.sP[1][s]; B = k.Hd[1][s]; }
        t.E = E;
        t.F = 0.0 - f;
        t.barrier = B;
    }
}

// InitializePeriodicIndices / UpdatePeriodicIndices, S.h:1838-1884,
// D.h:2156-2235: well = floor(x/L), cell = rint(x/L) (ties to even),
// local barrier = (xp < xc) ? 0 : 1.
template <bool DBL>
__device__ __forceinline__ void indices(const KConst& k, T64& t) {
    const double red = t.x * k.invL;
    t.well = (int64_t)floor(red);
    t.cell = (int64_t)rint(red);
    if (DBL) {
        const double xp = t.x - (double)t.cell * k.L;
        t.lb = (xp < k.xc) ? 0 : 1;
    } else {
        t.lb = 0;
    }
}

template <bool DBL>
__device__ __forceinline__ int table_state(const KConst& k, const TrajState& st, int64_t i, uint32_t g,
                                           int64_t cell) {
    int s;
    int64_t nf;
    bool found;
    ring_load<DBL>(k, st, i, g, cell_key<DBL>(cell, 0), &s, &nf, &found);
    return s;
}

// Initial-barrier bookkeeping of the FPT statistic, S.h:2187-2211 and
// S.h:2364-2388; the two recorded states live in bits B_INIT0/B_INIT1.
template <bool DBL>
__device__ __forceinline__ void fpt_set_initial(const KConst& k, const TrajState& st, int64_t i, uint32_t g,
                                                T64& t) {
    int s0, s1;
    if (t.well == t.cell) {
        s0 = t.state;
        t.init_idx0 = t.cell;
        s1 = table_state<DBL>(k, st, i, g, t.cell + 1);
        t.init_idx1 = t.cell + 1;
    } else {
        s0 = table_state<DBL>(k, st, i, g, t.cell - 1);
        t.init_idx0 = t.cell - 1;
        s1 = t.state;
        t.init_idx1 = t.cell;
    }
    t.bits = (t.bits & ~(B_INIT0 | B_INIT1)) | (s0 ? B_INIT0 : 0u) | (s1 ? B_INIT1 : 0u);
}

__device__ __forceinline__ void fpt2_set_idx(T64& t) {
    if (t.well == t.cell) { t.idx2_0 = t.cell; t.idx2_1 = t.cell + 1; }
    else { t.idx2_0 = t.cell - 1; t.idx2_1 = t.cell; }
}

__device__ __forceinline__ bool cg_hit(int64_t well, int size) { return ((int)well % size) == 0; }

// Appends an event duration to list `list` of trajectory i (the reference's
// push_back on its per-lane vectors, S.h:2391, 2447, 2504, 2524, 2580); c is
// the list's count before the event.  A full list flags the trajectory.
__device__ __noinline__ uint32_t ev_push(const KConst& k, const TrajState& st, int list, int64_t i, int64_t c,
                                         double d) {
    if (c >= k.ev_cap) return LDP_FLAG_EVENT_OVERFLOW;
    st.ev[((int64_t)list * st.n + i) * k.ev_cap + c] = d;
    return 0u;
}

__device__ __forceinline__ void record(const KConst& k, const TrajState& st, const T64& t, int64_t i,
                                       int64_t frame) {
    if (frame >= k.nframe) return;   // the frame arrays hold nframe rows
    const int64_t o = frame * st.n + i;
    if (st.fx) st.fx[o] = t.x;
    if (k.write_x) {
        if (st.fv) st.fv[o] = t.v;
        if (st.ff) st.ff[o] = t.F;
        if (st.fb) st.fb[o] = t.barrier;
        if (st.fpe) st.fpe[o] = t.E;
        if (st.fke) st.fke[o] = k.mhalf * (t.v * t.v);
        if (st.fst) st.fst[o] = (double)t.state;
    }
}

__device__ __forceinline__ void store_traj(const TrajState& st, const T64& t, int64_t i) {
    st.x[i] = t.x; st.v[i] = t.v; st.F[i] = t.F; st.rprev[i] = t.rprev;
    st.cell[i] = t.cell; st.well[i] = t.well; st.state[i] = t.state; st.lb[i] = t.lb; st.bits[i] = (int32_t)t.bits;
    st.fpt_last[i] = t.fpt_last; st.fpt2_last[i] = t.fpt2_last; st.tpt_last[i] = t.tpt_last;
    st.tpt2_last[i] = t.tpt2_last;
    st.init_idx0[i] = t.init_idx0; st.init_idx1[i] = t.init_idx1; st.idx2_0[i] = t.idx2_0; st.idx2_1[i] = t.idx2_1;
    st.tpt2_well[i] = t.tpt2_well; st.wt_tick[i] = t.wt_tick;
}

__device__ __forceinline__ void load_traj(const TrajState& st, T64& t, int64_t i) {
    t.x = st.x[i]; t.v = st.v[i]; t.F = st.F[i]; t.rprev = st.rprev[i];
    t.cell = st.cell[i]; t.well = st.well[i]; t.state = st.state[i]; t.lb = st.lb[i]; t.bits = (uint32_t)st.bits[i];
    t.fpt_last = st.fpt_last[i]; t.fpt2_last = st.fpt2_last[i]; t.tpt_last = st.tpt_last[i];
    t.tpt2_last = st.tpt2_last[i];
    t.init_idx0 = st.init_idx0[i]; t.init_idx1 = st.init_idx1[i]; t.idx2_0 = st.idx2_0[i]; t.idx2_1 = st.idx2_1[i];
    t.tpt2_well = st.tpt2_well[i]; t.wt_tick = st.wt_tick[i];
    t.E = 0.0; t.barrier = 0.0;
}

// IntegrateStep0 (S.h:1619-1652, overdamped S.h:2825-2832; D.h:1938-1971)
// with InitializeBarrierState (S.h:1885-1915) and InitializeStatistics
// (S.h:2166-2333, D.h:2759-2930).
template <bool DBL, bool OVER>
__global__ void __launch_bounds__(128) fp64_init_kernel(const KConst k, const TrajState st, int64_t g0) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= st.n) return;
    const uint32_t g = (uint32_t)(g0 + i);
    for (int s = 0; s < k.slots; ++s) {
        st.ring_tag[(int64_t)s * st.n + i] = INT64_MIN;
        st.ring_data[(int64_t)s * st.n + i] = 0;
    }
    for (int f = 0; f < LDP_NCOUNT; ++f) st.counts[(int64_t)f * st.n + i] = 0;
    for (int f = 0; f < LDP_NSUM; ++f) st.sums[(int64_t)f * st.n + i] = 0.0;

    T64 t;
    t.x = k.x0;
    t.v = 0.0; t.F = 0.0; t.E = 0.0; t.rprev = 0.0; t.barrier = 0.0;
    t.bits = 0;
    t.fpt_last = t.fpt2_last = t.tpt_last = t.tpt2_last = 0.0;
    t.init_idx0 = t.init_idx1 = t.idx2_0 = t.idx2_1 = 0;
    t.wt_tick = 0;
    indices<DBL>(k, t);
    const Words w0 = philox_at(0, g, TAG_INIT, k.key0, k.key1);
    t.state = k.rs ? (((double)w0.w0 * 0x1p-32 <= k.p_first) ? 0 : 1) : k.init_state;
    st.state0[i] = t.state;
    st.counts[(int64_t)(t.state ? LDP_C_STATE1 : LDP_C_STATE0) * st.n + i] = 1;
    double zv, zr;
    gauss_pair_f64(w0.w1, w0.w2, &zv, &zr);
    t.v = k.rv ? k.sig_v0 * zv : k.v0;
    st.v0[i] = t.v;
    {
        // waiting time to the initial barrier's first flip
        const Words wf = philox_at(0, g, TAG_FLIP, k.key0, k.key1);
        st.nflip[i] = flip_schedule(0, wf.w0, wf.w1, k.ln1m[t.state]);
    }
    energy_force<DBL>(k, t);
    if (k.at_bottom) {
        if (!DBL && k.fpt) fpt_set_initial<DBL>(k, st, i, g, t);
        fpt2_set_idx(t);
    } else {
        t.bits |= B_FPT_UP | B_FPT2_UP;
    }
    if (!k.at_bottom) t.bits |= B_TPT_UP | B_TPT2_UP;
    t.tpt2_well = t.well;
    for (int j = 0; j < k.n_cg; ++j) {
        st.cg_last[(int64_t)j * st.n + i] = 0.0;
        st.cg_well[(int64_t)j * st.n + i] = t.well;
        if (!(k.at_bottom && cg_hit(t.well, k.cg_size[j]))) t.bits |= (B_CG0 << j);
    }
    if (OVER) t.rprev = k.sig_r * zr;
    if (!k.fp_mode) record(k, st, t, i, 0);
    store_traj(st, t, i);
}

// Where a step's flip schedule comes from.  FlipDraw draws it on the spot
// (the TAG_FLIP words at the flip step, geometric waiting time in FP64) and
// hands the words on, so that a cell entry at the same step reuses them.
struct FlipDraw {
    __device__ __forceinline__ int64_t schedule(const KConst& k, uint32_t g, uint64_t s, int state, Words* wf,
                                                bool* have) const {
        *wf = philox_at(s, g, TAG_FLIP, k.key0, k.key1);
        *have = true;
        return flip_schedule(s, wf->w0, wf->w1, k.ln1m[state]);
    }
};

// One step s of a trajectory (Integrate's loop body, S.h:1403-1511):
// IntegrateStepEta / IntegrateStep (S.h:1654-1706, 2833-2886; D.h:1973-2024,
// 3448-3505) followed by UpdateStatistics (S.h:2334-2592, D.h:2931-3209).
// src supplies the flip schedule of a flip at s.  Returns 0 to continue, 1
// when the trajectory stops before completing s (non-finite position), 2 when
// it stops after s (first passage reached).
//
// The position (and velocity) update of a step, IntegrateStepEta's first
// part (S.h:1680-1695, 2860-2870).  rf: the step's noise, its Gaussian times
// sig_r (overdamped) or sig_v.
template <bool OVER>
__device__ __forceinline__ void fp64_move(const KConst& k, T64& t, double rf) {
    if (OVER) {
        t.x = fma(t.F, k.c_drift, t.x);
        t.x = t.x + rf;
        t.x = t.x + t.rprev;
        t.rprev = rf;
    } else {
        t.v = t.v + (k.invM * t.F) * k.hdt;
        t.x = t.x + t.v * k.hdt;
        t.v = k.expg * t.v + rf;
        t.x = t.x + t.v * k.hdt;
    }
}

// A barrier in state `state` whose flip at step `base` was missed, entered
// at step s: its state then (S.h:2025-2068) and its new pending flip.
__device__ __forceinline__ void catch_up(const KConst& k, uint32_t g, uint64_t s, int64_t base, int state,
                                         const Words* wf, int* now, int64_t* nflip) {
    const double lap = (double)((int64_t)s - base);
    const double pl = k.c_lap[k.eq ? 0 : state] * -expm1_f64(k.a_lap * lap);
    const uint64_t Tl = prob_to_u64(pl);
    const Words wc = philox_at(s, g, TAG_CATCHUP, k.key0, k.key1);
    const uint64_t U = ((uint64_t)wc.w0 << 32) | wc.w1;
    *now = (U < Tl) ? (state ^ 1) : state;
    *nflip = flip_schedule(s, wf->w2, wf->w3, k.ln1m[*now]);
}

// The barrier (cell, or in the double model local barrier) that a step left:
// its state and pending flip, as stored in the cell table.
struct LeftKey {
    int64_t nflip;
    int state;
};

// The rest of step s after fp64_move: indices, barrier flips and cell
// entries, the state count, the force and the statistics (the frame is the
// caller's).  cell_prev, well_prev, lb_prev: the indices before the move; lk:
// the barrier left, when one was.
template <bool DBL, bool OVER, bool ETA, class Src>
__device__ __forceinline__ int fp64_after_move(const KConst& k, const TrajState& st, int64_t i, uint32_t g, T64& t,
                                               uint64_t s, const Src& src, int64_t& nflip, int64_t& sc1,
                                               uint32_t& flags, int64_t cell_prev, int64_t well_prev, int lb_prev,
                                               LeftKey& lk) {
    const int64_t n = st.n;
    if (!isfinite(t.x)) {
        flags |= LDP_FLAG_NONFINITE;
        t.bits |= B_DONE;
        return 1;
    }
    indices<DBL>(k, t);
    const bool dWell = t.well != well_prev;
    const bool dCell = t.cell != cell_prev;
    const bool dKey = DBL ? (t.lb != lb_prev) : dCell;

    if (ETA) {
        // UpdateBarrierStateEta, S.h:1998-2153 / D.h:2435-2736, with
        // every barrier's flips on a schedule (geometric waiting times of
        // the per-step Bernoulli flips): the current barrier flips at its
        // pending flip step; a barrier left keeps its pending flip in the
        // cell table; one re-entered before that step has not flipped
        // meanwhile (no draw); one whose flip came while it was away (or
        // never visited: created at step 0) is caught up from that step
        // with the two-state transition probability (S.h:2025-2068).
        const bool flip = (int64_t)s == nflip;
        Words wf{};
        bool have_wf = false;
        if (flip) {
            t.state ^= 1;
            nflip = src.schedule(k, g, s, t.state, &wf, &have_wf);
        }
        if (dKey) {
            lk = LeftKey{nflip, t.state};
            int ps;
            int64_t nb;
            bool found;
            ring_swap<DBL>(k, st, i, g, cell_key<DBL>(cell_prev, lb_prev), t.state, nflip,
                           cell_key<DBL>(t.cell, t.lb), &ps, &nb, &found);
            if (found && nb > (int64_t)s) {
                t.state = ps;
                nflip = nb;
            } else {
                if (!have_wf) wf = philox_at(s, g, TAG_FLIP, k.key0, k.key1);
                catch_up(k, g, s, found ? nb : 0, found ? (ps ^ 1) : ps, &wf, &t.state, &nflip);
            }
        }
    } else {
        // UpdateBarrierState (TAU == 0), S.h:1933-1997 / D.h:2299-2434.
        if (dKey) {
            lk = LeftKey{nflip, t.state};
            int ps;
            int64_t nb;
            bool found;
            ring_swap<DBL>(k, st, i, g, cell_key<DBL>(cell_prev, lb_prev), t.state, nflip,
                           cell_key<DBL>(t.cell, t.lb), &ps, &nb, &found);
            t.state = ps;
        }
    }
    sc1 += t.state;   // UpdateBarrierStateEtaParamter
    energy_force<DBL>(k, t);
    if (!OVER) t.v = t.v + (k.invM * t.F) * k.hdt;

    // UpdateStatistics.
    if (dWell || dCell) {
        const double now = k.dt * (double)s;
        if (!DBL && k.wt && !k.fp_mode) {
            if (dWell) { t.wt_tick = (int64_t)s; t.bits |= B_WT_PASSED; }
            else if (dCell && (t.bits & B_WT_PASSED)) {
                int64_t& nwt = st.counts[(int64_t)LDP_C_WT * n + i];
                if (nwt < k.tick_cap) st.ticks[i * k.tick_cap + nwt] = t.wt_tick;
                else flags |= LDP_FLAG_TICK_OVERFLOW;
                nwt += 1;
                t.bits &= ~B_WT_PASSED;
            }
        }
        if (k.fpt || k.fp_mode) {
            if (!DBL && !k.fp_mode) {
                if ((t.bits & B_FPT_UP) && dCell) {
                    t.bits &= ~B_FPT_UP;
                    t.fpt_last = now;
                    fpt_set_initial<DBL>(k, st, i, g, t);
                }
                if (!(t.bits & B_FPT_UP) && dWell) {
                    t.bits |= B_FPT_UP;
                    const int64_t c = st.counts[(int64_t)LDP_C_FPT * n + i];
                    if (c == 0) st.sums[(int64_t)LDP_S_FIRST_FPT * n + i] = now - t.fpt_last;
                    st.sums[(int64_t)LDP_S_FPT * n + i] += now - t.fpt_last;
                    st.counts[(int64_t)LDP_C_FPT * n + i] = c + 1;
                    const bool ib = ((double)t.cell == (double)t.init_idx0) ? ((t.bits & B_INIT0) != 0)
                                                                            : ((t.bits & B_INIT1) != 0);
                    if (k.ev_cap) {
                        flags |= ev_push(k, st, LDP_E_FPT, i, c, now - t.fpt_last);
                        if (c < k.ev_cap) st.ev_st[i * k.ev_cap + c] = (uint8_t)((t.state ? 1 : 0) | (ib ? 2 : 0));
                    }
                    st.counts[(int64_t)(ib ? LDP_C_INIT1 : LDP_C_INIT0) * n + i] += 1;
                    st.counts[(int64_t)(t.state ? LDP_C_INST1 : LDP_C_INST0) * n + i] += 1;
                }
            }
            if ((t.bits & B_FPT2_UP) && dCell) {
                t.bits &= ~B_FPT2_UP;
                t.fpt2_last = now;
                fpt2_set_idx(t);
            }
            if (dCell && !(t.bits & B_FPT2_UP) && t.idx2_0 != t.cell && t.idx2_1 != t.cell) {
                const int64_t c = st.counts[(int64_t)LDP_C_FPT2 * n + i];
                if (c == 0) st.sums[(int64_t)LDP_S_FIRST_FPT2 * n + i] = now - t.fpt2_last;
                st.sums[(int64_t)LDP_S_FPT2 * n + i] += now - t.fpt2_last;
                st.counts[(int64_t)LDP_C_FPT2 * n + i] = c + 1;
                if (k.ev_cap) flags |= ev_push(k, st, LDP_E_FPT2, i, c, now - t.fpt2_last);
                t.fpt2_last = now;
                fpt2_set_idx(t);
                if (k.fp_mode) t.bits |= B_DONE;   // first passage reached
            }
        }
        if (!DBL && k.tpt && !k.fp_mode) {
            if (dCell) { t.bits &= ~B_TPT_UP; t.tpt_last = now; }
            if (!(t.bits & B_TPT_UP) && dWell) {
                t.bits |= B_TPT_UP;
                const int64_t c = st.counts[(int64_t)LDP_C_TPT * n + i];
                if (c == 0) st.sums[(int64_t)LDP_S_FIRST_TPT * n + i] = now - t.tpt_last;
                st.sums[(int64_t)LDP_S_TPT * n + i] += now - t.tpt_last;
                st.counts[(int64_t)LDP_C_TPT * n + i] = c + 1;
                if (k.ev_cap) flags |= ev_push(k, st, LDP_E_TPT, i, c, now - t.tpt_last);
            }
            if (dCell) {
                if (t.bits & B_TPT2_UP) t.bits &= ~B_TPT2_UP;
                else if (t.well != t.tpt2_well) {
                    const int64_t c = st.counts[(int64_t)LDP_C_TPT2 * n + i];
                    if (c == 0) st.sums[(int64_t)LDP_S_FIRST_TPT2 * n + i] = now - t.tpt2_last;
                    st.sums[(int64_t)LDP_S_TPT2 * n + i] += now - t.tpt2_last;
                    st.counts[(int64_t)LDP_C_TPT2 * n + i] = c + 1;
                    if (k.ev_cap) flags |= ev_push(k, st, LDP_E_TPT2, i, c, now - t.tpt2_last);
                }
                t.tpt2_last = now;
                t.tpt2_well = t.well;
            }
        }
        if (k.cg && !k.fp_mode && dCell) {
            for (int jj = 0; jj < k.n_cg; ++jj) {
                if (cg_hit(t.well, k.cg_size[jj])) {
                    const int64_t o = (int64_t)jj * n + i;
                    if (t.bits & (B_CG0 << jj)) {
                        t.bits &= ~(B_CG0 << jj);
                        st.cg_last[o] = now;
                        st.cg_well[o] = t.well;
                    } else if (t.well != st.cg_well[o]) {
                        st.sums[(int64_t)(LDP_S_CG0 + jj) * n + i] += now - st.cg_last[o];
                        const int64_t c = st.counts[(int64_t)(LDP_C_CG0 + jj) * n + i];
                        st.counts[(int64_t)(LDP_C_CG0 + jj) * n + i] = c + 1;
                        if (k.ev_cap) flags |= ev_push(k, st, LDP_E_CG0 + jj, i, c, now - st.cg_last[o]);
                        st.cg_last[o] = now;
                        st.cg_well[o] = t.well;
                    }
                }
            }
        }
    }
    if (t.bits & B_DONE) return 2;
    return 0;
}

// The open interval of positions (absolute x) in which a step cannot change
// the cell, the well, the local barrier or the force: the interval between
// the breakpoints of energy_force (and indices) around the current
// cell-local position -- the cell edges, the barrier top 0, the flanks --
// shrunk at both ends by a margin, 1e-9 (1 + |x|), far above the rounding of
// x * invL and x - cell * L (~2e-16 |x|), so that for x inside it the full
// step would compute the same indices and force.  Empty (lo > hi) when x is
// within the margin of a breakpoint.
template <bool DBL>
__device__ __forceinline__ void quiet_band(const KConst& k, const T64& t, double* lo, double* hi) {
    const double cL = (double)t.cell * k.L;
    const double xp = t.x - cL;
    const double hL = 0.5 * k.L;
    double l = -hL, h = hL;
    auto cut = [&](double b) {
        if (b > -hL && b < hL) {
            if (b <= xp) l = fmax(l, b);
            if (b >= xp) h = fmin(h, b);
        }
    };
    cut(0.0);
    if (!DBL) {
        cut(0.0 - k.w);
        cut(k.w);
    } else {
        cut(k.lo0);
        cut(k.xb[0]);
        cut(k.xc);
        cut(k.xb[1]);
        cut(k.hi1);
    }
    const double m = 1e-9 * (1.0 + fabs(cL) + fabs(t.x));
    *lo = cL + l + m;
    *hi = cL + h - m;
}

// The force energy_force gives at the current position for either barrier
// state (constant over the quiet band).
template <bool DBL>
__device__ __forceinline__ void band_forces(const KConst& k, const T64& t, double* f0, double* f1) {
    T64 a = t;
    a.state = 0;
    energy_force<DBL>(k, a);
    *f0 = a.F;
    a.state = 1;
    energy_force<DBL>(k, a);
    *f1 = a.F;
}

// ---------------------------------------------------------------------------
// Steps of a lane
//
// A lane steps one trajectory; all lanes of a launch are at the same step.
// Steps are taken in blocks without a test between them (quiet_moves): they
// stand when the position stayed in the quiet band and, with rare flips, no
// flip was pending in the block.  The lanes whose block does not stand take
// its steps one by one (take_steps): quiet; quick (the flank of the barrier
// entered or left, or the edge between the cells of a pair crossed); or full
// (fp64_after_move).  Same operations on the same values in every case, so
// the results are those of full steps throughout, bit for bit.
// ---------------------------------------------------------------------------
enum : uint32_t {
    Q_PAIR = 1,    // the lane's cell and a neighbour are a pair: see full_step
    Q_RIGHT = 2,   // ... the right neighbour
    Q_TAGGED = 4,  // the cell table has an entry of the lane's cell
    Q_RUN = 8,     // the trajectory goes on
    Q_FORCE = 16   // the quiet band has a force in some state
};

struct Lane {
    T64 t;
    double mid, bF0, bF1;   // quiet band: its middle, the force in it for either state
    int half;               // ... high word of its half width (0: empty)
    int pstate;             // the pair's other barrier: state ...
    int64_t pnflip;         // ... and pending flip
    int64_t nflip, sc1;
    uint32_t q, flags;
};

// |x - mid| below the band's half width, by the high words: true only when it
// is (NaN and infinity are not).
__device__ __forceinline__ int off_band(const Lane& a, double x) {
    return __double2hiint(x - a.mid) & 0x7fffffff;
}

template <bool DBL>
__device__ __forceinline__ void set_band(const KConst& k, Lane& a, double mid, int half) {
    a.mid = mid;
    a.half = half;
    band_forces<DBL>(k, a.t, &a.bF0, &a.bF1);
    a.q = (a.q & ~Q_FORCE) | (a.bF0 != 0.0 || a.bF1 != 0.0 ? Q_FORCE : 0u);
}

template <bool DBL>
__device__ __forceinline__ void open_band(const KConst& k, Lane& a) {
    double lo, hi;
    quiet_band<DBL>(k, a.t, &lo, &hi);
    const double h = 0.5 * (hi - lo);
    set_band<DBL>(k, a, 0.5 * (lo + hi), (h > 0.0) ? __double2hiint(h) : 0);
}

template <bool DBL, bool OVER>
__device__ __forceinline__ void load_lane(const KConst& k, const TrajState& st, int64_t i, bool mine, Lane& a) {
    a.q = 0;
    a.flags = 0;
    a.half = 0;
    a.mid = a.bF0 = a.bF1 = 0.0;
    a.pstate = 0;
    a.pnflip = a.nflip = a.sc1 = 0;
    a.t = T64{};
    if (!mine) return;
    load_traj(st, a.t, i);
    if (a.t.bits & B_DONE) return;
    a.q = Q_RUN;
    a.sc1 = st.counts[(int64_t)LDP_C_STATE1 * st.n + i];
    a.nflip = st.nflip[i];
    energy_force<DBL>(k, a.t);   // not stored between launches
}

// s: the first step not integrated; before: the launch's first.
__device__ __forceinline__ void store_lane(const KConst& k, const TrajState& st, int64_t i, const Lane& a, uint64_t s,
                                           uint64_t before, uint64_t s_end) {
    const int64_t n = st.n;
    const int64_t sc1 = st.counts[(int64_t)LDP_C_STATE1 * n + i];
    st.counts[(int64_t)LDP_C_STATE1 * n + i] = a.sc1;
    st.counts[(int64_t)LDP_C_STATE0 * n + i] += (int64_t)(s - before) - (a.sc1 - sc1);
    st.counts[(int64_t)LDP_C_STEPS * n + i] = (int64_t)s - 1;
    uint32_t flags = a.flags;
    if (k.fp_mode && !(a.t.bits & B_DONE) && s_end > k.step_cap) flags |= LDP_FLAG_CENSORED;
    if (flags) st.counts[(int64_t)LDP_C_FLAGS * n + i] |= (int64_t)flags;
    st.nflip[i] = a.nflip;
    store_traj(st, a.t, i);
}

// A full step after its move.  When it crossed a cell edge and no statistic
// is left waiting for a crossing, the cell left and the cell entered are a
// pair: crossing their edge again, in this well, changes the barrier and
// restarts the transition clocks, and nothing else, as long as the well stays
// the same (the other barrier caught up when its pending flip has come).
template <bool DBL, bool OVER, bool ETA, class Src>
__device__ __forceinline__ int full_step(const KConst& k, const TrajState& st, int64_t i, uint32_t g, Lane& a,
                                         uint64_t s, const Src& src) {
    const int64_t cell = a.t.cell, well = a.t.well;
    const int lb = a.t.lb;
    LeftKey lk{};
    const int r = fp64_after_move<DBL, OVER, ETA>(k, st, i, g, a.t, s, src, a.nflip, a.sc1, a.flags, cell, well, lb,
                                                  lk);
    a.q &= Q_RUN;
    if (r) {
        a.q = 0;
        a.half = 0;
        return r;
    }
    open_band<DBL>(k, a);
    const int64_t d = cell - a.t.cell;
    if ((d == 1 || d == -1) && a.t.well == well && (!DBL || a.t.lb != lb)) {
        const bool fpt = !DBL && k.fpt && !k.fp_mode, fpt2 = k.fpt || k.fp_mode;
        const bool ok = !(fpt && (a.t.bits & B_FPT_UP)) &&
                        !(fpt2 && ((a.t.bits & B_FPT2_UP) || a.t.idx2_0 != well || a.t.idx2_1 != well + 1)) &&
                        !(!DBL && k.wt && !k.fp_mode && (a.t.bits & B_WT_PASSED));
        if (ok) {
            a.q |= Q_PAIR | (d == 1 ? Q_RIGHT : 0u);
            a.pstate = lk.state;
            a.pnflip = lk.nflip;
        }
    }
    return 0;
}

// A quick step after its move and the barrier's flip; false when the step must
// be a full one.
template <bool DBL, bool ETA>
__device__ __forceinline__ bool quick_step(const KConst& k, const TrajState& st, int64_t i, uint32_t g, Lane& a,
                                           uint64_t s) {
    T64& t = a.t;
    const bool right = t.well == t.cell;   // the half of the cell
    const double hL = 0.5 * k.L, m = 1e-8 * (1.0 + fabs(t.x));   // beyond quiet_band's margins
    const double xp = t.x - (double)t.cell * k.L;
    if (!(fabs(xp) < k.L)) return false;   // not finite, or far
    const bool leaves = right ? xp > hL : xp < -hL;
    if (!leaves) {
        // inside the cell: the same half and local barrier
        if (!(right ? xp > m : xp < -m)) return false;
        if (DBL && (t.lb ? !(xp > k.xc + m) : !(xp < k.xc - m))) return false;
    } else {
        if (!(a.q & Q_PAIR) || ((a.q & Q_RIGHT) != 0u) != right) return false;
        t.cell += right ? 1 : -1;
        if (DBL) t.lb ^= 1;
    }
    double lo, hi;
    quiet_band<DBL>(k, t, &lo, &hi);
    bool ok = t.x > lo && t.x < hi;
    if (leaves) {
        const double xn = t.x - (double)t.cell * k.L;
        ok = ok && (right ? xn < -m : xn > m) && (!DBL || (t.lb ? xn > k.xc + m : xn < k.xc - m));
        const int64_t left = t.cell - (right ? 1 : -1);
        if (!ok) {
            t.cell = left;
            if (DBL) t.lb ^= 1;
            return false;
        }
        const int64_t ck = cell_key<DBL>(left, t.lb ^ 1);
        const int64_t o = (ck & (int64_t)(k.slots - 1)) * st.n + i;
        if (a.q & Q_TAGGED) st.ring_data[o] = (a.nflip << 1) | (int64_t)t.state;
        else ring_store(k, st, i, ck, t.state, a.nflip);
        const int st0 = t.state;
        const int64_t nf = a.nflip;
        if (ETA && a.pnflip <= (int64_t)s) {
            const Words wf = philox_at(s, g, TAG_FLIP, k.key0, k.key1);
            catch_up(k, g, s, a.pnflip, a.pstate ^ 1, &wf, &t.state, &a.nflip);
        } else {
            t.state = a.pstate;
            a.nflip = a.pnflip;
        }
        a.pstate = st0;
        a.pnflip = nf;
        a.q = (a.q ^ Q_RIGHT) | Q_TAGGED;
        if (!DBL && k.tpt && !k.fp_mode) {
            const double now = k.dt * (double)s;
            t.bits &= ~(B_TPT_UP | B_TPT2_UP);
            t.tpt_last = now;
            t.tpt2_last = now;
            t.tpt2_well = t.well;
        }
    }
    if (!ok) return false;
    set_band<DBL>(k, a, 0.5 * (lo + hi), __double2hiint(0.5 * (hi - lo)));
    t.F = t.state ? a.bF1 : a.bF0;
    a.sc1 += t.state;
    return true;
}

// The rest of a lane's step s after its move, when it is not a quiet step
// (off: the position is outside the band).
template <bool DBL, bool OVER, bool ETA, class Src>
__device__ __forceinline__ void special_step(const KConst& k, const TrajState& st, int64_t i, uint32_t g, Lane& a,
                                             uint64_t s, bool off, const Src& src) {
    const int64_t nflip = a.nflip;
    const bool flip = ETA && (int64_t)s == nflip;
    if (flip) {
        a.t.state ^= 1;
        Words wf;
        bool have = false;
        a.nflip = src.schedule(k, g, s, a.t.state, &wf, &have);
    }
    if (!off) {
        // the current barrier's flip and nothing else
        a.t.F = a.t.state ? a.bF1 : a.bF0;
        a.sc1 += a.t.state;
    } else if (!quick_step<DBL, ETA>(k, st, i, g, a, s)) {
        if (flip) {   // as before the flip: a full step takes it too
            a.t.state ^= 1;
            a.nflip = nflip;
        }
        full_step<DBL, OVER, ETA>(k, st, i, g, a, s, src);
        return;   // the velocity's second half-kick included
    }
    if (!OVER) a.t.v = a.t.v + (k.invM * a.t.F) * k.hdt;
}

// N steps from the band, rf[m] their noise; true and the lane (one that wants
// to) moved on when they stand.  FLAT: no lane of the warp has a force (fma(0, c, x) is x).
template <bool OVER, bool FLAT, int N>
__device__ __forceinline__ bool quiet_moves(const KConst& k, Lane& a, bool want, const double* rf) {
    double x = a.t.x;
    int far = 0;
    if (OVER) {
        double r = a.t.rprev;
#pragma unroll
        for (int m = 0; m < N; ++m) {
            if (!FLAT) x = fma(a.t.F, k.c_drift, x);
            x = x + rf[m];
            x = x + r;
            r = rf[m];
            far = max(far, off_band(a, x));
        }
        want = want && far < a.half;
        if (want) {
            a.t.x = x;
            a.t.rprev = r;
        }
    } else {
        const double kick = (k.invM * a.t.F) * k.hdt;
        double v = a.t.v;
#pragma unroll
        for (int m = 0; m < N; ++m) {
            v = v + kick;
            x = x + v * k.hdt;
            v = k.expg * v + rf[m];
            x = x + v * k.hdt;
            v = v + kick;
            far = max(far, off_band(a, x));
        }
        want = want && far < a.half;
        if (want) {
            a.t.x = x;
            a.t.v = v;
        }
    }
    if (want) a.sc1 += N * a.t.state;
    return want;
}

// ---------------------------------------------------------------------------
// Group mode
//
// What bounds a run of few trajectories is the chain of a step, not the GPU:
// a Gaussian alone (Philox rounds, the FP64 logarithm and sincos, a square
// root) takes ~1000 cycles in one thread.  So the noise is drawn ahead by
// other warps: a CTA has nc consumer warps, T lanes of each stepping a
// trajectory, and producer warps that draw the noise of the CTA's M = nc T
// trajectories, B steps a buffer, one Philox block and two Box-Muller pairs
// for four steps of a trajectory.  A consumer's chain of a quiet step is then
// two additions (three operations where there is a force).  Two buffers
// alternate; four named barriers ("full" and "empty" of either) over a
// consumer warp and its producer warps hand them over, every arrival matched
// by one wait, with no spin loop.  Each consumer warp has its own: with the
// CTA's four on common barriers each waits for the slowest at every buffer
// (900 double-barrier trajectories 6.65 / 5.19 ms).
//
// T is chosen so that every scheduler of the GPU has one consumer warp
// (launch_fp64_group): a warp waits for each of its lanes' special steps, so
// fewer lanes a warp step faster.  TWO: two consumer warps a scheduler, of half
// as many lanes, in two CTAs an SM.  Overdamped steps (two or three FP64
// operations in a row) leave a scheduler to the other warp; underdamped ones
// (five, and more instructions) do not, and with frequent flips and eight
// lanes a warp the fewer producers count.  One / two, ms for 24000 steps: 900
// trajectories of two barriers 2.67 / 2.03, rare flips 1.54 / 1.35, 2000 3.42 /
// 2.93 and 1.79 / 1.63; 8000 6.33 / 6.52 and 3.03 / 2.64; underdamped 900 1.25 /
// 1.34, 5003 1.48 / 1.87.
//
// Within a buffer each lane is at its own step: after a special step it goes
// on with a new block of kGrpSteps steps, so a special step costs its warp
// itself and the steps walked up to it (1000-1800 cycles in all), not the
// block's remaining steps one by one as well (5000).
//
// DENSE: barriers flip so often that a lane could not draw its flips as they
// come.  Producers (with one trajectory per thread, the thread) then also draw
// the wait of a flip at every step for both states (its TAG_FLIP words, one
// logarithm), in 16 bits: -ln(2^-64) / -ln(1 - p) < 2^16 for p >= 1/1024.  A
// flip drawn by the consumer costs its warp ~1000 cycles, the waits of all
// steps ~25 cycles a step and a longer chain in the block: dense from
// p T = 1/40 on.
//
// What it measured (ns a step; one CTA a trajectory, or of 32 trajectories,
// with a producer warp or four, flips drawn for every step / this): the
// sample input, 32 trajectories, p = 1/2, a frame in 80 steps: 62.7 / 38.1;
// 900 of two barriers, a frame in 50: 199 / 61; rare flips, a frame in 20,
// 592: 135 / 53, 2000: 481 / 68, 16000: 575 / 150; 5003 underdamped, a frame
// in 30: 235 / 56.
// ---------------------------------------------------------------------------
constexpr int kGrpConsumers = 4;   // consumer warps of a CTA at most: one to a scheduler
constexpr int kGrpProducers = 8;   // producer warps (4: 16000 trajectories 263 ns a step, 12: 197)
constexpr int kGrpTwoProducers = 4;   // ... of a CTA with TWO
constexpr int kGrpSteps = 8;       // steps of a consumer's block (16: 5 % slower at 2 lanes a warp, 10 % faster at 1)
constexpr int kGrpItems = 8;       // items (four steps of a trajectory) of a producer lane in a buffer (4: 219 ns)
constexpr int kGrpBuffer = 256;    // steps of a buffer at most
constexpr int kGrpShared = 200 << 10;      // bytes of a CTA's buffers at most
constexpr int kGrpTwoShared = 100 << 10;   // ... with TWO (two CTAs an SM)
__device__ __forceinline__ void bar_sync(int id, int n) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int n) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// Waits of a flip into state 0 (low half) and 1 by the words of N steps:
// flip_wait for either state, the logarithms evaluated once and together.
template <int N>
__device__ __forceinline__ void dense_waits(const KConst& k, const Words (&wf)[N], uint32_t (&out)[N]) {
    double u[N], lu[N];
#pragma unroll
    for (int j = 0; j < N; ++j) u[j] = ((double)(((uint64_t)wf[j].w0 << 32) | wf[j].w1) + 1.0) * 0x1p-64;
    log_f64(u, lu);
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const uint32_t w0 = 1u + (uint32_t)floor(lu[j] / k.ln1m[0]);
        const uint32_t w1 = k.ln1m[1] == k.ln1m[0] ? w0 : 1u + (uint32_t)floor(lu[j] / k.ln1m[1]);
        out[j] = w0 | (w1 << 16);
    }
}

// The consumer's flip schedule source with DENSE: the producer's waits.
struct FlipFromBuffer {
    uint32_t w;
    __device__ __forceinline__ int64_t schedule(const KConst&, uint32_t, uint64_t s, int state, Words*, bool*) const {
        return (int64_t)s + (state ? (w >> 16) : (w & 0xffffu));
    }
};

// quiet_moves with flips taken from the producer's waits w[m]; l the first
// step's place in the buffer, flip that of the pending flip.  The state is
// kept as the byte selector of its half of a wait (kWait0 or kWait1), the
// steps in state 1 as the selectors' sum; FLAT as there.  One warp alone on
// its scheduler takes ~50 cycles a step: the sample input 6.66 / 6.55 ms with
// these.
constexpr uint32_t kWait0 = 0x4410, kWait1 = 0x4432;
template <bool OVER, bool FLAT, int N>
__device__ __forceinline__ bool dense_block(const KConst& k, Lane& a, bool want, int& flip, int l, const double* rf,
                                            const uint32_t* w) {
    double x = a.t.x, r = a.t.rprev, v = a.t.v, F = a.t.F;
    int nf = flip - l, far = 0;
    uint32_t sel = a.t.state ? kWait1 : kWait0, sum = 0;
#pragma unroll
    for (int m = 0; m < N; ++m) {
        if (OVER) {
            if (!FLAT) x = fma(F, k.c_drift, x);
            x = x + rf[m];
            x = x + r;
            r = rf[m];
        } else {
            v = v + (k.invM * F) * k.hdt;
            x = x + v * k.hdt;
            v = k.expg * v + rf[m];
            x = x + v * k.hdt;
        }
        far = max(far, off_band(a, x));
        if (nf == m) {
            sel ^= kWait0 ^ kWait1;
            nf = m + (int)__byte_perm(w[m], 0, sel);
        }
        if (!OVER || !FLAT) F = (sel & 2u) ? a.bF1 : a.bF0;
        sum += sel;
        if (!OVER) v = v + (k.invM * F) * k.hdt;
    }
    const int state = (int)(sel >> 1) & 1, n1 = (int)((sum - N * kWait0) / (kWait1 - kWait0));
    if (OVER && FLAT) F = state ? a.bF1 : a.bF0;
    if (!(want && far < a.half)) return false;
    a.t.x = x;
    a.t.rprev = r;
    a.t.v = v;
    a.t.F = F;
    a.t.state = state;
    flip = l + nf;
    a.sc1 += n1;
    return true;
}

// Where a lane's run of steps stands besides its Lane: the next frame and its
// place (null: no frames are kept), and the first step not integrated.
struct Course {
    int64_t frame;
    double* px;
    uint64_t s_done;
    int every;   // steps between frames, 2^30 at most
};

__device__ __forceinline__ Course course(const KConst& k, const TrajState& st, int64_t i, uint64_t s_begin,
                                         uint64_t s_end) {
    const uint64_t fs = k.freq_save;
    Course c;
    c.frame = (int64_t)((s_begin + fs - 1) / fs);
    c.px = st.fx ? st.fx + c.frame * st.n + i : nullptr;
    c.s_done = s_end;
    c.every = fs < (1u << 30) ? (int)fs : 1 << 30;
    return c;
}

// Steps s0 + l .. s0 + n - 1 of a warp's lanes, their noise in z[l ..] (DENSE:
// the waits of their flips in wt), in blocks of N.
template <bool DBL, bool OVER, bool ETA, bool DENSE, int N>
__device__ __forceinline__ void take_steps(const KConst& k, const TrajState& st, int64_t i, uint32_t g, Lane& a,
                                           Course& c, uint64_t s0, int l, const int n, const double* z,
                                           const uint32_t* wt) {
    auto near = [](int64_t d) { return d < (1 << 30) ? (int)d : 1 << 30; };
    // Steps s0 + l, l < n; each lane at its own l: a lane goes on from a
    // special step with a new block, and its warp waits for it at the
    // buffer's end only.
    if (!(a.q & Q_RUN)) l = n;
    // the places of the next frame (beyond every buffer where none is kept:
    // no frame is ever due, and save is not called) and of the pending flip,
    // and the last place a block can start at
    int fr = k.fp_mode || !c.px ? 1 << 30 : near(c.frame * (int64_t)k.freq_save - (int64_t)s0);
    int flip = near(a.nflip - (int64_t)s0);
    auto save = [&]() {
        if (c.frame < k.nframe) {   // the frame arrays hold nframe rows
            *c.px = a.t.x;
            if (k.write_x && st.fv) {   // the rest of WRITEX: fp64_series_kernel
                c.px[st.fv - st.fx] = a.t.v;
                c.px[st.fst - st.fx] = (double)a.t.state;
            }
        }
        c.px += st.n;
        ++c.frame;
        fr = min(fr + c.every, 1 << 30);
    };
    auto last_start = [&]() { return min(min(n, fr + 1), ETA && !DENSE ? flip : n) - N; };
    int lim = last_start();
    while (__any_sync(0xffffffffu, l < n)) {
        bool failed = false;
        if (!__any_sync(0xffffffffu, l < n && l > lim)) {
            // blocks, until a lane cannot go on with one
            const bool flat = OVER && !__any_sync(0xffffffffu, (a.q & Q_FORCE) != 0u);
            bool on, stop;
#pragma unroll 1
            do {
                on = l <= lim;
                const int lc = on ? l : 0;
                double rf[N];
#pragma unroll
                for (int m = 0; m < N; ++m) rf[m] = z[lc + m];
                bool stands;
                if (DENSE) {
                    uint32_t w[N];
#pragma unroll
                    for (int m = 0; m < N; ++m) w[m] = wt[lc + m];
                    stands = flat ? dense_block<OVER, true, N>(k, a, on, flip, lc, rf, w)
                                  : dense_block<OVER, false, N>(k, a, on, flip, lc, rf, w);
                } else if (flat) {
                    stands = quiet_moves<OVER, true, N>(k, a, on, rf);
                } else {
                    stands = quiet_moves<OVER, false, N>(k, a, on, rf);
                }
                l += stands ? N : 0;
                failed = on && !stands;
                stop = on && (failed || l > lim);
            } while (!__any_sync(0xffffffffu, stop));
        }
        if (l < n && (failed || l > lim)) {
            if (l != fr + 1) {
                // one by one, to the first special step and over it, or
                // to the next place where blocks can go on
                const int end = min(failed ? l + N : n, fr + 1);
                int n1 = 0;
                bool off;
                do {
                    fp64_move<OVER>(k, a.t, z[l]);
                    off = !(off_band(a, a.t.x) < a.half);
                    if (off || (ETA && !DENSE && l == flip)) break;
                    if (DENSE && l == flip) {
                        a.t.state ^= 1;
                        flip = l + (int)__byte_perm(wt[l], 0, a.t.state ? 0x4432 : 0x4410);
                        a.t.F = a.t.state ? a.bF1 : a.bF0;
                    }
                    n1 += a.t.state;
                    if (!OVER) a.t.v = a.t.v + (k.invM * a.t.F) * k.hdt;
                } while (++l < end);
                a.sc1 += n1;
                if (l < end) {
                    if (DENSE) {
                        a.nflip = (int64_t)s0 + flip;
                        const FlipFromBuffer src{wt[l]};
                        special_step<DBL, OVER, ETA>(k, st, i, g, a, s0 + l, off, src);
                    } else {
                        const FlipDraw src;
                        special_step<DBL, OVER, ETA>(k, st, i, g, a, s0 + l, off, src);
                    }
                    flip = near(a.nflip - (int64_t)s0);
                    ++l;
                }
            }
            if (!(a.q & Q_RUN)) {
                c.s_done = s0 + l - ((a.flags & LDP_FLAG_NONFINITE) ? 1 : 0);
                l = n;
            } else if (l == fr + 1) {
                save();
            }
            lim = last_start();
        }
        __syncwarp();
    }
    if (l == fr + 1 && (a.q & Q_RUN)) save();   // at the buffer's end
    if (DENSE && (a.q & Q_RUN)) a.nflip = (int64_t)s0 + flip;
}

// Steps s_begin .. s_end-1, one trajectory per thread, each drawing its own
// noise, kOwnSteps steps at a time (two Philox blocks and four Box-Muller
// pairs at once) into its row of shared memory, and then taking these steps
// as in group mode, each lane at its own.  Bound by the issue of ~125
// instructions a step, 100 of them the noise, at four warps a scheduler (122
// registers).  65536 trajectories, kernel ms: 29.3 with two pairs at once one
// after the other and four steps between votes, 25.5 with the pairs together,
// 23.9 with rows of noise (blocks of four steps, or a try of four before the
// steps one by one: 24.1).  DENSE: see group mode above.
constexpr int kOwnSteps = 32, kOwnDense = 16;
template <bool DBL, bool OVER, bool ETA, bool DENSE>
__global__ void __launch_bounds__(128, 4) fp64_steps_kernel(const KConst k, const TrajState st, int64_t g0,
                                                         uint64_t s_begin, uint64_t s_end) {
    constexpr int S = DENSE ? kOwnDense : kOwnSteps;
    // Blocks of four where flips are frequent and steps overdamped, the edge
    // between two cells being crossed often (65536 x 24400, p = 0.5, blocks of
    // eight / four: one barrier 28.4 / 26.6 ms, two 42.4 / 39.6; underdamped
    // first passage 10.0 / 10.1).
    constexpr int kSteps = DENSE && OVER ? 4 : kGrpSteps;
    __shared__ double rows[128 * (S + 1)];   // of an odd length: see fp64_group_kernel
    __shared__ uint32_t wrows[DENSE ? 128 * (S + 1) : 1];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t g = (uint32_t)(g0 + i);
    Lane a;
    load_lane<DBL, OVER>(k, st, i, i < st.n, a);
    const bool active = (a.q & Q_RUN) != 0u;
    Course c = course(k, st, i, s_begin, s_end);
    const double sig = OVER ? k.sig_r : k.sig_v;
    double* z = rows + threadIdx.x * (S + 1);
    uint32_t* wt = wrows + (DENSE ? threadIdx.x * (S + 1) : 0);
    uint64_t s0 = ((s_begin - 1) & ~3ull) + 1;   // the first step of a Philox block
    int l = (int)(s_begin - s0);
    while (s0 < s_end && __any_sync(0xffffffffu, (a.q & Q_RUN) != 0u)) {
        const int n = s_end - s0 < (uint64_t)S ? (int)(s_end - s0) : S;
#pragma unroll 1
        for (int m = 0; m < n; m += 8) {
            const uint64_t q = (s0 + (uint64_t)m - 1) >> 2;
            const Words w = philox_at(q, g, TAG_STEP, k.key0, k.key1);
            const Words w2 = philox_at(q + 1, g, TAG_STEP, k.key0, k.key1);
            const uint32_t wa[4] = {w.w0, w.w2, w2.w0, w2.w2}, wb[4] = {w.w1, w.w3, w2.w1, w2.w3};
            double r[8];
            gauss_pairs_f64(wa, wb, r);
#pragma unroll
            for (int j = 0; j < 8; ++j) z[m + j] = sig * r[j];
        }
        if (DENSE) {
#pragma unroll 1
            for (int m = 0; m < n; m += 2) {
                const uint64_t q = s0 + (uint64_t)m;
                const Words wf[2] = {philox_at(q, g, TAG_FLIP, k.key0, k.key1),
                                     philox_at(q + 1, g, TAG_FLIP, k.key0, k.key1)};
                uint32_t w[2];
                dense_waits(k, wf, w);
                wt[m] = w[0];
                wt[m + 1] = w[1];
            }
        }
        take_steps<DBL, OVER, ETA, DENSE, kSteps>(k, st, i, g, a, c, s0, l, n, z, wt);
        l = 0;
        s0 += S;
    }
    if (active) store_lane(k, st, i, a, c.s_done, s_begin, s_end);
}

template <bool DBL, bool OVER, bool ETA, bool DENSE, bool TWO>
__global__ void __launch_bounds__(32 * (kGrpConsumers + (TWO ? kGrpTwoProducers : kGrpProducers)), TWO ? 2 : 1)
    fp64_group_kernel(const KConst k, const TrajState st, int64_t g0, uint64_t s_begin, uint64_t s_end, int nc, int T,
                      int B) {
    // noise [2][M][R], then with DENSE waits [2][M][R]; rows of an odd length,
    // so that lanes at the same step are in different banks
    extern __shared__ double buf[];
    const int M = nc * T, R = B + 1, P = (blockDim.x >> 5) - nc;
    uint32_t* waits = (uint32_t*)(buf + 2 * R * M);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // its consumer warp (producer warp p draws for the warp p mod nc), that
    // warp's trajectories, and the threads that share its barriers
    const int cw = warp < nc ? warp : (warp - nc) % nc, t0 = cw * T;
    const int64_t i0 = (int64_t)blockIdx.x * M + t0;
    const int nthreads = 32 * (1 + (P - cw + nc - 1) / nc);
    const int full = 4 * cw, empty = 4 * cw + 2;
    const uint64_t a0 = (s_begin - 1) >> 2;           // the first buffer starts on a Philox block
    const uint64_t sb = 4 * a0 + 1;
    const uint64_t nblk = s_end > s_begin ? (s_end - sb + B - 1) / B : 0;
    if (warp >= nc) {
        // ---- producers ----
        const int p = (warp - nc) / nc * 32 + lane, np = nthreads - 32;
        const double sig = OVER ? k.sig_r : k.sig_v;
        for (uint64_t b = 0; b < nblk; ++b) {
            const int u = (int)(b & 1);
            if (b >= 2) bar_sync(empty + u, nthreads);   // buffer u released by the consumer
            double* z = buf + (u * M + t0) * R;
            for (int e = p; e < (B >> 2) * T; e += np) {
                const int quad = e / T, tr = e - quad * T;
                const uint64_t q = a0 + b * (uint64_t)(B >> 2) + (uint64_t)quad;
                if (i0 + tr >= st.n || 4 * q + 1 >= s_end) continue;
                const Words w = philox_at(q, (uint32_t)(g0 + i0 + tr), TAG_STEP, k.key0, k.key1);
                double n[4];
                gauss_block_f64(w, n);
                double* o = z + tr * R + quad * 4;
#pragma unroll
                for (int m = 0; m < 4; ++m) o[m] = sig * n[m];
            }
            if (DENSE) {
                uint32_t* wt = waits + (u * M + t0) * R;
                for (int e = p; e < B * T; e += np) {
                    const int step = e / T, tr = e - step * T;
                    const uint64_t s = sb + b * (uint64_t)B + (uint64_t)step;
                    if (i0 + tr >= st.n || s >= s_end) continue;
                    const Words wf[1] = {philox_at(s, (uint32_t)(g0 + i0 + tr), TAG_FLIP, k.key0, k.key1)};
                    uint32_t w[1];
                    dense_waits(k, wf, w);
                    wt[tr * R + step] = w[0];
                }
            }
            __syncwarp();
            bar_arrive(full + u, nthreads);          // buffer u full
        }
        // the consumer's release of the last two buffers
        for (uint64_t b = (nblk > 2 ? nblk - 2 : 0); b < nblk; ++b) bar_sync(empty + (int)(b & 1), nthreads);
        return;
    }
    // ---- consumers ----
    const int64_t i = i0 + lane;
    const uint32_t g = (uint32_t)(g0 + i);
    Lane a;
    load_lane<DBL, OVER>(k, st, i, lane < T && i < st.n, a);
    const bool active = (a.q & Q_RUN) != 0u;
    Course c = course(k, st, i, s_begin, s_end);
    const int tl = t0 + (lane < T ? lane : 0);   // idle lanes read a lane's noise
    __syncwarp();   // load_lane parts the lanes; the barriers want the warp together
    for (uint64_t b = 0; b < nblk; ++b) {
        const int u = (int)(b & 1);
        bar_sync(full + u, nthreads);                // buffer u full
        const double* z = buf + (u * M + tl) * R;
        const uint32_t* wt = waits + (u * M + tl) * R;
        const uint64_t s0 = sb + b * (uint64_t)B;
        const int n = s_end - s0 < (uint64_t)B ? (int)(s_end - s0) : B;
        take_steps<DBL, OVER, ETA, DENSE, kGrpSteps>(k, st, i, g, a, c, s0, b == 0 ? (int)(s_begin - sb) : 0, n, z, wt);
        __syncwarp();
        bar_arrive(empty + u, nthreads);             // buffer u released
    }
    if (active) store_lane(k, st, i, a, c.s_done, s_begin, s_end);
}

// WRITEX's other series of frames f0 .. f1 - 1 from their position, velocity
// and barrier state: force, energy and barrier height are those of the
// position, whatever kind of step led there.  The steps save three of the
// seven series only, which keeps the rest out of the stepping warps' chains
// (the sample input, a frame in 80 steps, 6.83 / 6.66 ms; a frame a step 0.544
// / 0.523); this pass over the frames is memory-bound.
template <bool DBL>
__global__ void __launch_bounds__(256) fp64_series_kernel(const KConst k, const TrajState st, int64_t f0, int64_t f1) {
    const int64_t n = st.n, end = f1 * n, stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t o = f0 * n + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < end; o += stride) {
        const int64_t f = o / n;
        // (not past the end of a trajectory that ended early)
        if (f * (int64_t)k.freq_save > st.counts[(int64_t)LDP_C_STEPS * n + (o - f * n)]) continue;
        T64 t{};
        t.x = st.fx[o];
        t.v = st.fv[o];
        t.state = (int)st.fst[o];
        indices<DBL>(k, t);
        energy_force<DBL>(k, t);
        st.ff[o] = t.F;
        st.fb[o] = t.barrier;
        st.fpe[o] = t.E;
        st.fke[o] = k.mhalf * (t.v * t.v);
    }
}

int launch_fp64_series(const KConst& k, const TrajState& st, uint64_t s_begin, uint64_t s_end, int sms, void* stream) {
    const int64_t fs = (int64_t)k.freq_save;
    const int64_t f0 = ((int64_t)s_begin + fs - 1) / fs;
    const int64_t f1 = std::min<int64_t>(k.nframe, ((int64_t)s_end - 1) / fs + 1);
    if (!k.write_x || !st.fx || !st.fv || f1 <= f0 || st.n <= 0) return 0;
    const int64_t blocks = std::min<int64_t>(((f1 - f0) * st.n + 255) / 256, (int64_t)8 * sms);
    if (k.dbl) fp64_series_kernel<true><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(k, st, f0, f1);
    else fp64_series_kernel<false><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(k, st, f0, f1);
    return (int)cudaGetLastError();
}

// The larger and the smaller flip probability of a step.
static void flip_rates(const KConst& k, double* p, double* pmin) {
    *p = 0.0;
    *pmin = 1.0;
    for (int b = 0; b < 2; ++b) {
        const double f = k.eta ? -std::expm1(k.ln1m[b]) : 0.0;
        *p = std::max(*p, f);
        *pmin = std::min(*pmin, f);
    }
}

template <bool DBL, bool OVER>
static int launch_init_t(const KConst& k, const TrajState& st, int64_t g0, int block, cudaStream_t stream) {
    const int64_t grid = (st.n + block - 1) / block;
    fp64_init_kernel<DBL, OVER><<<(unsigned)grid, block, 0, stream>>>(k, st, g0);
    return (int)cudaGetLastError();
}

int launch_fp64_init(const KConst& k, const TrajState& st, int64_t g0, int block, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    block = 128;
    if (k.dbl) return k.over ? launch_init_t<true, true>(k, st, g0, block, s) : launch_init_t<true, false>(k, st, g0, block, s);
    return k.over ? launch_init_t<false, true>(k, st, g0, block, s) : launch_init_t<false, false>(k, st, g0, block, s);
}

template <bool DBL, bool OVER, bool ETA>
static int launch_steps_t(const KConst& k, const TrajState& st, int64_t g0, uint64_t s0, uint64_t s1, int block,
                          cudaStream_t stream) {
    const int64_t grid = (st.n + block - 1) / block;
    double p, pmin;
    flip_rates(k, &p, &pmin);
    // DENSE: drawing the waits of every step costs about as much as the noise,
    // a flip drawn as it comes a special step of its lane.  65536 trajectories
    // x 12000 steps, ms as they come / DENSE: p = 0.5 18.3 / 14.8, 0.1 16.3 /
    // 14.4, 0.01 9.3 / 13.7; two barriers 20.7 / 20.7, 19.4 / 19.5, 12.7 / 17.3;
    // underdamped 16.5 / 10.9, 14.5 / 10.8, 7.4 / 10.7.
    if (ETA && pmin > 0.05)
        fp64_steps_kernel<DBL, OVER, ETA, ETA><<<(unsigned)grid, block, 0, stream>>>(k, st, g0, s0, s1);
    else
        fp64_steps_kernel<DBL, OVER, ETA, false><<<(unsigned)grid, block, 0, stream>>>(k, st, g0, s0, s1);
    return (int)cudaGetLastError();
}

template <bool DBL, bool OVER, bool ETA>
static int launch_group_t(const KConst& k, const TrajState& st, int64_t g0, uint64_t s0, uint64_t s1, int nc, int T,
                          int P, int B, bool dense, bool two, cudaStream_t stream) {
    const int M = nc * T;
    const int64_t grid = (st.n + M - 1) / M;
    const size_t smem = (size_t)2 * (B + 1) * M * (dense ? 12 : 8);
    auto* kern = fp64_group_kernel<DBL, OVER, ETA, false, false>;
    if (ETA && dense) kern = fp64_group_kernel<DBL, OVER, ETA, ETA, false>;
    if (OVER && two) {
        kern = fp64_group_kernel<DBL, OVER, ETA, false, OVER>;
        if (ETA && dense) kern = fp64_group_kernel<DBL, OVER, ETA, ETA, OVER>;
    }
    // The limit is the kernel's, for all threads and contexts of the process,
    // so it is set to the most that a launch of it takes: with a launch's own
    // size here, another thread's smaller launch could lower it before this one.
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               OVER && two ? kGrpTwoShared : kGrpShared);
    if (e != cudaSuccess) return (int)e;
    kern<<<(unsigned)grid, 32 * (nc + P), smem, stream>>>(k, st, g0, s0, s1, nc, T, B);
    return (int)cudaGetLastError();
}

int launch_fp64_group(const KConst& k, const TrajState& st, int64_t g0, uint64_t s_begin, uint64_t s_end, int sms,
                      int min_lanes, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (st.n <= 0) return 0;
    double p, pmin;
    flip_rates(k, &p, &pmin);
    // One consumer warp to each of the GPU's schedulers, or two, with as many
    // lanes as that takes.
    int T = (int)std::min<int64_t>(32, (st.n + 4 * sms - 1) / (4 * sms));
    const bool two = k.over && T > min_lanes && (min_lanes == 1 || p < 1.0 / 1024);
    if (two) T = (int)std::min<int64_t>(32, (st.n + 8 * sms - 1) / (8 * sms));
    T = std::max(T, min_lanes);
    const int nc = (int)std::min<int64_t>(kGrpConsumers, (st.n + (int64_t)sms * T - 1) / ((int64_t)sms * T));
    const int M = nc * T;
    const bool dense = k.eta && pmin >= 1.0 / 1024 && p * T > 1.0 / 40;
    const int P = two ? kGrpTwoProducers : kGrpProducers;
    int B = 8 * ((32 * P * kGrpItems * 4 / M + 7) / 8);
    const int room = (two ? kGrpTwoShared : kGrpShared) / (2 * M * (dense ? 12 : 8)) - 1;   // shared memory
    B = std::min(std::min(std::max(B, 16), kGrpBuffer), room / 8 * 8);
    const int sel = (k.dbl ? 4 : 0) | (k.over ? 2 : 0) | (k.eta ? 1 : 0);
    switch (sel) {
        case 0: return launch_group_t<false, false, false>(k, st, g0, s_begin, s_end, nc, T, P, B, dense, two, s);
        case 1: return launch_group_t<false, false, true>(k, st, g0, s_begin, s_end, nc, T, P, B, dense, two, s);
        case 2: return launch_group_t<false, true, false>(k, st, g0, s_begin, s_end, nc, T, P, B, dense, two, s);
        case 3: return launch_group_t<false, true, true>(k, st, g0, s_begin, s_end, nc, T, P, B, dense, two, s);
        case 4: return launch_group_t<true, false, false>(k, st, g0, s_begin, s_end, nc, T, P, B, dense, two, s);
        case 5: return launch_group_t<true, false, true>(k, st, g0, s_begin, s_end, nc, T, P, B, dense, two, s);
        case 6: return launch_group_t<true, true, false>(k, st, g0, s_begin, s_end, nc, T, P, B, dense, two, s);
        default: return launch_group_t<true, true, true>(k, st, g0, s_begin, s_end, nc, T, P, B, dense, two, s);
    }
}

int launch_fp64_steps(const KConst& k, const TrajState& st, int64_t g0, uint64_t s_begin, uint64_t s_end, int block,
                      void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    block = 128;
    const int sel = (k.dbl ? 4 : 0) | (k.over ? 2 : 0) | (k.eta ? 1 : 0);
    switch (sel) {
        case 0: return launch_steps_t<false, false, false>(k, st, g0, s_begin, s_end, block, s);
        case 1: return launch_steps_t<false, false, true>(k, st, g0, s_begin, s_end, block, s);
        case 2: return launch_steps_t<false, true, false>(k, st, g0, s_begin, s_end, block, s);
        case 3: return launch_steps_t<false, true, true>(k, st, g0, s_begin, s_end, block, s);
        case 4: return launch_steps_t<true, false, false>(k, st, g0, s_begin, s_end, block, s);
        case 5: return launch_steps_t<true, false, true>(k, st, g0, s_begin, s_end, block, s);
        case 6: return launch_steps_t<true, true, false>(k, st, g0, s_begin, s_end, block, s);
        default: return launch_steps_t<true, true, true>(k, st, g0, s_begin, s_end, block, s);
    }
}

}  // namespace ldp
