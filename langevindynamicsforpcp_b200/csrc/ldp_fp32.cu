// ldp_fp32.cu -- FP32 batched persistent trajectory kernel.
//
// Same model as the FP64 plain path (src/langevinDynamicsSingleBarrier.h:
// 1292-1324, 1680-1706, 1861-1884, 1998-2165, 2334-2592, 2860-2886 and the
// double-barrier counterparts in src/langevinDynamicsDoubleBarrier.h), with
// the step in FP32:
//  * position = cell * L + xp with an int cell index and an FP32 cell-local
//    coordinate xp in [-L/2, L/2) (no FP32 absolute position);
//  * Box-Muller noise on the special-function units (lg2/sqrt/sin/cos
//    approximations) from the same Philox words the FP64 path uses, the
//    uniforms built from the words' high bits by exponent splicing;
//  * an exact integer step counter as the clock; event durations are summed
//    as integer step counts (exact), frames are saved as FP64 cell*L + xp.
//
// Hot loop.  The force of both models is piecewise constant in xp: between
// consecutive "breakpoints" (cell edges, barrier flanks, the barrier top and,
// for the double model, the flank meeting point) neither the force, the
// cell, the well nor the local barrier changes.  Each thread keeps the open
// band (lo, hi) around its position, the force of its current barrier state
// and a countdown to its next frame, flip or last step in registers.  A block
// of four steps is one Philox block, two Box-Muller pairs, the four moves and
// one test for the warp: whether every lane stayed in its band and no
// countdown ended.  If not (about one block in five), the lanes concerned take
// the block again step by step.  Their special steps are quick steps, inline
// (a frame, a flank entered or left, the edge between the two cells of a pair
// crossed, a flip where flips are frequent, and in the kernels of jobs with many
// special steps (M_FULL) nearly all kinds), or take the slow path out of line
// (special_step): at last the general step, which follows the FP64 step
// exactly (wrap, indices, flip, cell-table entry with lazy catch-up, force,
// renewal statistics, frame, end).
//
// What bounds it: instruction issue.  4 jobs x 65536 trajectories x 120000
// steps, frames every 100: 76.8 ms with a test and a branch at each step and
// ten dependent loads in each special step, 59.5 ms with this loop.
// The loop is a function without calls (run_blocks, no spills at 48 registers
// and more), the lane state in shared memory between it and the out-of-line
// parts: with the calls inside it the loop kept three of its values on the
// stack (63.7 ms, 59.6 ms without), or spilled at each block (71.4 ms).

// Rare state lives in shared memory (statistics clocks and flags, the cached
// state of the cell left last, the state-1 step count), counts and duration
// sums go out as fire-and-forget atomics, and the cell-table ring is written
// through on every cell exit, so re-crossing back into the cell just left
// needs no memory read.
//
// Batching: each thread is a slot that owns one trajectory; when it retires
// (fixed step count reached, or first passage in FIRST_PASSAGE mode) the
// warp's idle lanes claim new trajectories from the device work queue with
// one fetch-and-add per warp and a ballot/popc prefix.
#include <cuda_runtime.h>

#include <algorithm>

#include "ldp_device.cuh"
#include "ldp_fp32.h"
#include "ldp_share.h"

namespace ldp {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kMaxBlock = 256;
constexpr int kLeftMax = 1 << 30;      // countdown clamp; a clamped zero is a no-op general step

// Statistics flags used only by this path (bits 0..23 are the shared B_*).
enum : uint32_t { B_HAS_FPT = 1u << 24, B_HAS_FPT2 = 1u << 25, B_HAS_TPT = 1u << 26, B_HAS_TPT2 = 1u << 27 };
// Slot word: local barrier, eviction pending for the current cell, cache of
// the cell left last (valid, its state).
enum : int32_t { W_LB = 1, W_EVICT = 2, W_CVALID = 4, W_CSTATE = 8 };

// Model type K: 0-3 (double * 2 + overdamped), or 4, the job's, for code
// that serves all four; plus K_WIDE in the wide kernels (their own copies of
// the out-of-line parts, compiled for fewer registers) and K_FULL in the
// kernels for jobs of every mode (the others serve M_RARE and M_FLIPS).
constexpr int K_ANY = 4, K_WIDE = 8, K_FULL = 16;
template <int K>
__device__ __forceinline__ bool is_double(const JobF& J) { return (K & K_ANY) ? J.dbl != 0 : (K & 2) != 0; }
template <int K>
__device__ __forceinline__ bool is_over(const JobF& J) { return (K & K_ANY) ? J.over != 0 : (K & 1) != 0; }

// The word of a lane's quick steps (see quick_step), kept in a register by
// the hot loop: quick steps allowed (the barrier flanks do not reach the cell
// edges); the lane's cell and a neighbour form a pair whose shared edge it may
// cross quickly; it is in the pair's other cell now; the other cell is the
// right neighbour; the two barriers' states; the countdown ends at a frame
// and nothing else; the pair's edge was crossed at least once; the other
// cell's pending flip has come.  Then the step of a block that needs the slow
// path, one more than its place (three bits), and the job's mode (M_*).
enum : uint32_t {
    P_FAST = 1, P_PAIR = 2, P_SWAP = 4, P_RIGHT = 8, P_S0 = 16, P_S1 = 32, P_FRAME = 64, P_CROSSED = 128,
    P_OVERDUE = 256, P_HALT = 512, P_HALTS = 7 * P_HALT, P_MODE = 1u << 16
};

// Per-thread rare state, structure of arrays (conflict-free by thread).
struct RareSm {
    uint32_t bits[kMaxBlock];
    int32_t init0[kMaxBlock];     // first cell of the FPT initial-barrier pair
    int32_t idx2[kMaxBlock];      // first cell of the FPT2 reference pair
    int32_t tpt2w[kMaxBlock];     // well of the last TPT2 renewal
    int32_t ckey[kMaxBlock];      // key of the cell left last
    int32_t cgw[kMaxBlock];       // well of the last FPTCG evaluation
    int32_t fidx[kMaxBlock];      // index of the next frame
    long long nxf[kMaxBlock];     // step of the next frame
    long long fpt[kMaxBlock], fpt2[kMaxBlock], tpt[kMaxBlock], tpt2[kMaxBlock];
    long long cflip[kMaxBlock];   // pending flip step of the cached cell
    long long sc1[kMaxBlock];     // completed state-1 steps
    long long since[kMaxBlock];   // first step of the current state-1 run
    // Lane state the hot loop hands to the general step and takes back, and
    // the lane state only the general step uses.
    float xp[kMaxBlock], rv[kMaxBlock], F[kMaxBlock], lo[kMaxBlock], hi[kMaxBlock];
    uint4 fix[kMaxBlock];         // Philox constants of the lane's step blocks (philox_fix) ...
    uint2 fixk[kMaxBlock];        // ... the first key word of its third round, and the noise scale (float bits)
    uint32_t traj[kMaxBlock];
    float nz[3][kMaxBlock];       // noise of a block's steps after one that needs the slow path
    long long nflip[kMaxBlock];   // step of the current barrier's next flip
    int32_t left[kMaxBlock], job[kMaxBlock], cell[kMaxBlock], state[kMaxBlock], sw[kMaxBlock];
    uint32_t pw[kMaxBlock];       // P_* word (quick steps)
    long long nev[kMaxBlock];     // first step that is special for another reason than a frame
    long long xs[kMaxBlock];      // step of the last quick crossing
    uint32_t j[kMaxBlock], jh[kMaxBlock];   // next block of four steps, 4j+1 .. 4j+4: j's low and high word
    const SlotsDev* slots;        // the launch's slots
};
static_assert(sizeof(RareSm) <= 55 * 1024, "four blocks to an SM");

__device__ __forceinline__ void red_add(int64_t* p, int64_t v) {
    atomicAdd(reinterpret_cast<unsigned long long*>(p), (unsigned long long)v);
}

__device__ __forceinline__ int fkey(bool dbl, int cell, int lb) { return dbl ? cell * 2 + lb : cell; }

// Step of the next flip of a barrier now in state st, scheduled at step s
// (words w0:w1 of TAG_FLIP at a = s; geometric waiting time, FP64 as in the
// FP64 path, so both precisions schedule the same flips from the same
// history).
__device__ __forceinline__ long long next_flip(const JobF& J, uint32_t traj, uint64_t s, int st) {
    const Words w = philox_at(s, traj, TAG_FLIP, J.key0, J.key1);
    return flip_schedule(s, w.w0, w.w1, J.ln1m[st]);
}

// The Philox blocks of a lane's steps (counter: block index j, stream g,
// TAG_STEP = 0) differ only in j, and its high word changes every 2^34 steps.
// The products of g, hence the first round's second half and the second
// round's first multiply, are the same for all of them: philox_fix holds what
// follows from them, philox_step takes it from there (17 wide multiplies and
// 19 xors instead of 20 and 20, 15 key additions instead of 18); the words
// are philox's.
__device__ __forceinline__ uint4 philox_fix(uint32_t g, uint32_t jh, uint32_t k0, uint32_t k1) {
    const uint64_t p1 = (uint64_t)g * 0xCD9E8D57u;
    const uint32_t c0 = (uint32_t)(p1 >> 32) ^ jh ^ k0;   // after round 1 (its c1 is (uint32_t)p1)
    const uint64_t p0 = (uint64_t)c0 * 0xD2511F53u;       // of round 2
    return make_uint4(k1, (uint32_t)p1 ^ (k0 + 0x9E3779B9u), (uint32_t)(p0 >> 32) ^ (k1 + 0xBB67AE85u), (uint32_t)p0);
}
__device__ __forceinline__ Words philox_step(uint32_t jl, uint4 fix, uint32_t k0) {
    const uint64_t q0 = (uint64_t)jl * 0xD2511F53u;       // round 1
    const uint64_t q1 = (uint64_t)((uint32_t)(q0 >> 32) ^ fix.x) * 0xCD9E8D57u;   // round 2
    uint32_t c0 = (uint32_t)(q1 >> 32) ^ fix.y, c1 = (uint32_t)q1, c2 = (uint32_t)q0 ^ fix.z, c3 = fix.w;
    uint32_t k1 = fix.x + 2u * 0xBB67AE85u;
#pragma unroll
    for (int r = 2; r < 10; ++r) {
        if (r > 2) { k0 += 0x9E3779B9u; k1 += 0xBB67AE85u; }
        const uint64_t p0 = (uint64_t)c0 * 0xD2511F53u;
        const uint64_t p1 = (uint64_t)c2 * 0xCD9E8D57u;
        c0 = (uint32_t)(p1 >> 32) ^ c1 ^ k0;
        c2 = (uint32_t)(p0 >> 32) ^ c3 ^ k1;
        c1 = (uint32_t)p1;
        c3 = (uint32_t)p0;
    }
    return Words{c0, c1, c2, c3};
}

// Uniform in (0, 1): the high 23 bits of w as a mantissa, offset by 2^-24.
__device__ __forceinline__ float unit_open(uint32_t w) {
    return __int_as_float((int)__funnelshift_r(w, 0x7fu, 9)) - 0.99999994039535522461f;
}
// w * 2^-32 folded into [-1/2, 1/2) (same angle mod 1), 23 high bits.
__device__ __forceinline__ float unit_centered(uint32_t w) {
    return __int_as_float((int)(__funnelshift_r(w, 0x7fu, 9) ^ 0x00400000u)) - 1.5f;
}

// Box-Muller pair scaled by sigma: k = -2 ln 2 sigma^2 (log2 is the native
// logarithm of the special-function unit).  Flush-to-zero forms: the
// uniforms are normal numbers in (2^-24, 1) and the angle in [-pi, pi).
__device__ __forceinline__ void noise_pair(uint32_t wa, uint32_t wb, float k, float* n0, float* n1) {
    float lg, r, sn, cs;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(lg) : "f"(unit_open(wa)));
    const float t = fmaxf(lg * k, 0.0f);
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(t));
    const float a = 6.28318530717958647692f * unit_centered(wb);
    asm("sin.approx.ftz.f32 %0, %1;" : "=f"(sn) : "f"(a));
    asm("cos.approx.ftz.f32 %0, %1;" : "=f"(cs) : "f"(a));
    *n0 = r * cs;
    *n1 = r * sn;
}

__device__ int f_default_state(const JobF& J, bool dbl, uint32_t g, int64_t ck) {
    if (J.us) {
        if (dbl) return J.init_state;
        const int64_t trial = ((int64_t)g / J.lanes) % J.nruns;
        if (trial == 0) return 0;
        if (!J.rs) return J.init_state;
        const Words w = philox_at(0, g - (uint32_t)J.lanes, TAG_INIT, J.key0, J.key1);
        return ((double)w.w0 * 0x1p-32 <= J.p_first) ? 0 : 1;
    }
    const Words w = philox_at((uint64_t)ck, g, TAG_CELL, J.key0, J.key1);
    return ((double)w.w0 * 0x1p-32 < J.p_cell0) ? 0 : 1;
}

__device__ __forceinline__ int f_ring_state(const JobF& J, const SlotsDev& S, int64_t slot, bool dbl, uint32_t g,
                                            int key) {
    const longlong2 e = S.ring[(int64_t)(key & (S.ring_slots - 1)) * S.nslots + slot];
    return (e.x == (long long)key) ? (int)(e.y & 1) : f_default_state(J, dbl, g, key);
}

// FP32 force of state st at xp (EnergyAndForce, S.h:1292-1324 /
// D.h:1464-1522).
__device__ __forceinline__ float force_of(const bool DBL, const JobF& J, float xp, int st) {
    if (!DBL) {
        const float a = fabsf(xp);
        return (a < J.w && a > 0.0f) ? copysignf(J.slope[st], xp) : 0.0f;
    } else {
        float f = 0.0f;
        if (xp < J.xb[0] && xp > J.lo0) f = J.sN[0][st];
        if (xp < J.xc && xp > J.xb[0]) f = J.sP[0][st];
        if (xp < J.xb[1] && xp > J.xc) f = J.sN[1][st];
        if (xp < J.hi1 && xp > J.xb[1]) f = J.sP[1][st];
        return -f;
    }
}

// force_of where no flank is: its zero's sign is the model's (a saved frame of
// WRITEX shows it).
__device__ __forceinline__ float flat_force(const bool DBL) { return DBL ? -0.0f : 0.0f; }

// Open band (lo, hi) of consecutive breakpoints around xp; lo = hi = xp when
// xp sits on a breakpoint, so that the next step takes the general path.
// Single barrier: the breakpoints are -L/2, -w, 0, w (clamped to the cell).
__device__ __forceinline__ void band_of(const bool DBL, const JobF& J, float xp, float* lo, float* hi) {
    if (!DBL) {
        const float w = J.w, hL = J.halfL, a = fabsf(xp);
        float l, h;
        if (a < w) { l = (xp > 0.0f) ? 0.0f : -w; h = (xp > 0.0f) ? w : 0.0f; }
        else { l = (xp > 0.0f) ? w : -hL; h = (xp > 0.0f) ? hL : -w; }
        l = fmaxf(l, -hL);
        h = fminf(h, hL);
        if (a == w || xp == 0.0f || xp == -hL) l = h = xp;
        *lo = l;
        *hi = h;
        return;
    }
    float l = -__int_as_float(0x7f800000), h = __int_as_float(0x7f800000);
    for (int i = 0; i < J.nbp; ++i) {
        const float b = J.bp[i];
        if (b < xp) { l = b; continue; }
        if (b == xp) l = h = xp; else h = b;
        break;
    }
    *lo = l;
    *hi = h;
}

__device__ __forceinline__ void f_energy(const bool DBL, const JobF& J, double xp, int s, double* E, double* B) {
    if (!DBL) {
        const double sp = J.Hs[s] / J.wd, sn = -sp;
        double e = 0.0;
        if (xp < 0.0 && xp > -J.wd) e = J.Hs[s] - xp * sn;
        if (xp < J.wd && xp > 0.0) e = J.Hs[s] - xp * sp;
        *E = e;
        *B = J.Hs[s];
    } else {
        double e = 0.0, b = 0.0;
        if (xp < J.xbd[0] && xp > J.lo0d) { e = xp * J.sNd[0][s] + J.iN[0][s]; b = J.Hd[0][s]; }
        if (xp < J.xcd && xp > J.xbd[0]) { e = xp * J.sPd[0][s] + J.iP[0][s]; b = J.Hd[0][s]; }
        if (xp < J.xbd[1] && xp > J.xcd) { e = xp * J.sNd[1][s] + J.iN[1][s]; b = J.Hd[1][s]; }
        if (xp < J.hi1d && xp > J.xbd[1]) { e = xp * J.sPd[1][s] + J.iP[1][s]; b = J.Hd[1][s]; }
        *E = e;
        *B = b;
    }
}

// WRITEX frame fields (velocity, force, barrier, energies, state).
__device__ __forceinline__ void record_extra(const bool DBL, const JobF& J, int64_t o, float xp, float v, float F,
                                             int state) {
    double E, B;
    f_energy(DBL, J, (double)xp, state, &E, &B);
    if (J.fv) J.fv[o] = (double)v;
    if (J.ff) J.ff[o] = (double)F;
    if (J.fb) J.fb[o] = B;
    if (J.fpe) J.fpe[o] = E;
    if (J.fke) J.fke[o] = J.mhalf * ((double)v * (double)v);
    if (J.fst) J.fst[o] = (double)state;
}
__device__ __noinline__ void f_record_extra(bool DBL, const JobF* Jp, int64_t o, float xp, float v, float F,
                                            int state) {
    record_extra(DBL, *Jp, o, xp, v, F, state);
}

__device__ __forceinline__ void f_record(const bool DBL, const JobF& J, uint32_t traj, int64_t frame, int cell,
                                         float xp, float v, float F, int state) {
    if (frame >= J.nframe) return;   // the frame arrays hold nframe rows
    const int64_t o = frame * J.ntraj + traj;
    if (J.fx) J.fx[o] = (double)cell * J.Ld + (double)xp;
    if (J.write_x) f_record_extra(DBL, &J, o, xp, v, F, state);
}

__device__ __forceinline__ bool cg_hit32(int well, int size) { return (well % size) == 0; }

// Step 0 of a trajectory (IntegrateStep0 + InitializeBarrierState +
// InitializeStatistics), FP64 where it is cheap and exact, then the hot
// state is rounded to FP32.  Writes the thread's rare state.
template <int K>
__device__ __noinline__ void f_start(const JobF* Jp, longlong2* ring, int64_t nslots, int ring_slots, int64_t slot,
                                     uint32_t traj, RareSm* sm, int t) {
    const JobF& J = *Jp;
    const bool DBL = is_double<K>(J), OVER = is_over<K>(J);
    const uint32_t g = traj + J.g0;   // the trajectory's random streams
    float* xp = &sm->xp[t];
    float* rv = &sm->rv[t];
    int32_t *cell = &sm->cell[t], *state = &sm->state[t], *sw = &sm->sw[t];
    if (J.resume) {
        // Continue from the state kept at step S = step0 - 1: the ring, the
        // hot state, the statistics clocks; the state-1 steps counted so far
        // complete, a state-1 run going on restarting at S + 1 (the same
        // total); frames continue after frame S / FREQSAVE.
        const int64_t n = J.ntraj;
        for (int r = 0; r < ring_slots; ++r) ring[(int64_t)r * nslots + slot] = J.ck_ring[(int64_t)r * n + traj];
        // a trajectory frozen as non-finite stays so (its first step retires it)
        *xp = (J.counts[(int64_t)LDP_C_FLAGS * n + traj] & LDP_FLAG_NONFINITE) ? __int_as_float(0x7fc00000)
                                                                                : J.ck_xp[traj];
        *rv = J.ck_rv[traj];
        *cell = J.ck_cell[traj];
        *sw = J.ck_sw[traj];
        *state = J.state_final[traj];
        sm->bits[t] = (uint32_t)J.bits[traj];
        sm->init0[t] = J.init_idx0[traj];
        sm->idx2[t] = J.idx2_0[traj];
        sm->tpt2w[t] = J.tpt2_well[traj];
        sm->ckey[t] = J.ck_ckey[traj];
        sm->cflip[t] = J.ck_cflip[traj];
        sm->nflip[t] = J.ck_nflip[traj];
        sm->fpt[t] = J.fpt_last[traj];
        sm->fpt2[t] = J.fpt2_last[traj];
        sm->tpt[t] = J.tpt_last[traj];
        sm->tpt2[t] = J.tpt2_last[traj];
        sm->cgw[t] = INT32_MIN;
        const uint64_t S0 = J.step0 - 1, fs = J.freq_save;
        sm->fidx[t] = (int)(S0 / fs) + 1;
        sm->nxf[t] = (long long)((S0 / fs + 1) * fs);
        sm->sc1[t] = J.counts[(int64_t)LDP_C_STATE1 * n + traj];
        sm->since[t] = (long long)J.step0;
        return;
    }
    for (int r = 0; r < ring_slots; ++r) ring[(int64_t)r * nslots + slot] = make_longlong2((long long)INT64_MIN, 0);
    const double red = J.x0 * J.invL;
    const int c = (int)rint(red);
    const int well = (int)floor(red);
    const double xpd = J.x0 - (double)c * J.Ld;
    int l = 0;
    if (DBL) l = (xpd < J.xcd) ? 0 : 1;
    const Words w0 = philox_at(0, g, TAG_INIT, J.key0, J.key1);
    const int st = J.rs ? (((double)w0.w0 * 0x1p-32 <= J.p_first) ? 0 : 1) : J.init_state;
    double zv, zr;
    gauss_pair_f64(w0.w1, w0.w2, &zv, &zr);
    const double v = J.rv ? J.sig_v0 * zv : J.v0;
    J.state0[traj] = st;
    J.v0s[traj] = v;
    uint32_t bits = 0;
    int init0 = 0, idx2 = 0;
    if (J.at_bottom) {
        if (!DBL && J.fpt && !J.fp_mode) {
            // FPT initial barrier pair (S.h:2187-2211); the ring is empty, so
            // the neighbour has its default state.
            int s0, s1;
            if (well == c) { s0 = st; s1 = f_default_state(J, false, g, c + 1); init0 = c; }
            else { s0 = f_default_state(J, false, g, c - 1); s1 = st; init0 = c - 1; }
            bits |= (s0 ? B_INIT0 : 0u) | (s1 ? B_INIT1 : 0u);
        }
        idx2 = (well == c) ? c : c - 1;
    } else {
        bits |= B_FPT_UP | B_FPT2_UP | B_TPT_UP | B_TPT2_UP;
    }
    for (int j = 0; j < J.n_cg; ++j) {
        J.cg_last[(int64_t)j * J.ntraj + traj] = 0;
        J.cg_well[(int64_t)j * J.ntraj + traj] = well;
        if (!(J.at_bottom && cg_hit32(well, J.cg_size[j]))) bits |= (B_CG0 << j);
    }
    if (!DBL && J.wt) J.wt_tick[traj] = 0;
    sm->bits[t] = bits;
    sm->init0[t] = init0;
    sm->idx2[t] = idx2;
    sm->tpt2w[t] = well;
    sm->ckey[t] = 0;
    sm->cgw[t] = INT32_MIN;
    sm->fidx[t] = 1;
    sm->nxf[t] = (!J.fp_mode && J.freq_save) ? (long long)J.freq_save : INT64_MAX;
    sm->nflip[t] = next_flip(J, g, 0, st);
    sm->fpt[t] = sm->fpt2[t] = sm->tpt[t] = sm->tpt2[t] = 0;
    sm->cflip[t] = 0;
    sm->sc1[t] = 0;
    sm->since[t] = 0;
    *xp = (float)xpd;
    *cell = c;
    *state = st;
    *sw = l ? W_LB : 0;
    *rv = OVER ? (float)(J.sig_r_d * zr) : (float)v;
    if (!J.fp_mode) {
        const float F = force_of(DBL, J, *xp, st);
        f_record(DBL, J, traj, 0, c, *xp, OVER ? 0.0f : (float)v, F, st);
    }
}

__device__ __noinline__ void f_retire(const JobF* Jp, unsigned long long* retired, uint32_t traj, uint64_t steps_done,
                                      int64_t sc1, int cell, float xp, float v, int state, uint32_t flags) {
    const JobF& J = *Jp;
    const int64_t n = J.ntraj;
    J.counts[(int64_t)LDP_C_STATE1 * n + traj] = sc1;
    J.counts[(int64_t)LDP_C_STATE0 * n + traj] = (int64_t)steps_done + 1 - sc1;
    J.counts[(int64_t)LDP_C_STEPS * n + traj] = (int64_t)steps_done;
    if (flags) J.counts[(int64_t)LDP_C_FLAGS * n + traj] |= (int64_t)flags;
    J.x_final[traj] = (double)cell * J.Ld + (double)xp;
    J.v_final[traj] = (double)v;
    J.state_final[traj] = state;
    atomicAdd(J.remaining, ~0ull);   // -1 modulo 2^64
    atomicAdd(retired, 1ull);
}

// Resolves a claimed queue index to (job, trajectory).
__device__ __noinline__ int64_t f_resolve(const int64_t* range_end, const int32_t* range_job,
                                          const int64_t* range_first, const int32_t* nranges, int64_t idx, int* job) {
    int lo = 0, hi = *(volatile const int32_t*)nranges - 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (range_end[mid] > idx) hi = mid; else lo = mid + 1;
    }
    const int64_t begin = lo ? range_end[lo - 1] : 0;
    *job = range_job[lo];
    return range_first[lo] + (idx - begin);
}

// Steps from step s to the next frame (step nxf), flip (step nf) or the
// last step.
__device__ __forceinline__ int steps_to_special(const JobF& J, uint64_t s, long long nxf, long long nf) {
    uint64_t e = (uint64_t)nxf < J.nsteps ? (uint64_t)nxf : J.nsteps;
    e = (uint64_t)nf < e ? (uint64_t)nf : e;
    const uint64_t d = e - s;
    return (int)(d < (uint64_t)kLeftMax ? d : (uint64_t)kLeftMax);
}

// 1 - e^x for x <= 0 in FP32: a degree-5 Taylor polynomial of -expm1 on
// (-1/32, 0] (truncation below 1e-10 relative), 1 - expf(x) below.
__device__ __forceinline__ float one_minus_exp(float x) {
    if (x > -0.03125f)
        return -x * fmaf(x, fmaf(x, fmaf(x, fmaf(x, 1.0f / 120.0f, 1.0f / 24.0f), 1.0f / 6.0f), 0.5f), 1.0f);
    return 1.0f - expf(x);
}

// State at step s of a barrier entered then that was in state sb after its
// missed flip at step nb, and its new pending flip: flip with probability
// c (1 - e^{a lap}) over the steps since, FP32, against the high word of the
// same catch-up uniform the FP64 path draws.
__device__ __forceinline__ int caught_up(const JobF& J, uint32_t g, uint64_t s, long long nb, int sb, const Words& wf,
                                         long long* nf) {
    const float pl = J.c_lapf[J.eq ? 0 : sb] * one_minus_exp(J.a_lapf * (float)((long long)s - nb));
    const uint32_t w0 = philox_at(s, g, TAG_CATCHUP, J.key0, J.key1).w0;
    const int sn = ((pl >= 1.0f) || (w0 < (uint32_t)(pl * 4294967296.0f))) ? (sb ^ 1) : sb;
    *nf = flip_schedule(s, wf.w2, wf.w3, J.ln1m[sn]);
    return sn;
}

// End of a trajectory after step `done` (v: velocity after that step).
__device__ __forceinline__ void retire_lane(const bool OVER, const JobF& J, unsigned long long* retired, RareSm& sm, int t,
                                            uint64_t done, float xp, float v, uint32_t flags) {
    const int state = sm.state[t];
    const int64_t sc1 = sm.sc1[t] + (state ? (int64_t)done + 1 - sm.since[t] : 0);
    if (J.fp_mode && !(flags & LDP_FLAG_NONFINITE) && !(sm.bits[t] & B_HAS_FPT2)) flags |= LDP_FLAG_CENSORED;
    f_retire(&J, retired, sm.traj[t], done, sc1, sm.cell[t], xp, OVER ? 0.0f : v, state, flags);
}

// Keeps the continuation state of a trajectory that completed its last
// step (see JobF::ck_*); rv: the velocity after the step (underdamped) or
// the step's random force (overdamped).
__device__ __noinline__ void f_keep_state(const JobF* Jp, const SlotsDev* Sp, const RareSm* smp, int t, int64_t slot,
                                          uint32_t traj, float xp, float rv, int cell, int sw) {
    const JobF& J = *Jp;
    const SlotsDev& S = *Sp;
    const RareSm& sm = *smp;
    const int64_t n = J.ntraj;
    J.ck_xp[traj] = xp;
    J.ck_rv[traj] = rv;
    J.ck_cell[traj] = cell;
    J.ck_sw[traj] = sw;
    J.ck_ckey[traj] = sm.ckey[t];
    J.ck_cflip[traj] = sm.cflip[t];
    J.ck_nflip[traj] = sm.nflip[t];
    for (int r = 0; r < S.ring_slots; ++r) J.ck_ring[(int64_t)r * n + traj] = S.ring[(int64_t)r * S.nslots + slot];
    J.bits[traj] = (int32_t)sm.bits[t];
    J.init_idx0[traj] = sm.init0[t];
    J.idx2_0[traj] = sm.idx2[t];
    J.tpt2_well[traj] = sm.tpt2w[t];
    J.fpt_last[traj] = sm.fpt[t];
    J.fpt2_last[traj] = sm.fpt2[t];
    J.tpt_last[traj] = sm.tpt[t];
    J.tpt2_last[traj] = sm.tpt2[t];
}

// A lane without a trajectory: at rest in an unbounded band.
__device__ __forceinline__ void idle_lane(RareSm& sm, int t) {
    const float kInf = __int_as_float(0x7f800000);
    sm.job[t] = -1;
    sm.xp[t] = sm.rv[t] = sm.F[t] = 0.f;
    sm.lo[t] = -kInf;
    sm.hi[t] = kInf;
    sm.fixk[t] = make_uint2(0u, 0u);   // no noise
    sm.left[t] = kLeftMax;
    sm.pw[t] = 0;
    sm.j[t] = sm.jh[t] = 0;
}

// Ends a lane's trajectory after step `done` (general step): keeps its
// continuation state when the job asks for it and the trajectory completed,
// then retires it.  The lane's cell, state and slot word in sm are current.
__device__ __noinline__ void f_end_lane(bool OVER, const JobF* Jp, const SlotsDev* Sp, RareSm* smp, int t, int64_t slot,
                                        uint64_t done, float xp, float v, float rv, uint32_t flags) {
    const JobF& J = *Jp;
    RareSm& sm = *smp;
    if (J.ck_xp && !flags && done == J.nsteps)
        f_keep_state(Jp, Sp, smp, t, slot, sm.traj[t], xp, OVER ? rv : v, sm.cell[t], sm.sw[t]);
    retire_lane(OVER, J, Sp->retired, sm, t, done, xp, v, flags);
}

// The general step s of one lane (position already advanced):
// the FP64 step order of ldp_fp64.cu from the index update on, on the lane
// state in shared memory.
__device__ __forceinline__ void general_step(const bool DBL, const bool OVER, const JobF* jobs, const SlotsDev* Sp,
                                             RareSm* smp, int t, int64_t slot, uint64_t s) {
    RareSm& sm = *smp;
    const SlotsDev& S = *Sp;
    const float kInf = __int_as_float(0x7f800000);
    int job = sm.job[t];
    if (job < 0) return;
    const JobF& J = jobs[job];
    const uint32_t traj = sm.traj[t];
    const uint32_t gp = traj + J.g0;   // the trajectory's random streams
    float xp = sm.xp[t];
    const float rv = sm.rv[t];
    float lo = sm.lo[t], hi = sm.hi[t];
    int cell = sm.cell[t], state = sm.state[t], sw = sm.sw[t];
    int left = sm.left[t];

    auto retire = [&](uint64_t done, float v, uint32_t flags) {
        sm.cell[t] = cell;
        sm.state[t] = state;
        sm.sw[t] = sw;
        f_end_lane(OVER, &J, &S, &sm, t, slot, done, xp, v, rv, flags);
        idle_lane(sm, t);
    };

    // Cell (double model: local barrier) entry (UpdateBarrierStateEta,
    // S.h:2025-2068 / D.h:2468-2517): write the state and pending flip step
    // of the key left (*nf) through to the ring and the one-entry cache, take
    // the entered key's from the cache or the ring.  A barrier re-entered
    // before its pending flip has not flipped meanwhile; one whose flip came
    // while it was away (or never visited: created at step 0) is caught up
    // from that step and gets a new schedule (words w2:w3 of TAG_FLIP at s,
    // *wf when the flip of this step already drew them).
    auto enter = [&](int key_prev, int st, int key_cur, long long* nf, Words* wf, bool have_wf) -> int {
        const int64_t n = J.ntraj;
        const int rmask = S.ring_slots - 1;
        if (sw & W_EVICT) red_add(&J.counts[(int64_t)LDP_C_EVICT * n + traj], 1);
        S.ring[(int64_t)(key_prev & rmask) * S.nslots + slot] =
            make_longlong2((long long)key_prev, (*nf << 1) | (long long)st);
        int ps;
        long long nb;
        bool found = true, ev = false;
        if ((sw & W_CVALID) && sm.ckey[t] == key_cur) {
            ps = (sw & W_CSTATE) ? 1 : 0;
            nb = sm.cflip[t];
        } else {
            const longlong2 e = S.ring[(int64_t)(key_cur & rmask) * S.nslots + slot];
            if (e.x == (long long)key_cur) {
                ps = (int)(e.y & 1);
                nb = e.y >> 1;
            } else {
                ps = f_default_state(J, DBL, gp, key_cur);
                nb = 0;
                found = false;
                ev = e.x != (long long)INT64_MIN;
            }
        }
        sm.ckey[t] = key_prev;
        sm.cflip[t] = *nf;
        sw = (sw & W_LB) | W_CVALID | (st ? W_CSTATE : 0) | (ev ? W_EVICT : 0);
        if (!J.eta) return ps;
        if (found && nb > (long long)s) {
            *nf = nb;
            return ps;
        }
        if (!have_wf) *wf = philox_at(s, gp, TAG_FLIP, J.key0, J.key1);
        return caught_up(J, gp, s, nb, found ? (ps ^ 1) : ps, *wf, nf);
    };

    // Renewal statistics (UpdateStatistics, S.h:2334-2592 / D.h:2931-3209)
    // with integer step clocks.  Returns true when a FIRST_PASSAGE
    // trajectory ends.
    auto events = [&](int64_t now, bool dWell, bool dCell, int well) -> bool {
        const int64_t n = J.ntraj;
        int64_t* C = J.counts;
        int64_t* U = J.ssum;
        uint32_t bits = sm.bits[t];
        bool done = false;
        const int evm = J.evm;
        if (!DBL && (evm & EV_WT)) {
            if (dWell) { J.wt_tick[traj] = now; bits |= B_WT_PASSED; }
            else if (dCell && (bits & B_WT_PASSED)) {
                int64_t& nwt = C[(int64_t)LDP_C_WT * n + traj];
                if (nwt < J.tick_cap) J.ticks[(int64_t)traj * J.tick_cap + nwt] = J.wt_tick[traj];
                else C[(int64_t)LDP_C_FLAGS * n + traj] |= LDP_FLAG_TICK_OVERFLOW;
                nwt += 1;
                bits &= ~B_WT_PASSED;
            }
        }
        if (evm & EV_FPT2) {
            if (!DBL && (evm & EV_FPT)) {
                if ((bits & B_FPT_UP) && dCell) {
                    // initial barrier pair (S.h:2364-2388)
                    bits &= ~(B_FPT_UP | B_INIT0 | B_INIT1);
                    sm.fpt[t] = now;
                    int s0, s1, i0;
                    if (well == cell) { s0 = state; s1 = f_ring_state(J, S, slot, false, gp, cell + 1); i0 = cell; }
                    else { s0 = f_ring_state(J, S, slot, false, gp, cell - 1); s1 = state; i0 = cell - 1; }
                    sm.init0[t] = i0;
                    bits |= (s0 ? B_INIT0 : 0u) | (s1 ? B_INIT1 : 0u);
                }
                if (!(bits & B_FPT_UP) && dWell) {
                    bits |= B_FPT_UP;
                    const int64_t d = now - sm.fpt[t];
                    if (!(bits & B_HAS_FPT)) { bits |= B_HAS_FPT; U[(int64_t)LDP_S_FIRST_FPT * n + traj] = d; }
                    red_add(&U[(int64_t)LDP_S_FPT * n + traj], d);
                    red_add(&C[(int64_t)LDP_C_FPT * n + traj], 1);
                    const bool ib = (cell == sm.init0[t]) ? ((bits & B_INIT0) != 0) : ((bits & B_INIT1) != 0);
                    red_add(&C[(int64_t)(ib ? LDP_C_INIT1 : LDP_C_INIT0) * n + traj], 1);
                    red_add(&C[(int64_t)(state ? LDP_C_INST1 : LDP_C_INST0) * n + traj], 1);
                }
            }
            if ((bits & B_FPT2_UP) && dCell) {
                bits &= ~B_FPT2_UP;
                sm.fpt2[t] = now;
                sm.idx2[t] = (well == cell) ? cell : cell - 1;
            }
            const int i2 = sm.idx2[t];
            if (dCell && !(bits & B_FPT2_UP) && i2 != cell && i2 + 1 != cell) {
                const int64_t d = now - sm.fpt2[t];
                if (!(bits & B_HAS_FPT2)) { bits |= B_HAS_FPT2; U[(int64_t)LDP_S_FIRST_FPT2 * n + traj] = d; }
                red_add(&U[(int64_t)LDP_S_FPT2 * n + traj], d);
                red_add(&C[(int64_t)LDP_C_FPT2 * n + traj], 1);
                sm.fpt2[t] = now;
                sm.idx2[t] = (well == cell) ? cell : cell - 1;
                if (evm & EV_FP) done = true;
            }
        }
        if (!DBL && (evm & EV_TPT)) {
            if (dCell) { bits &= ~B_TPT_UP; sm.tpt[t] = now; }
            if (!(bits & B_TPT_UP) && dWell) {
                bits |= B_TPT_UP;
                const int64_t d = now - sm.tpt[t];
                if (!(bits & B_HAS_TPT)) { bits |= B_HAS_TPT; U[(int64_t)LDP_S_FIRST_TPT * n + traj] = d; }
                red_add(&U[(int64_t)LDP_S_TPT * n + traj], d);
                red_add(&C[(int64_t)LDP_C_TPT * n + traj], 1);
            }
            if (dCell) {
                if (bits & B_TPT2_UP) bits &= ~B_TPT2_UP;
                else if (well != sm.tpt2w[t]) {
                    const int64_t d = now - sm.tpt2[t];
                    if (!(bits & B_HAS_TPT2)) { bits |= B_HAS_TPT2; U[(int64_t)LDP_S_FIRST_TPT2 * n + traj] = d; }
                    red_add(&U[(int64_t)LDP_S_TPT2 * n + traj], d);
                    red_add(&C[(int64_t)LDP_C_TPT2 * n + traj], 1);
                }
                sm.tpt2[t] = now;
                sm.tpt2w[t] = well;
            }
        }
        // An FPTCG evaluation at the well of the previous one changes nothing
        // (every entry it hits already holds that well), so it is skipped.
        if ((evm & EV_CG) && dCell && well != sm.cgw[t]) {
            sm.cgw[t] = well;
            for (int jj = 0; jj < J.n_cg; ++jj) {
                if (cg_hit32(well, J.cg_size[jj])) {
                    const int64_t o = (int64_t)jj * n + traj;
                    if (bits & (B_CG0 << jj)) {
                        bits &= ~(B_CG0 << jj);
                        J.cg_last[o] = now;
                        J.cg_well[o] = well;
                    } else if (well != J.cg_well[o]) {
                        red_add(&U[(int64_t)(LDP_S_CG0 + jj) * n + traj], now - J.cg_last[o]);
                        red_add(&C[(int64_t)(LDP_C_CG0 + jj) * n + traj], 1);
                        J.cg_last[o] = now;
                        J.cg_well[o] = well;
                    }
                }
            }
        }
        sm.bits[t] = bits;
        return done;
    };

    if (xp > lo && xp < hi && (long long)s != sm.nflip[t]) {
        // Only the countdown ran out: a frame and/or the last step.
        const float F = sm.F[t];
        const float vk = OVER ? 0.0f : fmaf(F, J.hdt_invM, rv);
        if ((long long)s == sm.nxf[t]) {
            f_record(DBL, J, traj, sm.fidx[t], cell, xp, vk, F, state);
            sm.fidx[t] += 1;
            sm.nxf[t] += (long long)J.freq_save;
        }
        sm.left[t] = steps_to_special(J, s, sm.nxf[t], sm.nflip[t]);
        if (s == J.nsteps) retire(s, vk, 0);
        return;
    }
    if (!(fabsf(xp) < kInf)) {
        retire(s - 1, rv, LDP_FLAG_NONFINITE);
        return;
    }
    const int cell_prev = cell;
    const int lb_prev = sw & W_LB;
    const int well_prev = cell_prev - (lo < 0.0f ? 1 : 0);
    const bool moved = !(xp > lo && xp < hi);
    if (moved) {
        if (xp >= J.halfL) { xp -= J.L; ++cell; }
        else if (xp < -J.halfL) { xp += J.L; --cell; }
        if (!(xp >= -J.halfL && xp < J.halfL)) {
            // more than one cell in one step
            const float k = floorf(xp * J.invLf + 0.5f);
            xp = fmaf(-k, J.L, xp);
            cell += (int)k;
            if (xp >= J.halfL) { xp -= J.L; ++cell; }
            else if (xp < -J.halfL) { xp += J.L; --cell; }
        }
    }
    const int well = cell - (xp < 0.0f ? 1 : 0);
    const int lb = DBL ? (xp < J.xc ? 0 : 1) : 0;
    const bool dCell = cell != cell_prev;
    const bool dWell = well != well_prev;
    const bool dKey = DBL ? (lb != lb_prev) : dCell;
    // the current barrier flips at its pending flip step and draws the next
    // one; a barrier change takes the entered barrier's schedule
    const bool flip = (long long)s == sm.nflip[t];
    int st = state ^ (int)flip;
    long long nf = sm.nflip[t];
    Words wf{};
    if (flip) {
        wf = philox_at(s, gp, TAG_FLIP, J.key0, J.key1);
        nf = flip_schedule(s, wf.w0, wf.w1, J.ln1m[st]);
    }
    if (dKey) st = enter(fkey(DBL, cell_prev, lb_prev), st, fkey(DBL, cell, lb), &nf, &wf, flip);
    if (DBL) sw = (sw & ~W_LB) | (lb ? W_LB : 0);
    if (st != state) {
        if (st) sm.since[t] = (long long)s;
        else sm.sc1[t] += (long long)s - sm.since[t];
        state = st;
    }
    if (J.eta && (flip || dKey)) {
        sm.nflip[t] = nf;
        left = 0;   // recompute the countdown below
    }
    band_of(DBL, J, xp, &lo, &hi);
    const float F = force_of(DBL, J, xp, state);
    bool finish = false;
    if (dCell || dWell) finish = events((int64_t)s, dWell, dCell, well);
    const float vk = OVER ? 0.0f : fmaf(F, J.hdt_invM, rv);
    if (left == 0) {
        if ((long long)s == sm.nxf[t]) {
            f_record(DBL, J, traj, sm.fidx[t], cell, xp, vk, F, state);
            sm.fidx[t] += 1;
            sm.nxf[t] += (long long)J.freq_save;
        }
        if (s == J.nsteps) finish = true;
        left = steps_to_special(J, s, sm.nxf[t], sm.nflip[t]);
    }
    sm.xp[t] = xp;
    sm.cell[t] = cell;
    sm.state[t] = state;
    sm.sw[t] = sw;
    sm.lo[t] = lo;
    sm.hi[t] = hi;
    sm.F[t] = F;
    sm.left[t] = left;
    if (finish) retire(s, vk, 0);
}

// The last step after s whose block index has the same high word as the
// next step's: a special step, since the lane's Philox constants hold it.
__device__ __forceinline__ long long block_wrap(uint64_t s) { return (long long)(((s >> 34) + 1) << 34); }

// The high word of the lane's block index and its Philox constants for next
// step s + 1.
__device__ __forceinline__ void bind_block(const JobF& J, RareSm& sm, int t, uint64_t s) {
    sm.jh[t] = (uint32_t)(s >> 34);
    sm.fix[t] = philox_fix(sm.traj[t] + J.g0, (uint32_t)(s >> 34), J.key0, J.key1);
    sm.fixk[t] = make_uint2(J.key0 + 2u * 0x9E3779B9u, __float_as_uint(J.bm_k));
}

// The countdown from step s to the next frame or to nev, the first step that
// is special for another reason; the lane's P_* word.
__device__ __forceinline__ void count_down(const JobF& J, RareSm& sm, int t, uint64_t s, long long nev, int& left,
                                           uint32_t& pw) {
    const long long nxf = sm.nxf[t];
    long long d = (nxf < nev ? nxf : nev) - (long long)s;
    d = d > 1 ? d : 1;   // (both lie after s)
    if (nxf < nev && d <= (long long)kLeftMax && !J.write_x) pw |= P_FRAME;
    sm.nev[t] = nev;
    left = (int)(d < (long long)kLeftMax ? d : (long long)kLeftMax);
}

// After a special step s (or before the first step, s one less): the word of
// the lane's quick steps and its countdown.  A pair is formed when a crossing
// of the nearer cell edge would change the barrier and restart the transition
// clocks and nothing else, and stays
// one, whatever the number of crossings, until the next special step: the
// neighbour is the cached cell, no statistic fires, no eviction is pending.
// The countdown also ends at the neighbour's pending flip, past which its
// cached state is no longer known (P_OVERDUE).
__device__ __noinline__ void settle(bool DBL, const JobF* Jp, RareSm* smp, int t, uint64_t s, float xp) {
    const JobF& J = *Jp;
    RareSm& sm = *smp;
    const int state = sm.state[t], sw = sm.sw[t], cell = sm.cell[t];
    uint32_t pw = (state ? P_S0 : 0u) | (J.edge_flat ? P_FAST : 0u) | P_MODE * (uint32_t)J.mode;
    long long nev = sm.nflip[t] < (long long)J.nsteps ? sm.nflip[t] : (long long)J.nsteps;
    const long long wrap = block_wrap(s);
    nev = wrap < nev ? wrap : nev;
    if ((s & ((1ull << 34) - 1)) == 0) bind_block(J, sm, t, s);   // a new high word from the next step on
    if ((sw & W_CVALID) && !(sw & W_EVICT)) {
        const bool right = !(xp < 0.0f);
        const int lb = sw & W_LB;
        const int well = cell - (right ? 0 : 1);
        const int key = fkey(DBL, right ? cell + 1 : cell - 1, lb ^ 1);
        const uint32_t bits = sm.bits[t];
        const int evm = J.evm;
        bool ok = sm.ckey[t] == key && (!DBL || (lb != 0) == right);
        ok = ok && !((evm & EV_FPT) && (bits & B_FPT_UP));
        ok = ok && !((evm & EV_FPT2) && ((bits & B_FPT2_UP) || sm.idx2[t] != well));
        ok = ok && !((evm & EV_TPT) && !(bits & B_TPT2_UP) && sm.tpt2w[t] != well);
        ok = ok && !((evm & EV_CG) && sm.cgw[t] != well);
        ok = ok && !((evm & EV_WT) && (bits & B_WT_PASSED));
        if (ok) {
            pw |= P_PAIR | (right ? P_RIGHT : 0u) | ((sw & W_CSTATE) ? P_S1 : 0u);
            if (sm.cflip[t] <= (long long)s) pw |= P_OVERDUE;
            else nev = sm.cflip[t] < nev ? sm.cflip[t] : nev;
        }
    }
    int left;
    count_down(J, sm, t, s, nev, left, pw);
    sm.left[t] = left;
    sm.pw[t] = pw;
}

// The current barrier's flip at step s and nothing else, the lane in its
// pair's first cell: its new state and pending flip, the state-1 run, the
// force, the countdown; a pair stays one.
__device__ __forceinline__ bool only_flip(const JobF& J, const RareSm& sm, int t, uint64_t s, uint32_t pw) {
    return !(pw & P_CROSSED) && (long long)s == sm.nflip[t] && (long long)s < sm.nxf[t] &&
           s < J.nsteps && (s & ((1ull << 34) - 1)) != 0;
}
__device__ __forceinline__ void flip_here(const bool DBL, const JobF& J, RareSm& sm, int t, uint64_t s, float xp,
                                          float& F, int& left, uint32_t& pw) {
    pw = (pw & ~P_FRAME) ^ P_S0;
    const int st = (pw & P_S0) ? 1 : 0;
    const Words w = philox_at(s, sm.traj[t] + J.g0, TAG_FLIP, J.key0, J.key1);
    const long long nf = flip_schedule(s, w.w0, w.w1, J.ln1m[st]);
    if (st) sm.since[t] = (long long)s;
    else sm.sc1[t] += (long long)s - sm.since[t];
    sm.state[t] = st;
    sm.nflip[t] = nf;
    F = force_of(DBL, J, xp, st);
    long long nev = block_wrap(s);
    nev = (long long)J.nsteps < nev ? (long long)J.nsteps : nev;
    nev = nf < nev ? nf : nev;
    if (sm.cflip[t] <= (long long)s) pw |= P_OVERDUE;
    if ((pw & (P_PAIR | P_OVERDUE)) == P_PAIR) nev = sm.cflip[t] < nev ? sm.cflip[t] : nev;
    count_down(J, sm, t, s, nev, left, pw);
}

// Leaves a pair: the lane state as general steps would have left it (the
// ring entry of the cell first left, the transition-path clocks, and, in the
// pair's other cell, the swapped barriers).
__device__ __forceinline__ void unpair(const bool DBL, const JobF& J, const SlotsDev& S, RareSm& sm, int t,
                                       int64_t slot, uint32_t pw) {
    if (!(pw & P_CROSSED)) return;
    const int cell = sm.cell[t], sw = sm.sw[t];
    const int key = fkey(DBL, cell, sw & W_LB);
    const int st = (pw & P_S0) ? 1 : 0;
    const long long nf = sm.nflip[t];
    S.ring[(int64_t)(key & (S.ring_slots - 1)) * S.nslots + slot] =
        make_longlong2((long long)key, (nf << 1) | (long long)st);
    if (J.evm & EV_TPT) {
        const long long xs = sm.xs[t];
        sm.bits[t] &= ~(B_TPT_UP | B_TPT2_UP);
        sm.tpt[t] = xs;
        sm.tpt2[t] = xs;
        sm.tpt2w[t] = cell - ((pw & P_RIGHT) ? 0 : 1);
    }
    if (pw & P_SWAP) {
        sm.cell[t] = cell + ((pw & P_RIGHT) ? 1 : -1);
        sm.state[t] = (pw & P_S1) ? 1 : 0;
        sm.ckey[t] = key;
        sm.nflip[t] = sm.cflip[t];
        sm.cflip[t] = nf;
        sm.sw[t] = (DBL ? ((sw & W_LB) ^ W_LB) : (sw & W_LB)) | W_CVALID | (st ? W_CSTATE : 0);
    }
}

// Leaves a pair's crossings behind: unpair, and the word of the same pair seen
// from the cell the lane is in.
__device__ __forceinline__ void from_here(const bool DBL, const JobF& J, const SlotsDev& S, RareSm& sm, int t,
                                          int64_t slot, uint32_t& pw) {
    unpair(DBL, J, S, sm, t, slot, pw);
    if (pw & P_SWAP) {   // the lane's cell is its pair's first now
        pw ^= P_RIGHT;
        if (((pw & P_S0) != 0u) != ((pw & P_S1) != 0u)) pw ^= P_S0 | P_S1;
    }
    pw &= ~(P_SWAP | P_CROSSED);
}

// A special step that is not a quick one: out of line, on the lane state in
// shared memory, so that the hot loop's registers do not carry its working
// set.  sm.left: 0 when the countdown ends at s.
template <int K>
__device__ __noinline__ void special_step(const JobF* jobs, const SlotsDev* Sp, RareSm* smp, int t, int64_t slot,
                                          uint64_t s) {
    RareSm& sm = *smp;
    const SlotsDev& S = *Sp;
    const int job = sm.job[t];
    if (job < 0) {
        sm.left[t] = kLeftMax;
        return;
    }
    const JobF& J = jobs[job];
    const bool DBL = is_double<K>(J), OVER = is_over<K>(J);
    uint32_t pw = sm.pw[t];
    from_here(DBL, J, S, sm, t, slot, pw);
    const float xp = sm.xp[t], lo = sm.lo[t], hi = sm.hi[t];
    if (sm.left[t] == 0 && xp > lo && xp < hi && only_flip(J, sm, t, s, pw)) {
        float F;
        int left;
        flip_here(DBL, J, sm, t, s, xp, F, left, pw);
        sm.F[t] = F;
        sm.left[t] = left;
        sm.pw[t] = pw;
        return;
    }
    if ((pw & P_PAIR) && (pw & P_OVERDUE) && sm.left[t] != 0 &&
        ((pw & P_RIGHT) ? xp >= J.halfL : xp < -J.halfL)) {
        // The pair's edge crossed, the other cell's pending flip past: as a
        // quick crossing, the barrier entered caught up from that flip.
        const bool right = (pw & P_RIGHT) != 0u;
        const float xn = right ? xp - J.L : xp + J.L;
        const float e1 = right ? -J.halfL : J.edge_hi, e2 = right ? J.edge_lo : J.halfL;
        if (xn > e1 && xn < e2) {   // (no breakpoint between the edge and edge_lo or edge_hi)
            const int st = sm.state[t];
            const uint32_t g = sm.traj[t] + J.g0;
            long long nf;
            const int now = caught_up(J, g, s, sm.cflip[t], (pw & P_S1) ? 0 : 1, philox_at(s, g, TAG_FLIP, J.key0, J.key1),
                                      &nf);
            pw = (pw | P_CROSSED | P_SWAP) & ~P_S1;
            if (now) pw |= P_S1;
            sm.cflip[t] = nf;
            sm.xs[t] = (long long)s;
            if (now != st) {
                if (now) sm.since[t] = (long long)s;
                else sm.sc1[t] += (long long)s - sm.since[t];
            }
            unpair(DBL, J, S, sm, t, slot, pw);   // into the cell entered
            sm.xp[t] = xn;
            sm.lo[t] = e1;
            sm.hi[t] = e2;
            sm.F[t] = J.edge_flat ? flat_force(DBL) : force_of(DBL, J, xn, now);
            settle(DBL, &J, &sm, t, s, xn);
            return;
        }
    }
    general_step(DBL, OVER, jobs, Sp, smp, t, slot, s);
    if (sm.job[t] < 0) return;
    settle(DBL, &J, &sm, t, s, sm.xp[t]);
}

// The frame of step s, at which the countdown ends for it and nothing else
// (P_FRAME).
__device__ __forceinline__ void only_frame(const JobF& J, RareSm& sm, int t, uint64_t s, float xp, int& left,
                                           uint32_t& pw) {
    const int fidx = sm.fidx[t];
    int cell = sm.cell[t];
    if (pw & P_SWAP) cell += (pw & P_RIGHT) ? 1 : -1;
    if (fidx < J.nframe && J.fx) J.fx[(int64_t)fidx * J.ntraj + sm.traj[t]] = (double)cell * J.Ld + (double)xp;
    sm.fidx[t] = fidx + 1;
    const long long nxf = sm.nxf[t] + (long long)J.freq_save, nev = sm.nev[t];
    sm.nxf[t] = nxf;
    const long long d = (nxf < nev ? nxf : nev) - (long long)s;
    if (!(nxf < nev && d <= (long long)kLeftMax)) pw &= ~P_FRAME;
    left = (int)(d < (long long)kLeftMax ? d : (long long)kLeftMax);
}

// The quick steps: the commonest special steps, in the hot loop, with the
// state the general step leaves (unpair fills in what a pair's crossings leave
// open).  Returns false when the step needs special_step.
//  * A frame, the position inside its band.
//  * A band change inside the cell (a flank entered or left) that changes
//    neither the well nor the local barrier.
//  * A crossing of the pair's edge into the flat band of the other cell: the
//    barriers change places.
__device__ __forceinline__ bool quick_step(const bool DBL, const bool flips, const JobF& J, RareSm& sm, int t,
                                           uint64_t s, bool countdown, float& xp,
                                           float& lo, float& hi, float& F, int& left, uint32_t& pw) {
    const uint32_t swapped = pw & P_SWAP;
    if (countdown) {
        if (!(xp > lo && xp < hi)) return false;
        if (!(pw & P_FRAME)) {
            if (flips && only_flip(J, sm, t, s, pw)) {
                flip_here(DBL, J, sm, t, s, xp, F, left, pw);
                return true;
            }
            // the other cell's pending flip, and nothing else: caught up with
            // when the cell is entered
            const bool other = (pw & (P_PAIR | P_OVERDUE)) == P_PAIR &&
                               (swapped ? sm.nflip[t] : sm.cflip[t]) == (long long)s && s != J.nsteps;
            const long long nxf = sm.nxf[t], own = swapped ? sm.cflip[t] : sm.nflip[t];
            if (!other || (long long)s == nxf || (long long)s == own) return false;
            long long nev = block_wrap(s - 1);
            if (nev == (long long)s) return false;
            nev = (long long)J.nsteps < nev ? (long long)J.nsteps : nev;
            nev = own < nev ? own : nev;
            pw |= P_OVERDUE;
            count_down(J, sm, t, s, nev, left, pw);
            return true;
        }
        only_frame(J, sm, t, s, xp, left, pw);
        return true;
    }
    if (!(pw & P_FAST)) return false;
    const float hL = J.halfL;
    const int st = (swapped ? pw & P_S1 : pw & P_S0) ? 1 : 0;
    if (fabsf(xp) < hL) {
        if ((xp < 0.0f) != (lo < 0.0f)) return false;
        if (!DBL) {
            const float a = fabsf(xp), w = J.w;
            if (a == w || a == 0.0f) return false;
            const bool in = a < w, neg = xp < 0.0f;
            const float m0 = in ? 0.0f : w, m1 = in ? w : hL;
            lo = neg ? -m1 : m0;
            hi = neg ? -m0 : m1;
            F = in ? copysignf(J.slope[st], xp) : 0.0f;
        } else {
            const float xc = J.xc;
            if ((xp < xc) != (lo < xc)) return false;   // lo < xc: local barrier 0
            float l2, h2;
            band_of(DBL, J, xp, &l2, &h2);
            if (!(xp > l2 && xp < h2)) return false;
            lo = l2;
            hi = h2;
            F = force_of(DBL, J, xp, st);
        }
        return true;
    }
    if ((pw & (P_PAIR | P_OVERDUE)) != P_PAIR) return false;
    const bool right = ((pw & P_RIGHT) != 0u) != (swapped != 0u);   // the pair's other cell is the right neighbour
    const float xn = right ? xp - J.L : xp + J.L;
    const float e1 = right ? -hL : J.edge_hi, e2 = right ? J.edge_lo : hL;
    if (!(right ? xp >= hL : xp < -hL) || !(xn > e1 && xn < e2)) return false;
    pw = (pw ^ P_SWAP) | P_CROSSED;
    sm.xs[t] = (long long)s;
    if (((pw & P_S0) != 0u) != ((pw & P_S1) != 0u)) {
        if (st) sm.sc1[t] += (long long)s - sm.since[t];
        else sm.since[t] = (long long)s;
    }
    xp = xn;
    lo = e1;
    hi = e2;
    F = flat_force(DBL);
    return true;
}

// The quick steps of jobs whose other special steps are frequent too (JobF::
// full): those of quick_step, flips of the current barrier in every position
// of a pair, crossings into a barrier whose pending flip has passed, frames with
// the series of WRITEX, and all of these at the same step.  The step order is
// the general step's: position and cell, flip, cell entry, force, frame.  Returns
// false, and has done nothing, when the step needs special_step.
template <bool DBL, bool OVER>
__device__ __forceinline__ bool full_quick_step(const JobF& J, const SlotsDev& S, RareSm& sm, int t, uint64_t s,
                                                bool countdown, float& xp, float rv, float& lo, float& hi, float& F,
                                                int& left, uint32_t& pw) {
    const bool in = xp > lo && xp < hi;
    const bool frame = countdown && (pw & P_FRAME) != 0u;   // and nothing else
    if (in && frame) {
        only_frame(J, sm, t, s, xp, left, pw);
        return true;
    }
    if (in && countdown && !frame && only_flip(J, sm, t, s, pw)) {
        flip_here(DBL, J, sm, t, s, xp, F, left, pw);
        return true;
    }
    const bool other = countdown && !frame;   // a flip, a barrier's pending flip, the last step ...
    if (other && (s == J.nsteps || (s & ((1ull << 34) - 1)) == 0)) return false;
    float xn = xp, l2 = lo, h2 = hi;
    bool cross = false;
    if (!in) {
        const float hL = J.halfL;
        if (fabsf(xp) < hL) {
            if ((xp < 0.0f) != (lo < 0.0f)) return false;
            if (DBL && (xp < J.xc) != (lo < J.xc)) return false;   // lo < xc: local barrier 0
        } else {
            if (!(pw & P_PAIR)) return false;
            // the pair's other cell is the right neighbour
            const bool right = ((pw & P_RIGHT) != 0u) != ((pw & P_SWAP) != 0u);
            xn = right ? xp - J.L : xp + J.L;
            if (!(right ? xp >= hL && xn > -hL && xn < J.edge_lo : xp < -hL && xn < hL && xn > J.edge_hi)) return false;
            cross = true;
        }
        band_of(DBL, J, xn, &l2, &h2);
        if (!(xn > l2 && xn < h2)) return false;
    }
    bool flip = false;
    if (other) {
        const long long a = sm.nflip[t], b = sm.cflip[t];
        const bool swapped = (pw & P_SWAP) != 0u;
        flip = (swapped ? b : a) == (long long)s;
        if ((pw & P_PAIR) && (swapped ? a : b) == (long long)s) pw |= P_OVERDUE;
    }
    const bool overdue = cross && (pw & P_OVERDUE);
    if (flip || overdue) {
        const int64_t slot = (int64_t)blockIdx.x * blockDim.x + t;
        from_here(DBL, J, S, sm, t, slot, pw);
        const uint32_t g = sm.traj[t] + J.g0;
        const Words w = philox_at(s, g, TAG_FLIP, J.key0, J.key1);
        // the state-1 run of the lane's barrier
        auto state_now = [&](int st) {
            if (st) sm.since[t] = (long long)s;
            else sm.sc1[t] += (long long)s - sm.since[t];
        };
        if (flip) {
            pw ^= P_S0;
            const int st = (pw & P_S0) ? 1 : 0;
            sm.state[t] = st;
            sm.nflip[t] = flip_schedule(s, w.w0, w.w1, J.ln1m[st]);
            state_now(st);
        }
        if (overdue) {
            long long nf;
            const int st = caught_up(J, g, s, sm.cflip[t], (pw & P_S1) ? 0 : 1, w, &nf);
            if (st != ((pw & P_S0) ? 1 : 0)) state_now(st);
            sm.cflip[t] = nf;
            sm.xs[t] = (long long)s;
            pw = (pw & ~(P_S1 | P_OVERDUE)) | P_CROSSED | P_SWAP | (st ? P_S1 : 0u);
            from_here(DBL, J, S, sm, t, slot, pw);   // into the cell entered
        }
    }
    if (cross && !overdue) {
        pw = (pw ^ P_SWAP) | P_CROSSED;
        sm.xs[t] = (long long)s;
        if (((pw & P_S0) != 0u) != ((pw & P_S1) != 0u)) {
            if ((pw & P_SWAP) ? pw & P_S1 : pw & P_S0) sm.since[t] = (long long)s;
            else sm.sc1[t] += (long long)s - sm.since[t];
        }
    }
    const int st = ((pw & P_SWAP) ? pw & P_S1 : pw & P_S0) ? 1 : 0;
    if (!in || flip) F = force_of(DBL, J, xn, st);
    xp = xn;
    lo = l2;
    hi = h2;
    if (frame && !overdue) {
        only_frame(J, sm, t, s, xp, left, pw);
        return true;
    }
    if (countdown && (long long)s == sm.nxf[t]) {
        const int fidx = sm.fidx[t];
        if (fidx < J.nframe) {
            int cell = sm.cell[t];
            if (pw & P_SWAP) cell += (pw & P_RIGHT) ? 1 : -1;
            const int64_t o = (int64_t)fidx * J.ntraj + sm.traj[t];
            if (J.fx) J.fx[o] = (double)cell * J.Ld + (double)xp;
            if (J.write_x) record_extra(DBL, J, o, xp, OVER ? 0.0f : fmaf(F, J.hdt_invM, rv), F, st);
        }
        sm.fidx[t] = fidx + 1;
        sm.nxf[t] += (long long)J.freq_save;
    }
    if (countdown || overdue) {
        const long long a = sm.nflip[t], b = sm.cflip[t];
        const bool swapped = (pw & P_SWAP) != 0u;
        const long long own = swapped ? b : a, other = swapped ? a : b;
        long long nev = block_wrap(s);
        nev = (long long)J.nsteps < nev ? (long long)J.nsteps : nev;
        nev = own < nev ? own : nev;
        if (other <= (long long)s) pw |= P_OVERDUE;
        if ((pw & (P_PAIR | P_OVERDUE)) == P_PAIR) nev = other < nev ? other : nev;
        pw &= ~P_FRAME;
        count_down(J, sm, t, s, nev, left, pw);
    }
    return true;
}

// One step's move.
__device__ __forceinline__ void f_move(const bool OVER, float& xp, float& rv, float F, float c1, float c2, float c3,
                                       float nz) {
    if (OVER) {
        xp = fmaf(F, c1, xp);
        xp = xp + nz;
        xp = xp + rv;
        rv = nz;
    } else {
        rv = fmaf(F, c1, rv);
        xp = fmaf(rv, c2, xp);
        rv = fmaf(c3, rv, nz);
        xp = fmaf(rv, c2, xp);
    }
}

// One lane's steps 4j+1+h .. 4j+4 one by one, step 4j+1+h a special one that
// is moved already; the later steps' noise in sm.nz.  Out of line, on the lane
// state in shared memory.
template <int K>
__device__ __noinline__ void slow_steps(const JobF* jobs, const SlotsDev* Sp, RareSm* smp, int t, int64_t slot,
                                        uint64_t j, int h) {
    RareSm& sm = *smp;
    int job = sm.job[t];
    bool moved = true;
    int next = 0;
#pragma unroll 1
    for (; h < 4; ++h) {
        const JobF& J = jobs[job < 0 ? 0 : job];
        const bool OVER = is_over<K>(J);
        const float c1 = OVER ? J.c_drift : J.hdt_invM;
        if (!moved && job >= 0) {
            float xp = sm.xp[t], rv = sm.rv[t];
            f_move(OVER, xp, rv, sm.F[t], c1, J.hdt, J.expg, sm.nz[next++][t]);
            sm.xp[t] = xp;
            sm.rv[t] = rv;
            sm.left[t] -= 1;
        }
        const float xp = sm.xp[t];
        if (moved || !(xp > sm.lo[t] && xp < sm.hi[t]) || sm.left[t] == 0) {
            special_step<K>(jobs, Sp, smp, t, slot, 4 * j + 1 + h);
            job = sm.job[t];
            if (job < 0) {
                sm.rv[t] = 0.f;
                return;
            }
        }
        if (!OVER) sm.rv[t] = fmaf(sm.F[t], c1, sm.rv[t]);
        moved = false;
    }
}

// Lowest and highest of four, NaN if one is.
__device__ __forceinline__ void range4(float a, float b, float c, float d, float* mn, float* mx) {
    float u, v;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(u) : "f"(a), "f"(b), "f"(c));
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(v) : "f"(a), "f"(b), "f"(c));
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(*mn) : "f"(u), "f"(d));
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(*mx) : "f"(v), "f"(d));
}

}  // namespace

// Resident 256-thread blocks per SM the register budget is sized for.  Three
// (80 registers) leave room on the SM for the finished jobs' mean-square
// displacements and step their own lanes 3-4 % faster; four (64) hold 151552
// trajectories instead of 113664 and hide more latency: 2 x 65536 x 48000 16.8
// / 15.1 ms, 4 x 65536 x 120000 59.4 / 56.6, a graph of two times 80000 x 24000
// 19.4 / 20.2, 20011 double 6.9 / 7.2.  So four where the trajectories of the
// queue do not fit three blocks (Fp32Queue::wide).  (Four at 56 registers,
// which leave that room too: 15.0, 56.4, 20.3, 7.8.)
constexpr int kNarrowBlocks = 3, kWideBlocks = 4;

namespace {

// A lane's per-job constants, band, force and countdown from its position
// (sm.xp) and statistics state; s: its next step.
__device__ __forceinline__ void bind_lane(const bool DBL, const JobF& J, RareSm& sm, int t, uint32_t traj, uint64_t s) {
    sm.traj[t] = traj;
    sm.j[t] = (uint32_t)((s - 1) >> 2);
    bind_block(J, sm, t, s - 1);
    const float xp = sm.xp[t];
    float lo, hi;
    band_of(DBL, J, xp, &lo, &hi);
    sm.lo[t] = lo;
    sm.hi[t] = hi;
    sm.F[t] = force_of(DBL, J, xp, sm.state[t]);
    settle(DBL, &J, &sm, t, s - 1, xp);
}

// The state a slot kept since the last launch, into sm.
template <int K>
__device__ __noinline__ void load_slot(const QueueDev* qp, const SlotsDev* Sp, RareSm* smp, int t, int64_t slot) {
    const SlotsDev& S = *Sp;
    RareSm& sm = *smp;
    idle_lane(sm, t);
    const int job = (slot < S.nslots) ? S.job[slot] : -1;
    if (job < 0) return;
    const JobF& J = qp->jobs[job];
    const bool DBL = is_double<K>(J);
    const uint32_t traj = (uint32_t)S.traj[slot];
    const uint64_t s = (uint64_t)S.step[slot];
    sm.job[t] = job;
    sm.xp[t] = S.xp[slot];
    sm.rv[t] = S.rv[slot];
    sm.cell[t] = S.cell[slot];
    const int st = S.st[slot];
    sm.state[t] = st & 1;
    sm.sw[t] = st >> 1;
    sm.bits[t] = (uint32_t)J.bits[traj];
    sm.init0[t] = J.init_idx0[traj];
    sm.idx2[t] = J.idx2_0[traj];
    sm.tpt2w[t] = J.tpt2_well[traj];
    sm.fpt[t] = J.fpt_last[traj];
    sm.fpt2[t] = J.fpt2_last[traj];
    sm.tpt[t] = J.tpt_last[traj];
    sm.tpt2[t] = J.tpt2_last[traj];
    sm.ckey[t] = S.ckey[slot];
    sm.cflip[t] = S.cflip[slot];
    sm.sc1[t] = S.sc1[slot];
    sm.since[t] = S.since[slot];
    sm.cgw[t] = S.cgw[slot];
    sm.fidx[t] = S.fidx[slot];
    sm.nxf[t] = S.nxf[slot];
    sm.nflip[t] = S.nflip[slot];
    bind_lane(DBL, J, sm, t, traj, s);
}

// A lane's state into its slot, until the next launch.
template <int K>
__device__ __noinline__ void save_slot(const QueueDev* qp, const SlotsDev* Sp, RareSm* smp, int t, int64_t slot) {
    const SlotsDev& S = *Sp;
    RareSm& sm = *smp;
    if (slot >= S.nslots) return;
    const int job = sm.job[t];
    S.job[slot] = job;
    if (job < 0) return;
    const JobF& J = qp->jobs[job];
    const bool DBL = is_double<K>(J);
    const uint32_t traj = sm.traj[t];
    unpair(DBL, J, S, sm, t, slot, sm.pw[t]);
    S.traj[slot] = traj;
    S.step[slot] = (int64_t)(((uint64_t)sm.jh[t] << 34 | (uint64_t)sm.j[t] << 2) + 1);
    S.xp[slot] = sm.xp[t];
    S.rv[slot] = sm.rv[t];
    S.cell[slot] = sm.cell[t];
    S.st[slot] = sm.state[t] | (sm.sw[t] << 1);
    S.ckey[slot] = sm.ckey[t];
    S.cflip[slot] = sm.cflip[t];
    S.sc1[slot] = sm.sc1[t];
    S.since[slot] = sm.since[t];
    S.cgw[slot] = sm.cgw[t];
    S.fidx[slot] = sm.fidx[t];
    S.nxf[slot] = sm.nxf[t];
    S.nflip[slot] = sm.nflip[t];
    J.bits[traj] = (int32_t)sm.bits[t];
    J.init_idx0[traj] = sm.init0[t];
    J.idx2_0[traj] = sm.idx2[t];
    J.tpt2_well[traj] = sm.tpt2w[t];
    J.fpt_last[traj] = sm.fpt[t];
    J.fpt2_last[traj] = sm.fpt2[t];
    J.tpt_last[traj] = sm.tpt[t];
    J.tpt2_last[traj] = sm.tpt2[t];
}

// How a launch that finds fewer items than it has lanes shares them out
// (avail: items unclaimed at the last publication), by share_out.  Returns the
// lanes a warp fills at its first claim, 0 for a warp that leaves the items to
// others, 32 where every lane is wanted.  (24000 steps, frames every 20, warps
// filled one after the other / this way: 16000 trajectories 5.6 / 3.0 ms,
// 32000 5.8 / 3.4, 60000 5.7 / 4.3 overdamped; 1024 2.5 / 1.9.  One warp to a
// scheduler while 32 lanes hold the items: two half as full cost 3.8 ms at
// 16000.)  A warp's turn goes by its SM and by
// its block's rank among the SM's blocks: a count of arrivals, which need not
// start at zero (launches add one block per SM and rank); block indices do
// not tell the SM (6 of 148 SMs hold two of blocks 0-147, 6 none).  All
// threads of the block call.
__device__ __forceinline__ int first_claim(unsigned long long avail, const SlotsDev& S) {
    __shared__ unsigned rank;
    const unsigned sms = (unsigned)S.sms, wpb = blockDim.x >> 5, blocks = gridDim.x / sms;
    const Share share = share_out(avail, sms, blocks * wpb);
    if (share.lanes == 32 && share.warps == sms * blocks * wpb) return 32;
    unsigned smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    if (threadIdx.x == 0) rank = atomicAdd(&S.sm_rank[smid & (unsigned)(kSmRanks - 1)], 1u);
    __syncthreads();
    const unsigned layer = rank % blocks * wpb + (threadIdx.x >> 5);
    return layer * sms + smid % sms < share.warps ? (int)share.lanes : 0;
}

// Warp-aggregated refill of the warp's idle lanes (all lanes call): the
// first `most` lanes with `need` claim trajectories from the queue.  Returns
// whether the warp is done claiming: the queue had fewer than the lanes
// wanted.
template <int K>
__device__ __noinline__ bool refill(const QueueDev* qp, const SlotsDev* Sp, RareSm* smp, int t, int64_t slot,
                                    bool need, int most) {
    const QueueDev& q = *qp;
    const SlotsDev& S = *Sp;
    RareSm& sm = *smp;
    const unsigned lane = t & 31u;
    const unsigned all = __ballot_sync(kFull, need);
    need = need && __popc(all & ((1u << lane) - 1u)) < most;
    const unsigned m = __ballot_sync(kFull, need);
    if (!m) return false;
    const int leader = __ffs(m) - 1;
    unsigned long long base = 0, got = 0;
    if ((int)lane == leader) {
        // One fetch-and-add per warp.  A claim that runs past the
        // tail gets the part below it; the overshoot of head is
        // clamped back to the tail when more work is published
        // (fp32_publish_kernel, stream-ordered between launches).
        const unsigned long long tail = *(volatile unsigned long long*)q.tail;
        if (*(volatile unsigned long long*)q.head < tail) {
            const unsigned long long want = (unsigned long long)__popc(m);
            const unsigned long long old = atomicAdd(q.head, want);
            if (old < tail) {
                base = old;
                got = min(want, tail - old);
            }
        }
    }
    base = __shfl_sync(kFull, base, leader);
    got = __shfl_sync(kFull, got, leader);
    const unsigned rank = __popc(m & ((1u << lane) - 1u));
    if (need && rank < got) {
        int job;
        const uint32_t traj = (uint32_t)f_resolve(q.range_end, q.range_job, q.range_first, q.nranges,
                                                  (int64_t)(base + rank), &job);
        const JobF* Jn = &q.jobs[job];
        const bool DBL = is_double<K>(*Jn), OVER = is_over<K>(*Jn);
        f_start<K>(Jn, S.ring, S.nslots, S.ring_slots, slot, traj, &sm, t);
        sm.job[t] = job;
        bind_lane(DBL, *Jn, sm, t, traj, Jn->step0);
        if (Jn->nsteps == 0) {
            retire_lane(OVER, *Jn, S.retired, sm, t, 0, sm.xp[t], sm.rv[t], 0);
            idle_lane(sm, t);
        }
    }
    return got < (unsigned long long)__popc(m);
}

// The hot loop: blocks of four steps of the warp's lanes, from their state
// in sm and back, until a lane needs the slow path or `most` blocks ran.
// Returns the blocks run, the last one unfinished for lanes with a step h
// that needs the slow path (P_HALT + h in their P_* word).  A function
// without calls, so that nothing in it is held for one.  M: which special
// steps it takes itself (persistent_run chooses).
template <int K, int M>
__device__ __noinline__ uint32_t run_blocks(const JobF* jobs, RareSm* smp, int t, uint32_t most) {
    constexpr bool DBL = (K & 2) != 0, OVER = (K & 1) != 0;
    RareSm& sm = *smp;
    const int job = sm.job[t];
    float xp = sm.xp[t], rv = sm.rv[t], F = sm.F[t], lo = sm.lo[t], hi = sm.hi[t];
    int left = sm.left[t];
    uint32_t pw = sm.pw[t], j = sm.j[t];
    float c1 = 0.f, c2 = 0.f, c3 = 0.f;
    if (job >= 0) {
        const JobF& J = jobs[job];
        if (OVER) c1 = J.c_drift;
        else { c1 = J.hdt_invM; c2 = J.hdt; c3 = J.expg; }
    }
    // nearly every block has a special step: its steps one by one at once
    const bool walk = M == M_FULL && job >= 0 && jobs[job].walk != 0;
    uint32_t it = 0;
    do {
        // ---- one Philox block, four steps ----
        const uint2 fk = sm.fixk[t];
        const Words w = philox_step(j, sm.fix[t], fk.x);
        const float kn = __uint_as_float(fk.y);
        float nq[4];
        noise_pair(w.w0, w.w1, kn, &nq[0], &nq[1]);
        noise_pair(w.w2, w.w3, kn, &nq[2], &nq[3]);
        // The four steps without a test between them: when the whole warp's
        // positions stayed inside their bands and no countdown ends, they
        // stand; else its lanes take them again one by one, the special ones
        // as quick steps where they can.
        const float x0 = xp, rv0 = rv;
        bool bad = true;
        left -= 4;
        ++it;
        if (M != M_WALK && !(M == M_FULL && walk)) {
            float xs[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                f_move(OVER, xp, rv, F, c1, c2, c3, nq[h]);
                xs[h] = xp;
                if (!OVER) rv = fmaf(F, c1, rv);
            }
            float xmin, xmax;
            range4(xs[0], xs[1], xs[2], xs[3], &xmin, &xmax);
            bad = !(xmin > lo) | !(xmax < hi) | (left <= 0);
        }
        if (__any_sync(kFull, bad)) {
            bool halt = false;
            if (bad) {
                xp = x0;
                rv = rv0;
                left += 4;
                const uint64_t s0 = (uint64_t)sm.jh[t] << 34 | (uint64_t)j << 2;
                float n0 = nq[0], n1 = nq[1], n2 = nq[2];
                const float n3 = nq[3];
#pragma unroll M <= M_WALK ? 4 : 1
                for (int h = 0; h < 4; ++h) {
                    if (halt) continue;
                    f_move(OVER, xp, rv, F, c1, c2, c3, n0);
                    n0 = n1;
                    n1 = n2;
                    n2 = n3;
                    --left;
                    if (!(xp > lo) | !(xp < hi) | (left == 0)) {
                        const uint64_t s = s0 + 1 + h;
                        if (job < 0 ||
                            !(M == M_FULL ? full_quick_step<DBL, OVER>(jobs[job], *sm.slots, sm, t, s, left == 0, xp,
                                                                       rv, lo, hi, F, left, pw)
                                          : quick_step(DBL, M == M_FLIPS, jobs[job], sm, t, s, left == 0, xp, lo, hi, F,
                                                       left, pw))) {
                            halt = true;
                            pw |= P_HALT * (1 + h);
                            sm.nz[0][t] = n0;
                            sm.nz[1][t] = n1;
                            sm.nz[2][t] = n2;
                            continue;
                        }
                    }
                    if (!OVER) rv = fmaf(F, c1, rv);
                }
            }
            if (__any_sync(kFull, halt)) break;
        }
        ++j;
    } while (it < most);
    sm.xp[t] = xp;
    sm.rv[t] = rv;
    sm.F[t] = F;
    sm.lo[t] = lo;
    sm.hi[t] = hi;
    sm.left[t] = left;
    sm.pw[t] = pw;
    sm.j[t] = j;
    return it;
}

}  // namespace

// The persistent loop of one model type for the calling warp: its slots'
// trajectories (and new ones claimed from queue q) for up to quad_budget
// blocks of four steps.  Returns the blocks run; *drained is set when it
// stopped early because every lane of the warp was idle and the queue had
// nothing left for it.  Slot state is loaded at entry and saved at exit.
template <int K, bool kMixed>
__device__ __forceinline__ uint32_t persistent_run(const QueueDev& q, const SlotsDev& S, RareSm& sm,
                                                   uint32_t quad_budget, bool* drained) {
    const int t = threadIdx.x;
    const int64_t slot = (int64_t)blockIdx.x * blockDim.x + t;
    // out-of-line parts of the model type, or of whichever type (kMixed)
    constexpr int B = K & ~K_FULL, C = kMixed ? K_ANY : B;
    sm.slots = &S;   // (all threads the same)
    load_slot<C>(&q, &S, &sm, t, slot);

    // Idle lanes look at the queue from block `look` on: kDry once it had
    // nothing left for this warp.
    constexpr uint32_t kDry = ~0u;
    uint32_t it = 0, look = 0;
    if (!kMixed) {
        const int most = first_claim(*q.avail, S);
        if (most < 32) {
            // leave the items to the warps that take them now; items still
            // there after that (warps that were to take them have
            // trajectories already) are claimed
            if (most == 0 && *(volatile unsigned long long*)q.head < *(volatile unsigned long long*)q.tail)
                __nanosleep(20000);
            // Lanes left out of the warp's share take what is still there
            // once the other warps have had theirs (lanes of theirs may hold
            // another job's trajectories): 64 blocks are 25-45 us.
            if (refill<C>(&q, &S, &sm, t, slot, sm.job[t] < 0 && slot < S.nslots, most ? most : 32)) look = kDry;
            else if (most) look = 64;
        }
    }
    while (it < quad_budget) {
        // lanes become idle in the slow path only
        if (__any_sync(kFull, sm.job[t] < 0)) {
            const bool need = sm.job[t] < 0 && it >= look && slot < S.nslots;
            const bool asked = __any_sync(kFull, need);
            if (asked) {
                if (refill<C>(&q, &S, &sm, t, slot, need, 32)) look = kDry;
            }
            if (__all_sync(kFull, sm.job[t] < 0)) {
                if (!kMixed && it < look && look != kDry) {   // the share has ended already
                    look = it;
                    continue;
                }
                if (look == kDry || !asked) {
                    *drained = true;
                    break;
                }
                ++it;
                continue;
            }
        }
        // The unrolled loop is the faster one for the single barrier with rare
        // flips (2 x 65536 x 48000, flip probability 1e-5 a step: 17.0 ms
        // against 18.6 rolled; 2e-4: 22.0 against 20.1, 1e-3: 40 against 28:
        // with the flips' code it no longer fits the instruction cache), the
        // rolled one for the double barrier (1e-5: 21.2 against 21.7) and for
        // warps of all types on one SM (mixed launches).
        // Kernels of every mode take the highest that a lane's job asks for
        // (JobF::mode).  They are kernels of their own: with that many callees
        // the loop here keeps its values on the stack, 13 % of the time of
        // 100000 trajectories of two barriers at p = 0.01.
        constexpr bool kOnlyRolled = kMixed || (K & 2) != 0;
        const uint32_t blocks = (!kMixed && it < look ? min(quad_budget, look) : quad_budget) - it;
        if (K & K_FULL) {
            const uint32_t mode = __reduce_max_sync(kFull, sm.pw[t] / P_MODE);
            if (mode == M_FULL) it += run_blocks<B, (K & K_FULL) ? M_FULL : M_FLIPS>(q.jobs, &sm, t, blocks);
            else if (!kMixed && mode == M_WALK)
                it += run_blocks<B, (K & K_FULL) && !kMixed ? M_WALK : M_FLIPS>(q.jobs, &sm, t, blocks);
            else if (kOnlyRolled || mode == M_FLIPS) it += run_blocks<B, M_FLIPS>(q.jobs, &sm, t, blocks);
            else it += run_blocks<B, kOnlyRolled ? M_FLIPS : M_RARE>(q.jobs, &sm, t, blocks);
        } else {
            const bool often = !kOnlyRolled && sm.pw[t] / P_MODE >= M_FLIPS;
            if (kOnlyRolled || __any_sync(kFull, often)) it += run_blocks<B, M_FLIPS>(q.jobs, &sm, t, blocks);
            else it += run_blocks<B, kOnlyRolled ? M_FLIPS : M_RARE>(q.jobs, &sm, t, blocks);
        }
        const uint32_t halt = (sm.pw[t] & P_HALTS) / P_HALT;
        if (__any_sync(kFull, halt != 0)) {
            if (halt) {
                sm.pw[t] &= ~P_HALTS;
                slow_steps<C>(q.jobs, &S, &sm, t, slot, (uint64_t)sm.jh[t] << 32 | sm.j[t], (int)halt - 1);
            }
            __syncwarp();
            sm.j[t] += 1;
        }
    }
    save_slot<C>(&q, &S, &sm, t, slot);
    return it;
}

template <int K>
__global__ void __launch_bounds__(256, (K & K_WIDE) ? kWideBlocks : kNarrowBlocks) fp32_persistent_kernel(
    const __grid_constant__ QueueDev q, const __grid_constant__ SlotsDev S, uint32_t quad_budget) {
    extern __shared__ uint4 sm_raw[];
    RareSm& sm = *reinterpret_cast<RareSm*>(sm_raw);
    bool drained = false;
    persistent_run<K, false>(q, S, sm, quad_budget, &drained);
}

// All four model types in one persistent launch (the serving loop's).  A
// warp serves one type at a time -- a warp-uniform switch over the four
// instantiated loops -- with every lane's trajectory from that type's queue;
// when all its lanes are idle and that queue is dry it takes another type
// with unclaimed items, so no type's work waits for another type's launch.
// Its pick is the type its SM serves (sm_type) while that queue has work,
// else the first type with work round robin from the SM's index, which then
// becomes the SM's type: the warps of an SM converge on one type, whose code
// alone then fills the SM's instruction caches (warps of different types on
// one SM measured as stalls on instruction fetch).  The warp's type is kept
// across launches in wtype (-1: none).  A warp ends its launch when the
// budget is spent, no queue has work, or eight type changes in a row found
// nothing to claim (claims raced away by other warps).
template <int KF>
__global__ void __launch_bounds__(256, kNarrowBlocks) fp32_mixed_kernel(const __grid_constant__ MixedDev m,
                                                                               uint32_t quad_budget) {
    extern __shared__ uint4 sm_raw[];
    RareSm& sm = *reinterpret_cast<RareSm*>(sm_raw);
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int type = m.wtype[w];
    uint32_t left = quad_budget;
    int empty_picks = 0;
    while (left > 0) {
        if (type < 0) {
            int pick = -1;
            if ((threadIdx.x & 31) == 0) {
                unsigned smid;
                asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
                volatile int32_t* home = m.sm_type + (smid & (unsigned)(kMixedSmTypes - 1));
                auto has_work = [&](int tt) {
                    const unsigned long long h = *(volatile const unsigned long long*)m.q[tt].head;
                    const unsigned long long tl = *(volatile const unsigned long long*)m.q[tt].tail;
                    return h < tl;
                };
                const int pref = *home;
                if (pref >= 0 && pref < 4 && has_work(pref)) {
                    pick = pref;
                } else {
                    for (int k = 0; k < 4; ++k) {
                        const int tt = (int)((smid + (unsigned)k) & 3u);
                        if (has_work(tt)) {
                            pick = tt;
                            break;
                        }
                    }
                    if (pick >= 0) *home = pick;
                }
            }
            pick = __shfl_sync(kFull, pick, 0);
            if (pick < 0) break;
            type = pick;
        }
        bool drained = false;
        uint32_t used;
        switch (type) {
            case 0: used = persistent_run<KF + 0, true>(m.q[0], m.S, sm, left, &drained); break;
            case 1: used = persistent_run<KF + 1, true>(m.q[1], m.S, sm, left, &drained); break;
            case 2: used = persistent_run<KF + 2, true>(m.q[2], m.S, sm, left, &drained); break;
            default: used = persistent_run<KF + 3, true>(m.q[3], m.S, sm, left, &drained); break;
        }
        left -= (used < left) ? used : left;
        if (drained) {
            type = -1;
            if (used == 0) {
                if (++empty_picks >= 8) break;
            } else {
                empty_picks = 0;
            }
        }
    }
    if ((threadIdx.x & 31) == 0 && w < m.nwarps) m.wtype[w] = type;
}

// Publishes item ranges [.., new_tail): clamps the head (claims may have run
// past the old tail) and moves the tail; one thread, between launches.
__global__ void fp32_publish_kernel(unsigned long long* head, unsigned long long* tail, unsigned long long* avail,
                                    int32_t* nranges, unsigned long long new_tail, int32_t new_nranges) {
    const unsigned long long t = *tail;
    if (*head > t) *head = t;
    *tail = new_tail;
    *avail = new_tail - *head;
    *nranges = new_nranges;
}

int launch_fp32_publish(const QueueDev& q, unsigned long long new_tail, int32_t new_nranges, void* stream) {
    fp32_publish_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(q.head, q.tail, q.avail, q.nranges, new_tail, new_nranges);
    return (int)cudaGetLastError();
}

using PersistentKernel = void (*)(QueueDev, SlotsDev, uint32_t);
template <int F>
static PersistentKernel persistent_kernel_of(bool dbl, bool over, bool wide) {
    switch ((wide ? 4 : 0) | (dbl ? 2 : 0) | (over ? 1 : 0)) {
        case 0: return fp32_persistent_kernel<F + 0>;
        case 1: return fp32_persistent_kernel<F + 1>;
        case 2: return fp32_persistent_kernel<F + 2>;
        case 3: return fp32_persistent_kernel<F + 3>;
        case 4: return fp32_persistent_kernel<F + K_WIDE + 0>;
        case 5: return fp32_persistent_kernel<F + K_WIDE + 1>;
        case 6: return fp32_persistent_kernel<F + K_WIDE + 2>;
        default: return fp32_persistent_kernel<F + K_WIDE + 3>;
    }
}
static PersistentKernel persistent_kernel(bool dbl, bool over, bool wide, bool full) {
    return full ? persistent_kernel_of<K_FULL>(dbl, over, wide) : persistent_kernel_of<0>(dbl, over, wide);
}

// Resident blocks per SM of either kernel (with all modes or the two common
// ones; the fewer, should they ever differ), 0 on error.
template <class Kernel>
static int resident_blocks(Kernel plain, Kernel full, int block) {
    int least = 0;
    for (Kernel kern : {plain, full}) {
        // The kernel reads little global memory: give shared memory the whole
        // carveout so that the occupancy the grid is sized for is resident.
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                             (int)cudaSharedmemCarveoutMaxShared);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RareSm));
        int n = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, block, sizeof(RareSm));
        if (e != cudaSuccess) return 0;
        least = kern == plain ? n : std::min(least, n);
    }
    return least;
}

int fp32_blocks_per_sm(bool dbl, bool over, bool wide, int block) {
    return resident_blocks(persistent_kernel(dbl, over, wide, false), persistent_kernel(dbl, over, wide, true), block);
}

int fp32_mixed_blocks_per_sm(int block) {
    return resident_blocks(fp32_mixed_kernel<0>, fp32_mixed_kernel<K_FULL>, block);
}

int launch_fp32_mixed(const MixedDev& m, bool full, uint32_t pair_budget, int grid, int block, void* stream) {
    const uint32_t quad_budget = pair_budget > 1 ? pair_budget / 2 : 1;
    if (block != 256 || (int64_t)grid * block > m.S.nslots) return (int)cudaErrorInvalidValue;
    auto* kern = full ? fp32_mixed_kernel<K_FULL> : fp32_mixed_kernel<0>;
    kern<<<grid, block, sizeof(RareSm), (cudaStream_t)stream>>>(m, quad_budget);
    return (int)cudaGetLastError();
}

int launch_fp32_persistent(bool dbl, bool over, bool wide, bool full, const QueueDev& q, const SlotsDev& s,
                           uint32_t pair_budget, int grid, int block, void* stream) {
    const uint32_t quad_budget = pair_budget > 1 ? pair_budget / 2 : 1;   // blocks of four steps
    if (block > kMaxBlock) return (int)cudaErrorInvalidValue;
    persistent_kernel(dbl, over, wide, full)<<<grid, block, sizeof(RareSm), (cudaStream_t)stream>>>(q, s, quad_budget);
    return (int)cudaGetLastError();
}

}  // namespace ldp
