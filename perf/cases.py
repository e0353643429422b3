"""Performance cases: the jobs that programs run through this package.

A case is one call sequence of a user's program: a job (or a batch, a graph
or a serving burst of jobs) from host parameters to host results.  The models
are those of the sample inputs (the CuIDB single and double barrier geometry,
the CuOPTz geometry of the scan), the sizes those of the tests, of bench.py
and of the scan, first-passage and serving workloads, or in between.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  parameters (and the handles a program keeps)
    run(state)           one pass through the public entry points
    work(case)           bytes and operations of a pass
    exact(case, seed)    the same results in 64 bits with numpy, where a
                         step-by-step evaluation there is quick enough
"""
import math
import random

import numpy as np

import langevindynamicsforpcp_b200 as ldp
from langevindynamicsforpcp_b200 import serve

# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
INP = """\
OUTPUTBASE perf
OVERDAMPED {over}
X0 {x0!r}
V0 1.0
GAMMA {gamma!r}
KB 1.0
TEMPERATURE 1.0
MASS 1.0
RANDOMIZEV true
PERIODICLENGTH {length!r}
TIMESTEP {dt!r}
NUMBEROFSTEPS {steps}
NUMBEROFPREVIOUSSTEPS 0
NUMBEROFRUNS 1
FREQSAVE {freq}
FREQSTAT 1
DISTRIBUTIONV0 false
DISTRIBUTIONS0 true
TAU {tau!r}
INITIALSTATE 0
RANDOMIZESTATES true
UNIFORMINITALSTATES false
EQ true 1.0
WAITINGTIME {full}
FPT true
TPT true
FPTCG true 2
FPTCG true 3
FPTCG true 10
READRESTART false
WRITERESTART {full}
INPUTRESTART none
OUTPUTRESTART none
WRITEX {full}
NUMBEROFLOGSAMPLES 40
RANDOMSEED {seed}
PRINTTIMER false
"""
SINGLE = "BARRIERHEIGHTS {high!r} {low!r}\nBARRIERHALFWIDTH {half!r}\n"
DOUBLE = ("BARRIERHEIGHTS0 {mid!r} {low!r}\nBARRIERHEIGHTS1 {high!r} {low!r}\nBARRIERHALFWIDTH0 0.70\n"
          "BARRIERHALFWIDTH1 0.65\nBARRIERPOSITION0 -1.42\nBARRIERPOSITION1 -0.56\n")
N_CG = 3


def model(case):
    """The numbers of one parameter set."""
    h = case["low"]
    scan = case.get("geometry") == "CuOPTz"
    return {"over": "true" if case["over"] else "false", "gamma": case.get("gamma", 1.0), "dt": case["dt"],
            "length": 2.1 if scan else 5.8, "x0": -1.05 if scan else -2.9, "half": 0.6 if scan else 0.65,
            "steps": case["steps"], "freq": case["freq"], "tau": case["tau"],
            "full": "true" if case.get("full") else "false", "low": h, "mid": 1.7 * h,
            "high": (2.7 if scan else 3.6) * h}


def params(case, seed):
    v = dict(model(case), seed=int(seed) & 0x7FFFFFFF)
    text = INP.format(**v) + (DOUBLE if case["double"] else SINGLE).format(**v)
    return ldp.params_from_inp_text(text, ldp.MODEL_DOUBLE if case["double"] else ldp.MODEL_SINGLE)


def one(**kw):
    """A single job's case: CuIDB single barrier, overdamped, dt 1e-5, a flip
    rate in the middle of the range, unless told otherwise."""
    c = {"kind": "job", "fp32": False, "double": False, "over": True, "dt": 1e-5, "tau": 1.0, "low": 2.0,
         "full": False, "frames": False}
    c.update(kw)
    return c


def many(**kw):
    """Several jobs; each job's trajectories and parameters come from the seed."""
    c = {"kind": "batch", "dt": 1e-5}
    c.update(kw)
    return c


def listed():
    return [
        # The smallest run the engine takes: one vector of 8 lanes, little
        # more than the 1000 frames a run must have.  Start-up, launches and
        # result reads are all of it.
        one(name="fp64 one vector 1200 steps", trajectories=8, steps=1200, freq=1, dt=1e-4, tau=1e-5, frames=True),
        # The reference's own sample input (4 ranks x 8 lanes, dt 1e-4, a flip
        # at about every second step, every statistic, every series and
        # event list), shortened: few long trajectories.
        one(name="fp64 sample input 32 long", trajectories=32, steps=160000, freq=80, dt=1e-4, tau=1e-5, full=True,
            frames=True),
        # A study of a double-barrier model on one GPU: some hundred
        # trajectories, the sample inputs' time step.
        one(name="fp64 double 900", double=True, trajectories=900, steps=60000, freq=50, dt=1e-4, tau=1e-2),
        # A few thousand underdamped trajectories, an odd number of them.
        one(name="fp64 underdamped 5003", over=False, trajectories=5003, steps=36000, freq=30),
        # A plain FP64 job of the benchmark's width.
        one(name="fp64 large 65536", trajectories=65536, steps=60000, freq=50, tau=0.2),
        # The smallest and an ordinary request of the serving ranges, alone.
        one(name="fp32 small 1024", fp32=True, trajectories=1024, steps=24000, freq=20, over=False),
        one(name="fp32 double 20011", fp32=True, double=True, trajectories=20011, steps=48000, freq=40, tau=0.1),
        # The benchmark's batch: jobs of 65536 trajectories with heights and
        # flip rates of the precision workload.
        many(name="fp32 batch 4 x 65536", jobs=4, fixed=65536, steps=120000, freq=100, mix="precision"),
        # The parameter scan: unequal jobs over both dampings in one graph.
        many(name="fp32 scan graph 16 sets", kind="graph", jobs=16, lo=10.0, hi=15.0, steps=24000, freq=20, mix="scan"),
        # Requests of all four model types served together.
        many(name="fp32 serving burst 20 jobs", kind="serve", jobs=20, lo=10.0, hi=15.0, steps=24000, freq=20,
             mix="serving"),
        # First passages of the double-barrier model: uneven lengths, capped.
        many(name="fp32 first passage 2 x 30000", kind="passage", jobs=2, fixed=30000, cap=100000, mix="passage",
             steps=24000, freq=20),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    k = rng.random()
    if k < 0.65:
        fp32 = rng.random() < 0.45
        c = one(fp32=fp32, double=rng.random() < 0.35, over=rng.random() < 0.7, low=rng.choice([2.0, 3.0, 4.0, 5.0]),
                tau=float("%.4g" % 10 ** rng.uniform(-5 if not fp32 else -2, 2)), dt=rng.choice([1e-5, 1e-5, 1e-4]))
        c["trajectories"] = log_int(rng, 200 if fp32 else 8, 65536)
        frames = rng.randint(1100, 2200)
        most = (8e9 if fp32 else 3.9e9) / c["trajectories"]
        c["freq"] = max(1, min(log_int(rng, 1, 75), int(most / frames)))
        c["steps"] = c["freq"] * frames
        c["frames"] = c["trajectories"] <= 64
        c["full"] = not fp32 and c["trajectories"] <= 64 and rng.random() < 0.5
        return c
    if k < 0.78:
        freq = rng.randint(20, 100)
        return many(jobs=rng.randint(2, 4), fixed=rng.randint(20000, 65536), steps=1200 * freq, freq=freq,
                    mix="precision")
    lo = rng.uniform(9.5, 11.0)
    if k < 0.88:
        return many(kind="graph", jobs=rng.randint(6, 16), lo=lo, hi=lo + rng.uniform(1.0, 4.0), steps=24000, freq=20,
                    mix="scan")
    if k < 0.95:
        return many(kind="serve", jobs=rng.randint(8, 20), lo=lo, hi=lo + rng.uniform(1.0, 4.0), steps=24000, freq=20,
                    mix="serving")
    return many(kind="passage", jobs=rng.randint(1, 3), fixed=rng.randint(8000, 30000), cap=rng.randint(40000, 100000),
                mix="passage", steps=24000, freq=20)


def jobs_of(case, seed):
    """The parameter sets of a batch: (case of one job, trajectories)."""
    rng = random.Random(int(seed) * 7919 + 17)
    out = []
    for i in range(case["jobs"]):
        mix = case["mix"]
        c = one(fp32=True, steps=case["steps"], freq=case["freq"], dt=case["dt"], tau=10 ** rng.uniform(-2, 2),
                low=rng.choice([2.0, 3.0, 4.0, 5.0]))
        if mix == "scan":
            c.update(geometry="CuOPTz", low=rng.choice([3.5, 4.5, 5.5, 6.5]), gamma=10 ** rng.uniform(-1, 1),
                     over=i % 2 == 0)
        elif mix == "serving":
            c.update(double=i % 4 >= 2, over=i % 2 == 1, gamma=10 ** rng.uniform(-1, 1))
        elif mix == "passage":
            c.update(double=True)
        # the trajectory counts are the case's (evenly spread exponents), so
        # that the work of a case does not hang on the seed
        n = case.get("fixed") or int(2 ** (case["lo"] + (case["hi"] - case["lo"]) * ((7 * i) % case["jobs"] + 0.5)
                                           / case["jobs"]))
        c["trajectories"] = n
        out.append(c)
    return out


# ---------------------------------------------------------------------------
# runs
# ---------------------------------------------------------------------------
_ctx = None


def context():
    """The program's context on device 0."""
    global _ctx
    if _ctx is None:
        _ctx = ldp.Context(0)
    return _ctx


class Serving:
    """A running server and its context, closed with the program's last use of it."""

    def __init__(self):
        self.ctx = ldp.Context(0)
        self.server = serve.Server(self.ctx, hbm_budget=6 << 30)

    def __del__(self):
        self.server.close()
        self.ctx.close()


def prepare(case, seed):
    state = {"case": case, "job_id": int(seed) % 1000003}
    if case["kind"] == "job":
        state["params"] = params(case, seed)
        state["ctx"] = context()
        return state
    cases = jobs_of(case, seed)
    state["work"] = [(params(c, seed), c["trajectories"]) for c in cases]
    if case["kind"] == "serve":
        state["serving"] = Serving()
    else:
        state["ctx"] = context()
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "job":
        return run_job(case, state)
    if case["kind"] == "serve":
        return run_serving(state)
    ctx, work, graph = state["ctx"], state["work"], case["kind"] != "batch"
    mode = {}
    if case["kind"] == "passage":
        mode = {"mode": ldp.MODE_FIRST_PASSAGE, "step_cap": case["cap"]}
    jobs = [ldp.Job(ctx, p, lanes=n, precision=ldp.PREC_FP32_BATCHED, job_id=state["job_id"] + i, **mode)
            for i, (p, n) in enumerate(work)]
    ldp.submit_batch(ctx, jobs, graph=graph)
    out = []
    for j in jobs:
        j.wait()
        if case["kind"] == "passage":
            out.append(j.results(frames=False, ticks=False))
        else:
            out.append({"means": j.means(), "msd": j.msd()[1]})
    for j in jobs:
        j.close()
    return out


def run_job(case, state):
    prec = ldp.PREC_FP32_BATCHED if case["fp32"] else ldp.PREC_FP64_PLAIN
    with ldp.Job(state["ctx"], state["params"], lanes=case["trajectories"], precision=prec, job_id=state["job_id"],
                 event_cap=-1 if case["full"] else 0) as job:
        job.run()
        out = job.results(frames=case["frames"])
        out["lags"], out["msd"] = job.msd()
    return out


def run_serving(state):
    server, out, tickets = state["serving"].server, [None] * len(state["work"]), {}
    for i, (p, n) in enumerate(state["work"]):
        tickets[server.submit(p, n, job_id=state["job_id"] + i)] = i
    while tickets:
        server.step()
        for t in server.ended():
            i = tickets.pop(t)
            job = server.job(t)
            out[i] = {"means": job.means(), "msd": job.msd()[1]}
            server.release(t)
    return out


# ---------------------------------------------------------------------------
# work of a pass
# ---------------------------------------------------------------------------
def lag_grid(steps, freq, dt):
    """The mean-square displacement's lags: 40 a decade from one frame to
    the frames past the first thousand."""
    nf, ts = steps // freq + 1, dt * freq
    t, last, lags = math.log10(ts), math.log10(ts * (nf - 1000)), [0]
    while t <= last:
        k = int(math.floor(10 ** t / ts + 0.5))
        if k != lags[-1]:
            lags.append(k)
        t += 1.0 / 40
    return lags


def work_one(c, rows):
    """bytes: the parameters and the results of a job (`rows` numbers of 8
    bytes a trajectory).  flops: 70 operations a particle-step (Philox 20,
    Box-Muller 6, move 3, indices 6, flip 2, force 7, clocks 6, loop 20) and
    3 a term of the mean-square displacement."""
    n, nf = c["trajectories"], c["steps"] // c["freq"] + 1
    lags = lag_grid(c["steps"], c["freq"], c["dt"])
    series = (7 if c["full"] else 1) * nf if c["frames"] else 0
    return {"bytes": 2048 + 8 * n * (rows + series) + 16 * len(lags),
            "flops": 70 * n * c["steps"] + 3 * n * sum(nf - k for k in lags)}


def work(case):
    if case["kind"] == "job":
        return work_one(case, 30 + 24 + 4)     # counts, sums, first and last state
    if case["kind"] == "passage":               # at most: how many reach the cap is not known before
        n = case["jobs"] * case["fixed"]
        return {"bytes": 2048 * case["jobs"] + 8 * n * 58, "flops": 70 * n * case["cap"]}
    each = [work_one(c, 4 + N_CG) for c in jobs_of(case, 0)]   # mean event times
    return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}


# ---------------------------------------------------------------------------
# the same in 64 bits, with numpy
# ---------------------------------------------------------------------------
U32 = np.uint64(0xFFFFFFFF)


def philox(a, g, tag, key0, key1):
    """Philox4x32-10 (Salmon et al., SC'11) of counter (a, g, tag): four
    arrays of 32-bit words (in 64)."""
    a, g = np.broadcast_arrays(np.asarray(a, np.uint64), np.asarray(g, np.uint64))
    s32 = np.uint64(32)
    c0, c1, c2, c3 = a & U32, a >> s32, g & U32, np.full(a.shape, tag, np.uint64)
    k0, k1 = int(key0), int(key1)
    for _ in range(10):
        p0, p1 = c0 * np.uint64(0xD2511F53), c2 * np.uint64(0xCD9E8D57)
        c0, c1, c2, c3 = (p1 >> s32) ^ c1 ^ np.uint64(k0), p1 & U32, (p0 >> s32) ^ c3 ^ np.uint64(k1), p0 & U32
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c1, c2, c3


def gauss(wa, wb):
    r = np.sqrt(-2.0 * np.log((wa.astype(np.float64) + 1.0) * 2.0 ** -32))
    t = 2.0 * np.pi * (wb.astype(np.float64) * 2.0 ** -32)
    return r * np.cos(t), r * np.sin(t)


def schedule(s, hi, lo, ln1m):
    """The step of the next flip: s and a geometric waiting time."""
    u = (((hi << np.uint64(32)) | lo).astype(np.float64) + 1.0) * 2.0 ** -64
    return s + 1.0 + np.floor(np.log(u) / ln1m)


STEP, INIT, CATCHUP, CELL, FLIP = range(5)
CHUNK = 2000    # steps drawn at once (a multiple of 4)


def forces(c):
    """force(cell-local position, state) of a parameter set, and the place
    where the double model's two barriers meet."""
    m = model(c)
    if not c["double"]:
        w, hs = m["half"], np.array([m["high"], m["low"]])

        def force(xp, s):
            return np.where((np.abs(xp) < w) & (xp != 0.0), np.sign(xp) * (hs / w)[s], 0.0)
        return force, 0.0
    b, w, h = (-1.42, -0.56), (0.70, 0.65), np.array([[m["mid"], m["low"]], [m["high"], m["low"]]])
    x1h, x2l, y1, y2 = b[0] + w[0], b[1] - w[1], h[0, 0], h[1, 0]
    d1, d2 = b[1] - x2l, x1h - b[0]
    xc = (x1h * y1 * d1 + x2l * y2 * d2) / (y1 * d1 + y2 * d2)
    yc = (x1h - xc) / d2 * y1
    slopes = [h[0] / w[0], (yc - h[0]) / (xc - b[0]), (h[1] - yc) / (b[1] - xc), -h[1] / w[1]]
    edges = [b[0] - w[0], b[0], xc, b[1], b[1] + w[1]]

    def force(xp, s):
        f = np.zeros(xp.shape)
        for k in range(4):
            f = np.where((xp > edges[k]) & (xp < edges[k + 1]), slopes[k][s], f)
        return -f
    return force, xc


def exact(case, seed):
    """Positions, saved frames and the mean-square displacement of one FP64
    job, step by step.  Counts are whole numbers; the FP32 path rounds each
    step to 32 bits, so a trajectory of it parts from the 64-bit one at the
    first crossing that the rounding decides."""
    if case["kind"] != "job" or case["fp32"]:
        return None
    n, steps, freq, dt = case["trajectories"], case["steps"], case["freq"], case["dt"]
    if steps * (4.5e-5 + 6e-7 * n) > 14.0:
        return None
    m = model(case)
    L, invL, dbl, over, gam = m["length"], 1.0 / m["length"], case["double"], case["over"], m["gamma"]
    k0, k1 = int(seed) & 0x7FFFFFFF, int(seed) % 1000003
    force, xc = forces(case)
    rate = -np.expm1(-2.0 * dt / case["tau"])
    ln1m = np.log1p(-0.5 * rate)
    sig_r, drift = np.sqrt(dt * 0.5 / gam), dt / gam
    sig_v, decay, h = np.sqrt(1.0 - np.exp(-2.0 * gam * dt)), np.exp(-gam * dt), dt * 0.5
    g = np.arange(n, dtype=np.uint64)
    w = philox(0, g, INIT, k0, k1)
    state = np.where(w[0].astype(np.float64) * 2.0 ** -32 <= 0.5, 0, 1)
    zv, zr = gauss(w[1], w[2])
    v0 = zv.copy()
    x, v, prev = np.full(n, m["x0"]), zv, sig_r * zr
    cell = np.rint(x * invL)
    side = np.zeros(n, bool) if not dbl else x - cell * L >= xc
    w = philox(0, g, FLIP, k0, k1)
    nflip = schedule(0.0, w[0], w[1], ln1m)
    f = force(x - cell * L, state)
    table = [{} for _ in range(n)]
    frames = np.empty((steps // freq + 1, n))
    frames[0] = x
    last = steps // freq * freq if freq >= 10 else steps
    for s in range(1, last + 1):
        q = (s - 1) % CHUNK
        if q == 0:
            a = np.arange((s - 1) // 4, (s - 1) // 4 + CHUNK // 4, dtype=np.uint64)[:, None]
            w = philox(a, g[None, :], STEP, k0, k1)
            z = np.stack(gauss(w[0], w[1]) + gauss(w[2], w[3]), axis=1).reshape(CHUNK, n)
            w = philox(np.arange(s, s + CHUNK, dtype=np.uint64)[:, None], g[None, :], FLIP, k0, k1)
            after = schedule(np.arange(s, s + CHUNK, dtype=np.float64)[:, None], w[0], w[1], ln1m)
        if over:
            r = sig_r * z[q]
            x = x + f * drift + r + prev
            prev = r
        else:
            v = v + f * h
            x = x + v * h
            v = decay * v + sig_v * z[q]
            x = x + v * h
        now = np.rint(x * invL)
        xp = x - now * L
        flip = nflip == s
        state = state ^ flip
        nflip = np.where(flip, after[q], nflip)
        new_side = xp >= xc if dbl else side
        moved = new_side != side if dbl else now != cell
        for i in np.flatnonzero(moved):
            old = int(cell[i]) * 2 + int(side[i]) if dbl else int(cell[i])
            key = int(now[i]) * 2 + int(new_side[i]) if dbl else int(now[i])
            table[i][old] = (int(state[i]), float(nflip[i]))
            if key in table[i] and table[i][key][1] > s:
                state[i], nflip[i] = table[i][key]
                continue
            if key in table[i]:
                since, st = table[i][key][1], table[i][key][0] ^ 1
            else:
                c = philox(np.uint64(key & 0xFFFFFFFFFFFFFFFF), g[i], CELL, k0, k1)[0]
                since, st = 0.0, 0 if float(c) * 2.0 ** -32 < 0.5 else 1
            p = 0.5 * -math.expm1(-2.0 * dt / case["tau"] * (s - since))
            c = philox(np.uint64(s), g[i], CATCHUP, k0, k1)
            u = (int(c[0]) << 32) | int(c[1])
            state[i] = st ^ 1 if u < int(math.ldexp(p, 64)) else st
            c = philox(np.uint64(s), g[i], FLIP, k0, k1)
            nflip[i] = schedule(float(s), c[2], c[3], ln1m)
        cell, side = now, new_side
        f = force(xp, state)
        if not over:
            v = v + f * h
        if s % freq == 0:
            frames[s // freq] = x
    lags = lag_grid(steps, freq, dt)
    msd = np.array([np.mean((frames[k:] - frames[:frames.shape[0] - k]) ** 2) for k in lags])
    out = {"x_final": x, "v0": v0, "v_final": v, "msd": msd}
    if case["frames"]:
        out["frames_x"] = frames
    return out
