"""The FP32 hot loop's quick steps (frames, flank crossings, crossings back
and forth over a cell edge) and its per-trajectory Philox constants.

A launch of one block of four steps ends every pair of cells and reloads
every constant at its end, and a job with WRITEX saves its frames in the
general step: both give the results of the long launches bit for bit.  Past
2^34 steps the block index's high word changes: the displacement follows the
noise drawn with numpy."""
import os
import struct

import numpy as np
import pytest

import langevindynamicsforpcp_b200 as ldp
from langevindynamicsforpcp_b200 import _tune, serve

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "inp")
pytestmark = pytest.mark.gpu


def params(kind, steps, **kw):
    if kind.startswith("double"):
        p = ldp.params_from_inp(os.path.join(GOLDEN, "CuIDB_double__2.0_7.2_m1.0_1.00e-05.inp"), ldp.MODEL_DOUBLE)
        p.barrier_heights[0][0], p.barrier_heights[0][1] = 1.2, 0.5
        p.barrier_heights[1][0], p.barrier_heights[1][1] = 1.5, 0.5
    else:
        p = ldp.params_from_inp(os.path.join(GOLDEN, "quick_test__2.0_7.2_m1.0_1.00e-05.inp"))
        p.barrier_heights[0][0], p.barrier_heights[0][1] = 1.5, 0.5
    p.overdamped = int(kind.endswith("over"))
    p.number_of_steps, p.freq_save, p.tau, p.random_seed, p.write_restart, p.write_x = steps, 7, 1e-2, 99, 0, 0
    for k, v in kw.items():
        setattr(p, k, v)
    return p


def run(p, lanes, budget=0):
    with ldp.Context(0) as c:
        if budget:
            _tune.set_fp32_shape(c, pair_budget=budget)
        with ldp.Job(c, p, lanes=lanes, precision=ldp.PREC_FP32_BATCHED, job_id=3) as j:
            return j.run().results()


@pytest.mark.parametrize("kind", ["single_over", "single_under", "double_over", "double_under"])
def test_quick_steps_equal_general_ones(kind):
    whole = run(params(kind, 9001), 333)
    for other in (run(params(kind, 9001), 333, budget=2), run(params(kind, 9001, write_x=1), 333)):
        for k in whole:
            np.testing.assert_array_equal(other[k], whole[k], err_msg=k)
    # the start is a cell edge: its crossings are among the steps
    assert (np.diff(np.sign(whole["frames_x"][1:] - whole["frames_x"][0]), axis=0) != 0).any()


def philox(a, g, k0, k1):
    u32, s32 = np.uint64(0xFFFFFFFF), np.uint64(32)
    c0, c1, c2, c3 = a & u32, a >> s32, np.full(a.shape, g, np.uint64), np.zeros(a.shape, np.uint64)
    for _ in range(10):
        p0, p1 = c0 * np.uint64(0xD2511F53), c2 * np.uint64(0xCD9E8D57)
        c0, c1, c2, c3 = (p1 >> s32) ^ c1 ^ np.uint64(k0), p1 & u32, (p0 >> s32) ^ c3 ^ np.uint64(k1), p0 & u32
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c1, c2, c3


def test_block_index_past_32_bits(tmp_path):
    # A saved state with its step count (and frame interval and frames)
    # rewritten: free diffusion from 2^23 steps before step 2^34 to 2^23
    # after it.  Rounding of the FP32 position: three roundings a step of at
    # most 2^-23 (|xp| < 4), random, over 2^24 steps: below 2e-3 (5 sigma).
    # A block drawn with the wrong high word would move it by the noise of
    # 2^23 steps, about 13.
    n, freq, before, more = 3, 1 << 24, (1 << 34) - (1 << 23), 1 << 24
    free = dict(tau=0.0, fpt=0, tpt=0, fptcg=0, waiting_time=0, timestep=1e-5)

    def p_of(steps, prev, fs):
        p = params("single_over", steps, freq_save=fs, number_of_previous_steps=prev, **free)
        p.barrier_heights[0][0] = p.barrier_heights[0][1] = 0.0
        return p
    src, dst = str(tmp_path / "a.state"), str(tmp_path / "b.state")
    with ldp.Context(0) as c:
        with ldp.Job(c, p_of(24_000, 0, 20), lanes=n, precision=ldp.PREC_FP32_BATCHED, job_id=3) as j:
            j.keep_state().run().save_state(src)
            x0 = j.results()["x_final"]
        b = bytearray(open(src, "rb").read())
        nframe = before // freq + 1
        struct.pack_into("<qQQ", b, 12 + 56, nframe, before, freq)
        at = 12
        at += _header_bytes(b)
        for _ in range(12):   # the arrays before the frames
            at += 8 + struct.unpack_from("<Q", b, at)[0]
        size = struct.unpack_from("<Q", b, at)[0]
        cut = nframe * n * 8
        open(dst, "wb").write(b[:at] + struct.pack("<Q", cut) + b[at + 8:at + 8 + cut] + b[at + 8 + size:])
        with ldp.Job(c, p_of(more, before, freq), lanes=n, precision=ldp.PREC_FP32_BATCHED, job_id=3) as j:
            j.load_state(dst)
            x1 = j.run().results()["x_final"]
    sig = np.sqrt(1e-5 * 0.5)
    for g in range(n):
        total = 0.0
        for lo in range(before // 4, (before + more) // 4, 1 << 20):
            w = philox(np.arange(lo, lo + (1 << 20), dtype=np.uint64), g, 99, 3)
            for a, c in ((w[0], w[1]), (w[2], w[3])):
                r = np.sqrt(-2.0 * np.log((a.astype(np.float64) + 1.0) * 2.0 ** -32))
                t = 2.0 * np.pi * (c.astype(np.float64) * 2.0 ** -32)
                total += float((r * (np.cos(t) + np.sin(t))).sum())
        # each step's noise is added twice; the first and last, once, and the
        # FP32 uniforms' 23 bits are below the noise's rounding
        assert abs(x1[g] - x0[g] - 2.0 * sig * total) < 0.05


def _header_bytes(b):
    """Size of the header: up to the first array's byte count, which is that
    of [LDP_NCOUNT = 30][3] 64-bit counts."""
    at = b.index(struct.pack("<Q", 30 * 3 * 8), 12)
    return at - 12


def test_every_job_size_is_claimed():
    # How a launch shares out few items: fewer than schedulers, one more than
    # a warp to each, partly filled ones, one more than all lanes; alone, and
    # published while another job's trajectories hold part of the lanes.
    p = params("single_over", 1050, freq_save=1)
    keys = ("counts", "sums", "x_final", "state_final")
    with ldp.Context(0) as c:
        def job(n, job_id=3):
            return ldp.Job(c, p, lanes=n, precision=ldp.PREC_FP32_BATCHED, job_id=job_id)
        with job(113_665) as j:
            whole = j.run().results(frames=False)
        for n in (1, 593, 18_945, 40_001, 113_664):
            with job(5_000, 4) as a, job(n) as b:
                a.submit()
                r = b.submit().wait().results(frames=False)
                for k in keys:
                    np.testing.assert_array_equal(r[k], whole[k][..., :n], err_msg=f"{n} {k}")
                a.wait()


@pytest.mark.parametrize("graph", [False, True])
def test_launches_of_four_blocks_to_an_sm(graph):
    """Jobs that outgrow three resident blocks to an SM together get launches
    of four: the same results as three blocks', also when trajectories are in
    the slots already, and the queue is back at three afterwards."""
    def outcome(blocks):
        with ldp.Context(0) as c:
            _tune.set_fp32_shape(c, blocks_per_sm=blocks, pair_budget=2500)
            jobs = [ldp.Job(c, params("single_over", 24_000, freq_save=20, tau=1e-3), lanes=n,
                            precision=ldp.PREC_FP32_BATCHED, job_id=i) for i, n in enumerate((lanes, 2000, 40, 9))]
            if graph:
                ldp.submit_batch(c, jobs[:3], graph=True)
            else:
                for j in jobs[:3]:
                    j.submit()
            for j in jobs[:3]:
                j.wait()
            jobs[3].run()
            out = [j.results(frames=False) for j in jobs]
            for j in jobs:
                j.close()
            return out, _tune.get_fp32_shape(c)["grid"]

    lanes = 113_000                  # with 2000 more, past 3 x 256 x 148
    three, grid = outcome(3)
    assert lanes < grid * 256 < lanes + 2000
    for a, b in zip(three, outcome(0)[0]):
        for k in a:
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("kind", ["single_over", "single_under", "double_over", "double_under"])
@pytest.mark.parametrize("tau", [1e-3, 1.0])
def test_saved_forces_after_quick_steps_to_the_bit(kind, tau):
    # The force of a frame after a crossing taken as a quick step is that of
    # the general step, the sign of its zero included: the double barrier's
    # is negative where there is no flank.
    whole = run(params(kind, 9001, write_x=1, tau=tau, freq_save=5), 333)
    short = run(params(kind, 9001, write_x=1, tau=tau, freq_save=5), 333, budget=2)
    series = [k for k in whole if k.startswith("frames")]
    assert len(series) == 7
    for k in series:
        np.testing.assert_array_equal(whole[k].view(np.int64), short[k].view(np.int64), err_msg=k)
    f = whole["frames_f"]
    assert (f == 0).any() and (np.signbit(f[f == 0]) == kind.startswith("double")).all()


@pytest.mark.parametrize("kind", ["single_over", "single_under", "double_over", "double_under"])
def test_pairs_of_barriers_that_never_flip(kind):
    # TAU 0: crossings back and forth over a cell edge are quick steps too.
    whole = run(params(kind, 9001, tau=0.0), 333)
    for other in (run(params(kind, 9001, tau=0.0), 333, budget=2), run(params(kind, 9001, tau=0.0, write_x=1), 333)):
        for k in whole:
            np.testing.assert_array_equal(other[k], whole[k], err_msg=k)
    assert (np.diff(np.sign(whole["frames_x"][1:] - whole["frames_x"][0]), axis=0) != 0).any()


FULL = [  # kind, parameters: what makes lanes take every quick step in the loop, or walk
    ("single_over", dict(tau=1e-5)), ("double_over", dict(tau=1e-5)),              # flips at p = 0.5
    ("single_over", dict(tau=4e-4)), ("double_over", dict(tau=4e-4)),              # and 0.2
    ("single_under", dict(tau=1e-5, write_x=1)), ("double_under", dict(tau=2e-3, write_x=1)),
    ("single_over", dict(tau=1.0, write_x=1)), ("double_over", dict(tau=0.0, write_x=1)),
    ("single_over", dict(tau=1e-2, freq_save=1)), ("double_over", dict(tau=1.0, freq_save=3)),   # frames
    ("single_under", dict(tau=1.0, freq_save=1)), ("double_under", dict(tau=1.0, freq_save=4)),
    ("single_under", dict(tau=1e-3, freq_save=2)),                                 # flips at frame steps
    ("single_over", dict(tau=1e-3, flank=1.0)), ("single_under", dict(tau=1e-5, flank=1.2)),   # no flat band
    ("single_over", dict(tau=1e-5, eq=0, eq_constant=8.0)), ("double_over", dict(tau=1e-5, timestep=1e-3)),
]


@pytest.mark.parametrize("kind,kw", FULL)
def test_quick_steps_of_every_kind_equal_general_ones(kind, kw):
    # Launches of one block of steps end every pair of cells; the job alone,
    # in one launch with a job of rare special steps (the same kernel, lanes
    # of both jobs in a warp), and in the serving kernel give the same bits.
    kw = dict(kw)
    steps = 1201 * kw.get("freq_save", 7)
    p = params(kind, steps, **{k: v for k, v in kw.items() if k != "flank"})
    if "flank" in kw:
        p.barrier_half_width[0] = kw["flank"] * p.periodic_length / 2
    whole = run(p, 333)
    assert len([k for k in whole if k.startswith("frames")]) == (7 if p.write_x else 1)
    short = run(p, 333, budget=2)
    rare = params(kind, 1201 * 7, tau=1.0)
    with ldp.Context(0) as c:
        jobs = [ldp.Job(c, q, lanes=n, precision=ldp.PREC_FP32_BATCHED, job_id=i)
                for q, n, i in ((rare, 100, 8), (p, 333, 3), (rare, 50, 9))]
        ldp.submit_batch(c, jobs)
        mixed = jobs[1].wait().results()
        for j in jobs:
            j.close()
    served = {}
    with ldp.Context(0) as c, serve.Server(c) as srv:
        work = [(rare, 64, {}), (rare, 65, {}), (rare, 66, {}), (p, 333, {})]   # job ids 0 to 3
        serve.run_stream(srv, work, np.zeros(len(work)), timeout_s=60,
                         on_done=lambda i, j: served.__setitem__(i, j.results(frames=False)))
    for other in (short, mixed, served[3]):
        assert len(other) >= 7
        for k in other:
            a, b = other[k], whole[k]
            if a.dtype == np.float64:
                a, b = a.view(np.int64), b.view(np.int64)
            np.testing.assert_array_equal(a, b, err_msg=k)
