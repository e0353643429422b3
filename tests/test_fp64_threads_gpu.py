"""FP64 jobs of different sizes submitted by two host threads at once, each
with its own context: both run the same kernel, one with a few kilobytes of
shared memory a block and one with more than a hundred, and each gets the
results of the job alone."""
import os
import threading

import numpy as np
import pytest

import langevindynamicsforpcp_b200 as ldp

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "inp")
pytestmark = pytest.mark.gpu


def test_two_threads_launch_one_kernel_with_other_shared_memory():
    p = ldp.params_from_inp(os.path.join(GOLDEN, "quick_test__2.0_7.2_m1.0_1.00e-05.inp"))
    p.overdamped, p.tau, p.write_x, p.write_restart, p.random_seed = 0, 1.0, 0, 0, 5
    p.number_of_steps, p.freq_save = 1100, 1
    keys = ("counts", "sums", "x_final")

    def run(c, n, times):
        out = []
        for _ in range(times):
            with ldp.Job(c, p, lanes=n, job_id=2, steps_per_launch=8) as j:   # 138 launches
                r = j.run().results(frames=False)
                out.append({k: r[k] for k in keys})
        return out

    sizes = (1, 5003)
    alone = {}
    for n in sizes:
        with ldp.Context(0) as c:
            alone[n] = run(c, n, 1)[0]
    got, failed, start = {}, [], threading.Barrier(len(sizes))

    def work(n):
        try:
            with ldp.Context(0) as c:
                start.wait(60)
                got[n] = run(c, n, 40)
        except Exception as e:   # a refused launch, reported by the main thread
            failed.append((n, e))

    threads = [threading.Thread(target=work, args=(n,)) for n in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for n in sizes:
        for r in got[n]:
            for k in keys:
                np.testing.assert_array_equal(r[k], alone[n][k], err_msg=f"{n} {k}")


@pytest.mark.parametrize("precision", [ldp.PREC_FP64_PLAIN, ldp.PREC_FP32_BATCHED])
def test_two_threads_launch_displacements_of_other_lengths(precision):
    # The mean-square displacements' kernels hold trajectories of the job's
    # frame count in shared memory: 1201 frames (94 KB a block in FP64, 5 KB
    # a block for a batch's FP32 jobs) and 7001 (56 and 28 KB).
    p = ldp.params_from_inp(os.path.join(GOLDEN, "quick_test__2.0_7.2_m1.0_1.00e-05.inp"))
    p.tau, p.freq_save, p.write_x, p.write_restart, p.random_seed = 1.0, 1, 0, 0, 5

    def run(c, steps, njobs):
        p2 = type(p).from_buffer_copy(p)
        p2.number_of_steps = steps
        jobs = [ldp.Job(c, p2, lanes=3, job_id=2, precision=precision) for _ in range(njobs)]
        try:
            ldp.submit_batch(c, jobs)
            return [j.wait().msd() for j in jobs]
        finally:
            for j in jobs:
                j.close()

    steps = (1200, 7000)
    alone = {}
    for m in steps:
        with ldp.Context(0) as c:
            alone[m] = run(c, m, 1)[0]
    got, failed, start = {m: [] for m in steps}, [], threading.Barrier(len(steps))

    def work(m):
        try:
            with ldp.Context(0) as c:
                start.wait(60)
                for _ in range(15):
                    got[m] += run(c, m, 48)
        except Exception as e:   # a refused launch, reported by the main thread
            failed.append((m, e))

    threads = [threading.Thread(target=work, args=(m,)) for m in steps]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for m in steps:
        for lags, msd in got[m]:
            np.testing.assert_array_equal(lags, alone[m][0])
            np.testing.assert_array_equal(msd, alone[m][1])
