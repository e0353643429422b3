"""Latency and group mode of FP64 plain jobs against one trajectory per
thread, bit for bit, where the split over warps changes (one trajectory, one
more than SMs, one more than schedulers, one more than eight lanes to each or
to two warps of each, one more than two lanes),
with rare and frequent flips (drawn by the stepping warps, or ahead for every
step), frames at every step, inside blocks and at their ends, and launches
that start anywhere in a block of four steps."""
import os

import numpy as np
import pytest

import langevindynamicsforpcp_b200 as ldp

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "inp")
pytestmark = pytest.mark.gpu


def run(p, n, latency, group, spl):
    with ldp.Context(0) as c:
        c.set_fp64_latency(latency)
        c.set_fp64_group(group)
        with ldp.Job(c, p, lanes=n, job_id=2, steps_per_launch=spl) as j:
            r = j.run().results()
            r["msd_traj"] = j.msd_traj()
    return r


@pytest.mark.parametrize("n,double,over,tau,freq,spl,write_x", [
    (1, 0, 1, 1e-5, 1, 0, 1), (149, 1, 1, 1e-1, 7, 333, 0), (593, 0, 0, 1e-3, 8, 1001, 1), (593, 1, 0, 1e-5, 3, 0, 0),
    (4737, 0, 1, 1e-2, 5, 0, 0), (1300, 0, 1, 0.0, 11, 2050, 0), (593, 1, 1, 1e-5, 3, 1500, 1),
    (1185, 0, 1, 1e-1, 4, 0, 0), (9473, 0, 1, 1e-1, 2, 0, 0)])
def test_modes_equal_one_trajectory_per_thread(n, double, over, tau, freq, spl, write_x):
    name = "CuIDB_double__2.0_7.2_m1.0_1.00e-05.inp" if double else "quick_test__2.0_7.2_m1.0_1.00e-05.inp"
    p = ldp.params_from_inp(os.path.join(GOLDEN, name), ldp.MODEL_DOUBLE if double else ldp.MODEL_SINGLE)
    p.overdamped, p.tau, p.freq_save, p.write_x, p.write_restart, p.random_seed = over, tau, freq, write_x, 0, 77
    p.number_of_steps = 1100 * freq
    p.barrier_heights[0][0], p.barrier_heights[0][1] = 1.5, 0.5
    if double:
        p.barrier_heights[1][0], p.barrier_heights[1][1] = 1.2, 0.5
    thread = run(p, n, 0, 0, spl)
    for latency, group in ((1 << 30, 0), (0, 1 << 30)):
        other = run(p, n, latency, group, spl)
        for k in thread:
            np.testing.assert_array_equal(other[k], thread[k], err_msg=k)
