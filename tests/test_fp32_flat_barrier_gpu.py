"""Double barriers without height in state 0, whose flanks' meeting point is
0/0: the FP32 path's force follows the position as the FP64 path's does."""
import os

import numpy as np
import pytest

import langevindynamicsforpcp_b200 as ldp

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "inp")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [0, 1])
def test_force_of_a_barrier_between_nothing_and_a_height(over):
    p = ldp.params_from_inp(os.path.join(GOLDEN, "CuIDB_double__2.0_7.2_m1.0_1.00e-05.inp"), ldp.MODEL_DOUBLE)
    p.overdamped, p.tau, p.timestep, p.random_seed, p.write_restart, p.write_x = over, 0.05, 1e-3, 17, 0, 1
    p.number_of_steps, p.freq_save = 12_000, 10
    for b in range(2):
        p.barrier_heights[b][0], p.barrier_heights[b][1] = 0.0, 3.0
    r = {}
    for precision in (ldp.PREC_FP64_PLAIN, ldp.PREC_FP32_BATCHED):
        with ldp.Context(0) as c, ldp.Job(c, p, lanes=500, precision=precision, job_id=6) as j:
            r[precision] = j.run().results()
    x64, f64, s64 = (r[ldp.PREC_FP64_PLAIN][k] for k in ("frames_x", "frames_f", "frames_state"))
    x32, f32, s32 = (r[ldp.PREC_FP32_BATCHED][k] for k in ("frames_x", "frames_f", "frames_state"))
    assert (f64 != 0).mean() > 0.01 and (f32 != 0).mean() > 0.01
    # the force is a function of cell-local position and state: constant in
    # slices of the cell that no breakpoint (in the 2000 slices, seven at
    # most) falls into
    L = p.periodic_length
    mixed = 0
    for st in (0, 1):
        def by_slice(x, f, s):
            m = s == st
            at = np.floor((x[m] / L - np.rint(x[m] / L) + 0.5) * 2000).astype(int)
            return at, f[m]
        a64, g64 = by_slice(x64, f64, s64)
        a32, g32 = by_slice(x32, f32, s32)
        for i in np.unique(a64):
            u = np.unique(g64[a64 == i])
            v = g32[a32 == i]
            if len(u) > 1:   # a breakpoint inside
                mixed += 1
            elif len(v):
                # the FP32 slopes and, at a slice's ends, positions are rounded
                wrong = np.abs(v - u[0]) > 1e-6 * (1 + abs(u[0]))
                assert wrong.mean() < 0.05, (st, i, u[0], v[wrong][:5])
    assert mixed <= 14
