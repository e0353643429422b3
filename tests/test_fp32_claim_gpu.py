"""How persistent FP32 launches claim trajectories, where their number is
bounded (a graph over a queue of few warps, a job beside another), and where
they just fill the grid."""
import os

import numpy as np
import pytest

import langevindynamicsforpcp_b200 as ldp
from langevindynamicsforpcp_b200 import _lib as L
from langevindynamicsforpcp_b200 import _tune

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "inp")
pytestmark = pytest.mark.gpu
KEYS = ("counts", "sums", "x_final", "state_final")


def params(steps, freq):
    p = ldp.params_from_inp(os.path.join(GOLDEN, "quick_test__2.0_7.2_m1.0_1.00e-05.inp"))
    p.overdamped, p.tau, p.write_x, p.write_restart, p.random_seed = 1, 1e-2, 0, 0, 21
    p.number_of_steps, p.freq_save = steps, freq
    return p


@pytest.mark.parametrize("block,n", [(32, 4736), (32, 1185), (64, 9472), (160, 23_680)])
def test_graph_of_few_warps_ends_within_its_launches(block, n):
    # Fewer warps (or fewer than the next multiple of four) to an SM than it
    # has schedulers, as many trajectories as lanes and fewer: the graph's
    # number of launches is a bound for slots that never idle beside
    # unclaimed items.  (148 SMs; on others the sizes are other ones.)
    p = params(4000, 3)
    with ldp.Context(0) as c, ldp.Job(c, p, lanes=n, precision=ldp.PREC_FP32_BATCHED, job_id=3) as j:
        alone = j.run().results(frames=False)
    with ldp.Context(0) as c:
        _tune.set_fp32_shape(c, block=block, blocks_per_sm=1, pair_budget=2048)
        with ldp.Job(c, p, lanes=n, precision=ldp.PREC_FP32_BATCHED, job_id=3) as j:
            ldp.submit_batch(c, [j], graph=True)
            got = j.wait().results(frames=False)
    for k in KEYS:
        np.testing.assert_array_equal(got[k], alone[k], err_msg=k)


def test_one_launch_claims_all_beside_another_jobs_trajectories():
    # A first-passage job's 5000 trajectories hold lanes here and there when
    # 105000 more come, nearly as many as the idle lanes: the warps that fill
    # only a share at first take the rest in the same launch, so the job runs
    # in as many launches as it does alone.
    p = params(4000, 3)
    slow = params(4000, 3)
    slow.tau, slow.barrier_heights[0][0], slow.barrier_heights[0][1] = 0.0, 80.0, 80.0   # no passage within the cap

    def job(c):
        return ldp.Job(c, p, lanes=105_000, precision=ldp.PREC_FP32_BATCHED, job_id=3)
    out = []
    for beside in (False, True):
        with ldp.Context(0) as c:
            _tune.set_fp32_shape(c, blocks_per_sm=3, pair_budget=2500)
            other = ldp.Job(c, slow, lanes=5000, precision=ldp.PREC_FP32_BATCHED, job_id=4,
                            mode=ldp.MODE_FIRST_PASSAGE, step_cap=40_000)
            if beside:
                other.submit()   # a launch or two of its eight
            with job(c) as j:
                r = j.submit().wait().results(frames=False)
                out.append((j.timing()["launches"], r))
            if beside:
                assert (other.wait().results(frames=False)["counts"][L.C_STEPS] == 40_000).all()
            other.close()
    assert out[1][0] == out[0][0]
    for k in KEYS:
        np.testing.assert_array_equal(out[1][1][k], out[0][1][k], err_msg=k)


def test_full_grids_and_one_trajectory_more():
    # As many trajectories as a launch of three blocks to an SM has lanes (one
    # trajectory each, launched alone), as one of four has, and one more than
    # each: the last one then waits in the queue, or makes the launch a wider
    # one.  All are prefixes of a run on one block to an SM, where nearly all
    # trajectories wait.
    p = params(1050, 1)
    with ldp.Context(0) as c:
        with ldp.Job(c, p, lanes=1, precision=ldp.PREC_FP32_BATCHED, job_id=3) as j:
            j.run()
        three = _tune.get_fp32_shape(c)["grid"] * 256
        assert three % (3 * 256) == 0
        four = three // 3 * 4
        with ldp.Context(0) as c1:
            _tune.set_fp32_shape(c1, blocks_per_sm=1)
            with ldp.Job(c1, p, lanes=four + 1, precision=ldp.PREC_FP32_BATCHED, job_id=3) as j:
                whole = j.run().results(frames=False)
        for n in (three - 1, three, three + 1, four, four + 1):
            with ldp.Job(c, p, lanes=n, precision=ldp.PREC_FP32_BATCHED, job_id=3) as j:
                got = j.run().results(frames=False)
            for k in KEYS:
                np.testing.assert_array_equal(got[k], whole[k][..., :n], err_msg=f"{n} {k}")
