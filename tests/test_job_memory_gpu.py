"""Job creation's check of device memory sees what others hold at that moment:
memory that another library of the process took a moment ago counts, and so
does its release; memory that the process's own earlier jobs freed is there
for a new one.  In processes of their own: the pool that jobs take their
memory from keeps what the process's jobs freed."""
import multiprocessing as mp
import os

import pytest

import langevindynamicsforpcp_b200 as ldp
from langevindynamicsforpcp_b200 import _lib as L
from langevindynamicsforpcp_b200 import _tune

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "inp")
pytestmark = pytest.mark.gpu


def params(steps):
    p = ldp.params_from_inp(os.path.join(GOLDEN, "quick_test__2.0_7.2_m1.0_1.00e-05.inp"))
    p.number_of_steps, p.freq_save, p.write_x, p.write_restart, p.random_seed = steps, 1, 0, 0, 5
    return p


def take(left):
    """All device memory but `left` bytes, as a torch tensor."""
    import torch
    torch.cuda.set_device(0)
    return torch.empty(torch.cuda.mem_get_info(0)[0] - left, dtype=torch.uint8, device="cuda")


def taken_since_the_last_job(precision):
    import torch
    p = params(12_000)
    with ldp.Context(0) as c:
        if precision == ldp.PREC_FP32_BATCHED:
            ldp.Job(c, p, precision=precision).run().close()   # the queue's memory is there
        with ldp.Job(c, p, lanes=100_000, precision=precision) as j:   # created, never submitted
            need = j.info.device_bytes
        assert need > 9 << 30
        ldp.Job(c, p, lanes=8, precision=precision).close()
        held = take(need // 2)
        with pytest.raises(L.LdpError) as e:
            ldp.Job(c, p, lanes=100_000, precision=precision)
        assert e.value.status == 2
        ldp.Job(c, p, lanes=8, precision=precision).close()   # a small one still fits
        del held
        torch.cuda.empty_cache()
        ldp.Job(c, p, lanes=100_000, precision=precision).close()


def freed_by_an_earlier_job(precision):
    import numpy as np
    p = params(1200)

    def run(c):
        with ldp.Job(c, p, lanes=60_000, precision=precision, job_id=4) as j:
            need = j.info.device_bytes
            r = j.run().results(frames=False)
        return need, r
    with ldp.Context(0) as c:
        need, before = run(c)
        held = take((256 << 20) + need // 2)   # the device alone would not hold it
        after = run(c)[1]
        del held
    for k in ("counts", "sums", "x_final"):
        np.testing.assert_array_equal(after[k], before[k], err_msg=k)


def no_room_for_the_slots_of_wide_launches(precision):
    # 16384 ring entries a slot: the slots of three blocks to an SM take 30 GB,
    # those of four 40 GB, and 36 GB are left.
    import numpy as np
    p = params(1200)
    out = []
    for ring in (0, 1 << 14):
        with ldp.Context(0) as c:
            held = None
            if ring:
                _tune.set_fp32_shape(c, ring_slots=ring)
                held = take(36 << 30)
            with ldp.Job(c, p, lanes=300, precision=precision, job_id=4) as j:
                out.append(j.run().results(frames=False))
            del held
    for k in ("counts", "sums", "x_final"):
        np.testing.assert_array_equal(out[1][k], out[0][k], err_msg=k)


@pytest.mark.parametrize("precision", [ldp.PREC_FP64_PLAIN, ldp.PREC_FP32_BATCHED])
@pytest.mark.parametrize("what", [taken_since_the_last_job, freed_by_an_earlier_job])
def test_creation_counts_memory_as_it_is(what, precision):
    in_a_process(what, precision)


def test_slots_that_fit_are_used():
    in_a_process(no_room_for_the_slots_of_wide_launches, ldp.PREC_FP32_BATCHED)


def in_a_process(what, precision):
    c = mp.get_context("spawn").Process(target=what, args=(precision,))
    c.start()
    c.join(120)
    assert c.exitcode == 0
