"""Job creation's check of device memory sees what others hold at that moment:
memory that another library of the process took a moment ago counts, and so
does its release."""
import os

import pytest

import langevindynamicsforpcp_b200 as ldp
from langevindynamicsforpcp_b200 import _lib as L

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "inp")
pytestmark = pytest.mark.gpu


def test_creation_counts_memory_taken_since_the_last_job():
    import torch
    p = ldp.params_from_inp(os.path.join(GOLDEN, "quick_test__2.0_7.2_m1.0_1.00e-05.inp"))
    p.number_of_steps, p.freq_save, p.write_x, p.write_restart, p.random_seed = 12_000, 1, 0, 0, 5
    torch.cuda.set_device(0)
    torch.cuda.init()
    with ldp.Context(0) as c:
        with ldp.Job(c, p, lanes=100_000) as j:   # created, never submitted
            need = j.info.device_bytes
        assert need > 9 << 30
        ldp.Job(c, p, lanes=8).close()
        free = torch.cuda.mem_get_info(0)[0]
        held = torch.empty(free - need // 2, dtype=torch.uint8, device="cuda")   # half of the need is left
        try:
            with pytest.raises(L.LdpError) as e:
                ldp.Job(c, p, lanes=100_000)
            assert e.value.status == 2
            ldp.Job(c, p, lanes=8).close()   # a small one still fits
        finally:
            del held
            torch.cuda.empty_cache()
        ldp.Job(c, p, lanes=100_000).close()
