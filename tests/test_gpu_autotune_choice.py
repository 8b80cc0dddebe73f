"""What the tuner tries, and which states its choice is kept for."""
import re

import numpy as np
import pytest

from micm_b200 import Solver, micm_bench
from gpu_helpers import make_state

pytestmark = pytest.mark.gpu


def _tuned(n, cache=None):
    mech = micm_bench.mechanism("chapman")
    solver = Solver(mech, 3, vector_length=128)
    st = make_state(solver, micm_bench.inputs("chapman", n, seed=4))
    solver.update_state_parameters(st)
    return solver, st, solver.autotune(micm_bench.DT, st, cache)


# at both counts the 32-register thread build is not what ctas_per_sm = 0 runs on the trial's cells
@pytest.mark.parametrize("n", [5000, 310000])
def test_every_thread_build_is_tried_as_itself(cuda_device, monkeypatch, capfd, n):
    monkeypatch.setenv("MICMB_AUTOTUNE_VERBOSE", "1")
    solver, st, chosen = _tuned(n)
    tried = re.findall(r"variant 2 .* ctas_per_sm (\d+): (\d+) cells", capfd.readouterr().err)
    assert {b for b, _ in tried} == {"16", "12", "8", "5"}, tried
    if n > 303104:  # the count of the solver's own cells that 0 leaves to the thread kernel
        assert chosen["variant"] != 2 or chosen["ctas_per_sm"] != 16
    res = solver.solve(micm_bench.DT, st, method="fused", step_control="per_cell")
    assert res.converged
