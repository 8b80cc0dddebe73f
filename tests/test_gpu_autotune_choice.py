"""What the tuner tries, and which states its choice is kept for."""
import re

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


def test_choices_of_other_counts_and_builds_are_not_taken(cuda_device, tmp_path):
    """A choice cached by a state on either side of the hand-over between cell groups
    and one cell per thread serves that side; entries without the version tag (variant
    0 was another kernel) serve none."""
    cache = tmp_path / "tune.txt"
    _tuned(100, str(cache))
    small = cache.read_text().splitlines()
    assert len(small) == 1
    key = small[0].split()[0]
    # as an earlier build would have written it
    cache.write_text(":".join(key.split(":")[:4]) + " 6 0 0 4 0\n")
    _, _, chosen = _tuned(100, str(cache))
    assert chosen["cells_per_cta"] != 6 and len(cache.read_text().splitlines()) == 2
    # a choice for few cells that no large state would make
    cache.write_text(key + " 0 1 1 0 1\n")
    _, _, chosen = _tuned(100, str(cache))
    assert (chosen["variant"], chosen["ctas_per_sm"]) == (1, 1)
    _, _, chosen = _tuned(400000, str(cache))
    assert (chosen["variant"], chosen["ctas_per_sm"]) != (1, 1)
    assert len(cache.read_text().splitlines()) == 2
