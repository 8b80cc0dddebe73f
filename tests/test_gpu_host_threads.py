"""Solvers of different mechanisms used from several host threads at once: the
kernels are the process's, the solvers' sizes are their own."""
import threading

import numpy as np
import pytest

from micm_b200 import Solver, synthetic
from gpu_helpers import make_state

pytestmark = pytest.mark.gpu


# 1,300 cells: eight cells per block of either mechanism, so that both threads launch
# the same kernels, with 217 KB and 40 KB of shared memory per block
@pytest.mark.parametrize("what", ["global", "per_cell", "fused", "euler"])
def test_two_mechanisms_on_two_threads_equal_one_after_the_other(cuda_device, what):
    n, rounds = 1300, 12
    jobs = []
    for make, stages, dt, seed in ((synthetic.CONFIGS["c210"]["mech"], 4, 60.0, 6),
                                   (synthetic.CONFIGS["c60_adjoint"]["mech"], 4, 60.0, 5)):
        mech = make()
        solver = Solver(mech, stages, vector_length=32)
        inp = synthetic.cell_inputs(mech, n, seed, t_range=(200.0, 310.0), night_fraction=0.5)
        jobs.append((solver, inp, dt))

    def once(solver, inp, dt):
        st = make_state(solver, inp)
        solver.update_state_parameters(st)
        if what == "euler":
            res = solver.solve_backward_euler(dt, st, step_control="global", per_cell=True)
        else:
            method, control = ("fused", "per_cell") if what == "fused" else ("plain", what)
            res = solver.solve(dt, st, method=method, step_control=control, per_cell=True)
        st.sync_outputs_to_host()
        return st.concentrations(), res.stats

    expected = [once(*job) for job in jobs]
    errors = []
    start = threading.Barrier(2, timeout=60)

    def run(q):
        try:
            import torch
            torch.cuda.set_device(0)
            start.wait()
            for _ in range(rounds):
                y, stats = once(*jobs[q])
                np.testing.assert_array_equal(y, expected[q][0])
                assert stats == expected[q][1]
        except Exception as e:  # reported below
            errors.append(e)

    threads = [threading.Thread(target=run, args=(q,)) for q in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=300)
    assert not errors, errors


def test_adjoints_on_two_threads_leave_the_solver_as_it_is(cuda_device):
    """The direct kernel keeps no stage vectors, so the adjoint's forward pass runs
    another configuration than the solver's: that stays what it is, also seen from
    other threads."""
    cfg = synthetic.CONFIGS["c60_adjoint"]
    mech = cfg["mech"]()
    solver = Solver(mech, cfg["stages"], vector_length=32)
    solver.set_fused_config(variant=1)
    before = solver.get_fused_config()
    inp = synthetic.cell_inputs(mech, 64, 5)
    ybar = np.ones((64, mech.n_species))
    got, seen, errors = [], [], []
    start = threading.Barrier(2, timeout=60)

    def run():
        try:
            import torch
            torch.cuda.set_device(0)
            start.wait()
            for _ in range(10):
                st = make_state(solver, inp)
                solver.update_state_parameters(st)
                g0, gk, _ = solver.solve_adjoint(600.0, st, ybar, max_checkpoints=300)
                got.append((g0, gk))
                seen.append(solver.get_fused_config())
        except Exception as e:  # reported below
            errors.append(e)

    threads = [threading.Thread(target=run) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=300)
    assert not errors, errors
    assert solver.get_fused_config() == before
    assert all(c == before for c in seen)
    for g0, gk in got[1:]:
        np.testing.assert_array_equal(g0, got[0][0])
        np.testing.assert_array_equal(gk, got[0][1])
