"""A captured solve (micmb_solve_graph) between other calls on the same state:
calls that replace a buffer the capture holds, and settings that it was captured
with."""
import ctypes as C

import numpy as np
import pytest

from micm_b200 import Solver, synthetic
from micm_b200._native import check, lib
from gpu_helpers import make_state

pytestmark = pytest.mark.gpu


def _stage(solver, st):
    check(lib().micmb_add_forcing_terms(solver.handle, st.handle))


def _adjoint(solver, st):
    solver.solve_adjoint(10.0, st, np.ones((st.n_cells, st.S)), max_checkpoints=200)


def _euler(solver, st):
    solver.solve_backward_euler(10.0, st, step_control="per_cell")


def _plain(solver, st):
    solver.solve(10.0, st, method="plain", step_control="global")


# variant 2 with ctas_per_sm, and variant 1: working sets that the other calls outgrow
@pytest.mark.parametrize("config", [dict(), dict(variant=2, lu_in_shared=0, ctas_per_sm=5),
                                    dict(variant=1, lu_in_shared=0)])
@pytest.mark.parametrize("between", [_stage, _adjoint, _euler, _plain])
def test_captured_solve_after_other_calls(cuda_device, config, between):
    cfg = synthetic.CONFIGS["c210"]
    mech = cfg["mech"]()
    inputs = synthetic.cell_inputs(mech, 300, 17, **cfg["inputs"])
    outs = []
    for graph in (False, True):
        solver = Solver(mech, cfg["stages"], vector_length=32)
        solver.set_fused_config(**config)
        st = make_state(solver, inputs)

        def steps(n):
            if graph:
                solver.solve_graph(30.0, st, n)
            else:
                for _ in range(n):
                    solver.update_state_parameters(st)
                    solver.solve(30.0, st, method="fused", step_control="per_cell")
        steps(2)
        between(solver, st)
        steps(2)
        st.sync_outputs_to_host()
        outs.append(st.concentrations())
    np.testing.assert_array_equal(outs[1], outs[0])


@pytest.mark.parametrize("what", ["tolerance", "params"])
def test_captured_solve_follows_changed_settings(cuda_device, what):
    """The relative tolerance and the solver's parameters are part of a capture."""
    cfg = synthetic.CONFIGS["c60_adjoint"]
    mech = cfg["mech"]()
    inputs = synthetic.cell_inputs(mech, 64, 18)
    outs = []
    for graph in (False, True):
        solver = Solver(mech, cfg["stages"], vector_length=32)
        st = make_state(solver, inputs)

        def steps(n):
            if graph:
                solver.solve_graph(600.0, st, n)
            else:
                for _ in range(n):
                    solver.update_state_parameters(st)
                    solver.solve(600.0, st, method="fused", step_control="per_cell")
        steps(2)
        if what == "tolerance":
            check(lib().micmb_state_set_relative_tolerance(st.handle, 1.0e-4))
        else:
            solver.params.safety_factor = 0.7
            check(lib().micmb_solver_set_params(solver.handle, C.byref(solver.params)))
        steps(2)
        st.sync_outputs_to_host()
        outs.append(st.concentrations())
    np.testing.assert_array_equal(outs[1], outs[0])
