"""The one-cell-per-thread kernels that run where the cell groups do not: above
their hand-over counts, and for mechanisms that have no groups."""
import numpy as np
import pytest

from micm_b200 import Solver, micm_bench, synthetic
from micm_b200 import solver as sv
from micm_b200._native import check, lib
from micm_b200.mechanism import padded_cells
from gpu_helpers import download_cols, make_state
from gpu_helpers import make_state

pytestmark = pytest.mark.gpu


# 9 and 60 species: a thread's eight entries and the rest of one more
@pytest.mark.parametrize("name,n,L", [("chapman", 1, 1), ("chapman", 257, 3), ("c60", 1, 128), ("c60", 1000, 32)])
def test_alpha_minus_jacobian(cuda_device, name, n, L):
    """alpha on the diagonal of every real cell, nothing anywhere else."""
    mech = micm_bench.mechanism("chapman") if name == "chapman" else synthetic.CONFIGS["c60_adjoint"]["mech"]()
    solver = Solver(mech, 3, vector_length=L)
    st = solver.get_state(n)
    nnz, npad = solver.compiled.info["jacobian_nnz"], padded_cells(n, L)
    j = np.random.default_rng(1).normal(size=npad * nnz)
    st.upload(sv.BUF_JACOBIAN, j)
    check(lib().micmb_alpha_minus_jacobian(solver.handle, st.handle, 0.25))
    expected = j.reshape(-1, nnz, L).copy()
    diagonal = solver.compiled.rows == solver.compiled.cols
    real = (np.arange(npad) < n).reshape(-1, 1, L)
    expected += np.where(real & diagonal[None, :, None], 0.25, 0.0)
    np.testing.assert_array_equal(st.download(sv.BUF_JACOBIAN, npad * nnz), expected.ravel())


def _inputs(n, equal=False):
    few = micm_bench.inputs("chapman", 1000, seed=4)
    pick = np.zeros(n, np.int64) if equal else np.arange(n) % 1000
    return {k: np.ascontiguousarray(v[pick]) for k, v in few.items()}


# Chapman on a GPU of 148 SMs: 44,400 cells are the last for which every stage runs on
# cell groups, 94,720 Backward Euler; 160,000 are one set of 151,552 threads and a part
# of the next; all of 310,000 run one cell per thread
@pytest.mark.parametrize("n", [44400, 44401, 160000, 310000])
def test_single_stages_on_both_sides_of_the_hand_over(cuda_device, n):
    mech = micm_bench.mechanism("chapman")
    inp = _inputs(n)
    S = mech.n_species

    def stages(cells):
        solver = Solver(mech, 3, vector_length=128)
        nnz = solver.compiled.info["jacobian_nnz"]
        st = make_state(solver, {k: np.ascontiguousarray(v[cells]) for k, v in inp.items()})
        solver.update_state_parameters(st)
        out = []
        for call, buf, cols in (("add_forcing_terms", sv.BUF_FORCING, S),
                                ("subtract_jacobian_terms", sv.BUF_JACOBIAN, nnz),
                                ("alpha_minus_jacobian", sv.BUF_JACOBIAN, nnz),
                                ("lu_decompose", sv.BUF_JACOBIAN, nnz), ("linear_solve", sv.BUF_FORCING, S)):
            args = (solver.handle, st.handle) + ((0.25,) if call == "alpha_minus_jacobian" else ())
            check(getattr(lib(), "micmb_" + call)(*args))
            out.append(download_cols(st, buf, cols))
        return out

    for a, b in zip(stages(slice(0, n)), stages(slice(n - 1000, n))):
        np.testing.assert_array_equal(a[n - 1000:], b)


@pytest.mark.parametrize("n", [94720, 94721, 160000, 310000])
@pytest.mark.parametrize("control", ["per_cell", "global"])
def test_backward_euler_on_both_sides_of_the_hand_over(cuda_device, n, control):
    """Globally, a state of equal cells: the step sequence is then each cell's own."""
    mech = micm_bench.mechanism("chapman")
    inp = _inputs(n, equal=control == "global")

    def solve(cells):
        solver = Solver(mech, 3, vector_length=128)
        st = make_state(solver, {k: np.ascontiguousarray(v[cells]) for k, v in inp.items()})
        solver.update_state_parameters(st)
        res = solver.solve_backward_euler(1000.0, st, step_control=control, per_cell=True)
        st.sync_outputs_to_host()
        return st.concentrations(), res

    (y, r), (y_few, r_few) = solve(slice(0, n)), solve(slice(n - 1000, n))
    np.testing.assert_array_equal(y[n - 1000:], y_few)
    np.testing.assert_array_equal(r.per_cell_status[n - 1000:], r_few.per_cell_status)
    np.testing.assert_array_equal(r.per_cell_accepted[n - 1000:], r_few.per_cell_accepted)
    if control == "global":
        assert {k: r.stats[k] for k in r.stats if k != "cells_not_converged"} == \
            {k: r_few.stats[k] for k in r_few.stats if k != "cells_not_converged"}


@pytest.mark.parametrize("n", [222000, 222001, 310000])
def test_fused_on_both_sides_of_the_hand_over(cuda_device, n):
    mech = micm_bench.mechanism("chapman")
    inp = _inputs(n)

    def solve(cells, variant):
        solver = Solver(mech, 3, vector_length=128)
        solver.set_fused_config(variant=variant, lu_in_shared=0)
        st = make_state(solver, {k: np.ascontiguousarray(v[cells]) for k, v in inp.items()})
        solver.update_state_parameters(st)
        solver.solve(micm_bench.DT, st, method="fused", step_control="per_cell")
        st.sync_outputs_to_host()
        return st.concentrations()

    y, y_few = solve(slice(0, n), 2), solve(slice(n - 1000, n), 0)
    np.testing.assert_array_equal(y[n - 1000:], y_few)


# MICMB_BLOCKED_SCHEDULES=1: no cell groups; the same sums one cell per thread
@pytest.mark.parametrize("name,n,L", [("c60_adjoint", 1201, 32), ("c210", 299, 128)])
def test_stages_and_backward_euler_equal_the_cell_groups(cuda_device, monkeypatch, name, n, L):
    """Also of cells that are not finite, statuses and counters included."""
    mech = synthetic.CONFIGS[name]["mech"]()
    inp = synthetic.cell_inputs(mech, n, 6, t_range=(200.0, 310.0), night_fraction=0.5)
    inp["concentrations"][[0, 7, n - 1], 3] = np.nan, np.inf, -1.0e-9
    got = []
    for blocked in (True, False):
        if blocked:
            monkeypatch.setenv("MICMB_BLOCKED_SCHEDULES", "1")
        else:
            monkeypatch.delenv("MICMB_BLOCKED_SCHEDULES", raising=False)
        solver = Solver(mech, 4, vector_length=L)
        S, nnz = mech.n_species, solver.compiled.info["jacobian_nnz"]
        st = make_state(solver, inp)
        solver.update_state_parameters(st)
        out = []
        for call, buf, cols in (("add_forcing_terms", sv.BUF_FORCING, S),
                                ("subtract_jacobian_terms", sv.BUF_JACOBIAN, nnz),
                                ("alpha_minus_jacobian", sv.BUF_JACOBIAN, nnz),
                                ("lu_decompose", sv.BUF_JACOBIAN, nnz), ("linear_solve", sv.BUF_FORCING, S)):
            args = (solver.handle, st.handle) + ((0.25,) if call == "alpha_minus_jacobian" else ())
            check(getattr(lib(), "micmb_" + call)(*args))
            out.append(download_cols(st, buf, cols))
        for control in ("per_cell", "global"):
            st.sync_inputs_to_device()
            res = solver.solve_backward_euler(600.0, st, step_control=control, per_cell=True)
            st.sync_outputs_to_host()
            out += [st.concentrations(), res.per_cell_status, res.per_cell_accepted, np.array(list(res.stats.values()))]
        got.append(out)
    for a, b in zip(*got):
        np.testing.assert_array_equal(b, a)
