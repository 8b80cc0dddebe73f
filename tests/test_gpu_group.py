"""The cell-group kernels (working sets in shared memory, several warps and
cells per block) against the one-cell-per-thread kernel, which runs the same
sums in the same order: bit for bit, over the block shapes that the cell count
and the mechanism's size select (one cell per block up to a lane per cell),
ragged last groups, vector lengths that split a block's cells, every tableau,
and cells whose state is not finite."""
import numpy as np
import pytest

from micm_b200 import Solver, micm_bench, synthetic
from micm_b200 import solver as sv
from micm_b200._native import check, lib
from micm_b200.mechanism import Mechanism, arrhenius
from gpu_helpers import download_cols, make_state, upload_cols

pytestmark = pytest.mark.gpu

CASES = {  # mechanism, inputs(n), dt
    "readme": (synthetic.readme_mechanism,
               lambda m, n: synthetic.cell_inputs(m, n, 3, readme_foo=(1.0, 30.0)), 500.0),
    "chapman": (lambda: micm_bench.mechanism("chapman"), lambda m, n: micm_bench.inputs("chapman", n, seed=4), 30.0),
    "c60": (synthetic.CONFIGS["c60_adjoint"]["mech"],
            lambda m, n: synthetic.cell_inputs(m, n, 5, t_range=(200.0, 310.0), night_fraction=0.5), 600.0),
    "c210": (synthetic.CONFIGS["c210"]["mech"],
             lambda m, n: synthetic.cell_inputs(m, n, 6, t_range=(200.0, 310.0), night_fraction=0.5), 60.0),
}


def _solve(solver, inp, dt, method, control):
    st = make_state(solver, inp)
    solver.update_state_parameters(st)
    res = solver.solve(dt, st, method=method, step_control=control, per_cell=True)
    st.sync_outputs_to_host()
    return st.concentrations(), res


# 1: one cell; 2 and 149: fewer cells than two per SM; 299, 1201 and 5000: groups
# of 2, 4-8 and (tiny mechanisms) 32 cells, the last one ragged
@pytest.mark.parametrize("name,n,L,stages", [
    ("readme", 1, 1, 2), ("readme", 10007, 32, 3), ("chapman", 149, 100, 3), ("chapman", 5000, 8, 60),
    ("c60", 1, 128, 4), ("c60", 299, 7, 4), ("c60", 1201, 32, 3), ("c60", 5000, 100, 40),
    ("c210", 2, 1, 4), ("c210", 299, 3, 60), ("c210", 1201, 128, 2)])
def test_group_kernels_equal_thread_kernel(cuda_device, name, n, L, stages):
    make, inputs, dt = CASES[name]
    mech = make()
    inp = inputs(mech, n)
    ref = Solver(mech, stages, vector_length=L)
    ref.set_fused_config(variant=2, lu_in_shared=0, ctas_per_sm=5)
    y_ref, r_ref = _solve(ref, inp, dt, "fused", "per_cell")
    for method in ("fused", "plain"):
        y, r = _solve(Solver(mech, stages, vector_length=L), inp, dt, method, "per_cell")
        np.testing.assert_array_equal(y, y_ref)
        np.testing.assert_array_equal(r.per_cell_status, r_ref.per_cell_status)
        np.testing.assert_array_equal(r.per_cell_accepted, r_ref.per_cell_accepted)
        assert r.stats == r_ref.stats


@pytest.mark.parametrize("bad", [np.nan, np.inf, -1.0e-9])
def test_cells_that_are_not_finite(cuda_device, bad):
    """A NaN, infinite or negative value stays in its own cell."""
    make, inputs, dt = CASES["c60"]
    mech, n = make(), 700
    inp = inputs(mech, n)
    inp["concentrations"][[0, 5, 333, 699], 7] = bad
    ref = Solver(mech, 4, vector_length=32)
    ref.set_fused_config(variant=2, lu_in_shared=0, ctas_per_sm=5)
    y_ref, r_ref = _solve(ref, inp, dt, "fused", "per_cell")
    y, r = _solve(Solver(mech, 4, vector_length=32), inp, dt, "fused", "per_cell")
    np.testing.assert_array_equal(y, y_ref)
    np.testing.assert_array_equal(r.per_cell_status, r_ref.per_cell_status)
    assert r.stats == r_ref.stats


def test_one_cell_global_equals_per_cell(cuda_device):
    """With one cell the single step size is the cell's own."""
    make, inputs, dt = CASES["c210"]
    mech = make()
    inp = inputs(mech, 1)
    y_p, r_p = _solve(Solver(mech, 4, vector_length=8), inp, dt, "plain", "per_cell")
    y_g, r_g = _solve(Solver(mech, 4, vector_length=8), inp, dt, "plain", "global")
    np.testing.assert_array_equal(y_g, y_p)
    assert r_g.stats["accepted"] == r_p.stats["accepted"] and r_g.stats["rejected"] == r_p.stats["rejected"]


@pytest.mark.parametrize("name,n", [("readme", 10007), ("c60", 1201), ("c210", 299)])
@pytest.mark.parametrize("control", ["per_cell", "global"])
def test_backward_euler_does_not_depend_on_the_block_shape(cuda_device, name, n, control):
    """Cells solved together (several per block) equal the same cells in states
    small enough for one per block; globally, a state of equal cells."""
    make, inputs, dt = CASES[name]
    mech = make()
    inp = inputs(mech, n)
    if control == "global":  # the step sequence is then each cell's own
        inp = {k: np.repeat(v[:1], n, axis=0) for k, v in inp.items()}

    def solve(cells):
        solver = Solver(mech, 3, vector_length=32)
        st = make_state(solver, {k: np.ascontiguousarray(v[cells]) for k, v in inp.items()})
        solver.update_state_parameters(st)
        res = solver.solve_backward_euler(dt, st, step_control=control, per_cell=True)
        st.sync_outputs_to_host()
        return st.concentrations(), res

    y, r = solve(slice(0, n))
    for cells in (slice(0, 1), slice(n - 100, n)):
        y_few, r_few = solve(cells)
        np.testing.assert_array_equal(y[cells], y_few)
        np.testing.assert_array_equal(r.per_cell_status[cells], r_few.per_cell_status)
        np.testing.assert_array_equal(r.per_cell_accepted[cells], r_few.per_cell_accepted)


@pytest.mark.parametrize("name,n,L", [("readme", 10007, 32), ("c60", 149, 7), ("c60", 1201, 32), ("c210", 299, 128)])
def test_single_stages_do_not_depend_on_the_block_shape(cuda_device, name, n, L):
    """The single-stage entry points on many cells (several per block) equal the
    same cells in a state small enough for one per block, signed zeros of the
    accumulated-into arrays included; values outside the real cells stay."""
    make, inputs, _ = CASES[name]
    mech = make()
    inp = inputs(mech, n)
    S = mech.n_species
    rng = np.random.default_rng(9)
    f0 = rng.choice([0.0, -0.0, 1.0e-7], size=(n, S))

    def stages(cells):
        solver = Solver(mech, 3, vector_length=L)
        nnz = solver.compiled.info["jacobian_nnz"]
        j0 = np.random.default_rng(10).choice([0.0, -0.0, 2.0e-3], size=(n, nnz))[cells]
        st = make_state(solver, {k: np.ascontiguousarray(v[cells]) for k, v in inp.items()})
        solver.update_state_parameters(st)
        upload_cols(st, sv.BUF_FORCING, f0[cells])
        upload_cols(st, sv.BUF_JACOBIAN, j0)
        out = []
        check(lib().micmb_add_forcing_terms(solver.handle, st.handle))
        out.append(download_cols(st, sv.BUF_FORCING, S))
        check(lib().micmb_subtract_jacobian_terms(solver.handle, st.handle))
        out.append(download_cols(st, sv.BUF_JACOBIAN, nnz))
        check(lib().micmb_alpha_minus_jacobian(solver.handle, st.handle, 0.25))
        out.append(download_cols(st, sv.BUF_JACOBIAN, nnz))
        check(lib().micmb_lu_decompose(solver.handle, st.handle))
        out.append(download_cols(st, sv.BUF_JACOBIAN, nnz))
        check(lib().micmb_linear_solve(solver.handle, st.handle))
        out.append(download_cols(st, sv.BUF_FORCING, S))
        return out

    many = stages(slice(0, n))
    few = stages(slice(n - 100, n))
    for a, b in zip(many, few):
        np.testing.assert_array_equal(a[n - 100:].view(np.int64), np.ascontiguousarray(b).view(np.int64))


def _reactant_orders():
    """One to three reactants, repeated ones among them, and a source."""
    m = Mechanism(species=["A", "B", "C", "D"], reactions=[], name="orders")
    m.add(arrhenius(A=0.3), [0, 0], [(1, 2.0), (1, 0.5)])
    m.add(arrhenius(A=0.2), [1, 1, 2], [(0, 1.0), (2, 1.0)])
    m.add(arrhenius(A=0.1), [2, 3, 0], [(2, 1.0)])
    m.add(arrhenius(A=0.01), [], [(3, 1.0)])
    m.add(arrhenius(A=0.05), [3], [(0, 1.0)])
    return m


CASES["orders"] = (_reactant_orders, lambda m, n: synthetic.cell_inputs(m, n, 8, log10_conc=(-1.0, 0.3)), 30.0)


# The backward sweep on cell groups needs the stored stages; a limit that has room
# for the states alone makes the one-cell-per-thread kernel recompute them.
@pytest.mark.parametrize("name,n,L,stages", [("readme", 5003, 32, 2), ("chapman", 149, 100, 3), ("orders", 1, 1, 4),
                                             ("orders", 777, 8, 60), ("c60", 299, 7, 40), ("c60", 1201, 32, 3),
                                             ("c210", 149, 128, 4)])
def test_backward_sweep_equals_thread_kernel(cuda_device, name, n, L, stages):
    make, inputs, dt = CASES[name]
    mech = make()
    inp = inputs(mech, n)
    ybar = np.random.default_rng(2).normal(size=(n, mech.n_species))
    got = []
    for recompute in (True, False):
        solver = Solver(mech, stages, vector_length=L)
        if recompute:
            solver.set_adjoint_memory_limit(-(-n // L) * L * 400 * (mech.n_species + 1) * 8 + 100)
        st = make_state(solver, inp)
        solver.update_state_parameters(st)
        g0, gk, res = solver.solve_adjoint(dt, st, ybar, max_checkpoints=400)
        assert res.converged
        got.append((g0.copy(), gk.copy()))
    np.testing.assert_array_equal(got[1][0], got[0][0])
    np.testing.assert_array_equal(got[1][1], got[0][1])
