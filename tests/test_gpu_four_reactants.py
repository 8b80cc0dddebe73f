"""A reaction with four reactants: no cell groups, so every entry point runs the
kernels that large counts run (one cell per thread, per stage) or that only such
mechanisms run by default (streamed), against the C restatement of micm's
algorithm, bit for bit, with the restatement's rate constants."""
import numpy as np
import pytest

import oracle
from micm_b200 import Solver, synthetic
from micm_b200 import solver as sv
from micm_b200.mechanism import arrhenius
from gpu_helpers import make_state, upload_cols

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not oracle.restatement_available(), reason="oracle not built")]
FIELDS = oracle.STATS_FIELDS[:7]


def _case(n):
    m = synthetic.synthetic_mechanism(60, 120, seed=601)
    m.add(arrhenius(A=1.0e18), [0, 1, 2, 3], [(4, 1.0), (1, 0.5)])
    m.add(arrhenius(A=1.0e17), [5, 5, 6, 7], [(8, 2.0)])
    return m, synthetic.cell_inputs(m, n, 21, t_range=(200.0, 310.0), night_fraction=0.5, log10_conc=(-10.0, -6.0))


def _state(m, inp, stages, k, L, **config):
    solver = Solver(m, stages, vector_length=L)
    if config:
        solver.set_fused_config(**config)
    st = make_state(solver, inp)
    upload_cols(st, sv.BUF_RATE_CONSTANTS, k)
    return solver, st


def _values(st):
    st.sync_outputs_to_host()
    return st.concentrations()


@pytest.mark.parametrize("method,config", [
    ("plain", {}), ("fused", {}), ("fused", dict(ring_slots=2, cells_per_cta=3)),
    ("fused", dict(lu_in_shared=0)), ("fused", dict(variant=1)), ("fused", dict(variant=2)),
    ("fused", dict(variant=2, ctas_per_sm=5)), ("fused", dict(variant=2, ctas_per_sm=8))])
@pytest.mark.parametrize("stages", [3, 4])
def test_per_cell(cuda_device, method, config, stages):
    m, inp = _case(333)
    R = oracle.Restatement(m, stages, correctly_rounded=True)
    k = R._k(inp)
    y_ref, st_ref = R.solve_per_cell(inp, 600.0, k=k)
    solver, st = _state(m, inp, stages, k, 32, **config)
    res = solver.solve(600.0, st, method=method, step_control="per_cell", per_cell=True)
    np.testing.assert_array_equal(_values(st), y_ref)
    np.testing.assert_array_equal(res.per_cell_status, st_ref[:, 7])
    np.testing.assert_array_equal(res.per_cell_accepted, st_ref[:, 3])
    for q, key in enumerate(FIELDS):
        assert res.stats[key] == st_ref[:, q].sum(), key


@pytest.mark.parametrize("n,L", [(1, 1), (257, 100), (600, 32)])
def test_global(cuda_device, n, L):
    m, inp = _case(n)
    R = oracle.Restatement(m, 4, correctly_rounded=True)
    k = R._k(inp)
    y_ref, st_ref = R.solve_global(inp, 600.0, k=k)
    solver, st = _state(m, inp, 4, k, L)
    res = solver.solve(600.0, st, method="plain", step_control="global")
    np.testing.assert_array_equal(_values(st), y_ref)
    for q, key in enumerate(FIELDS):
        assert res.stats[key] == st_ref[q], key
    assert res.state == st_ref[7]


@pytest.mark.parametrize("control", ["per_cell", "global"])
def test_backward_euler(cuda_device, control):
    m, inp = _case(333)
    R = oracle.Restatement(m, 3)
    k = R._k(inp)
    y_ref, st_ref = getattr(R, "backward_euler_" + control)(inp, 600.0, k=k)
    solver, st = _state(m, inp, 3, k, 32)
    res = solver.solve_backward_euler(600.0, st, step_control=control, per_cell=True)
    np.testing.assert_array_equal(_values(st), y_ref)
    rows = st_ref.reshape(-1, st_ref.shape[-1])
    np.testing.assert_array_equal(res.per_cell_status, np.broadcast_to(rows[:, 7], 333))
    np.testing.assert_array_equal(res.per_cell_accepted, np.broadcast_to(rows[:, 3], 333))
    for q, key in enumerate(FIELDS):
        assert res.stats[key] == rows[:, q].sum(), key


@pytest.mark.parametrize("variant", [0, 2])
def test_adjoint_with_stored_and_recomputed_stages(cuda_device, variant):
    """Forward values as the solve's, gradients as the CPU adjoint's, and the same
    from stored and recomputed stages."""
    m, inp = _case(149)
    ybar = np.random.default_rng(2).normal(size=(149, m.n_species))
    R = oracle.Restatement(m, 4, correctly_rounded=True)
    k = R._k(inp)
    y_ref, _ = R.solve_per_cell(inp, 600.0, k=k)
    cols = R.species_columns
    _, g_ref, gk_ref = R.adjoint_per_cell(inp, 600.0, ybar[:, cols], k=k)
    got = []
    for recompute in (False, True):
        solver, st = _state(m, inp, 4, k, 32, variant=variant, lu_in_shared=0 if variant == 2 else 1)
        if recompute:  # room for the states alone
            solver.set_adjoint_memory_limit(160 * 400 * (m.n_species + 1) * 8 + 100)
        g0, gk, res = solver.solve_adjoint(600.0, st, ybar, max_checkpoints=400)
        assert res.converged
        np.testing.assert_array_equal(_values(st), y_ref)
        got.append((g0, gk))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
    # the bounds of test_gpu_adjoint.py
    g = got[0][0][:, cols]
    scale = np.abs(g_ref).max(axis=1, keepdims=True)
    assert np.all(np.abs(g - g_ref) <= 1e-6 * scale + 1e-300)
    gk_sum = gk_ref.sum(axis=0)
    np.testing.assert_allclose(got[0][1], gk_sum, rtol=1e-8, atol=1e-9 * np.abs(gk_sum).max())
