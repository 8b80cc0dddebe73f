"""The streamed kernel (one cell per warp, program fed by TMA): variant 0 runs it
where the configuration sets one of its parameters."""
import numpy as np
import pytest
import torch

from micm_b200 import Solver, synthetic
from gpu_helpers import make_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config", [dict(ring_slots=4), dict(cells_per_cta=3), dict(ctas_per_sm=1)])
def test_settings_of_the_streamed_kernel_run_it(cuda_device, config):
    """It keeps everything in shared memory here, where the cell groups allocate
    their cells' vectors (eight cells per SM); the results are the cell groups'."""
    cfg = synthetic.CONFIGS["c210"]
    mech = cfg["mech"]()
    n = 2000
    inp = synthetic.cell_inputs(mech, n, 3, t_range=(200.0, 310.0), night_fraction=0.5)
    ref = Solver(mech, cfg["stages"], vector_length=32)
    st = make_state(ref, inp)
    ref.update_state_parameters(st)
    r_ref = ref.solve(60.0, st, method="fused", step_control="per_cell", per_cell=True)
    st.sync_outputs_to_host()
    y_ref = st.concentrations()

    solver = Solver(mech, cfg["stages"], vector_length=32)
    solver.set_fused_config(variant=0, lu_in_shared=1, **config)
    warm = make_state(solver, {k: v[:1] for k, v in inp.items()})  # the kernel is loaded
    solver.update_state_parameters(warm)
    solver.solve(60.0, warm, method="fused", step_control="per_cell")
    st = make_state(solver, inp)
    solver.update_state_parameters(st)
    free = torch.cuda.mem_get_info()[0]
    res = solver.solve(60.0, st, method="fused", step_control="per_cell", per_cell=True)
    used = free - torch.cuda.mem_get_info()[0]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert used < 8 * 8 * sms * (2 + cfg["stages"]) * mech.n_species, used
    st.sync_outputs_to_host()
    np.testing.assert_array_equal(st.concentrations(), y_ref)
    np.testing.assert_array_equal(res.per_cell_accepted, r_ref.per_cell_accepted)
    assert res.stats == r_ref.stats
