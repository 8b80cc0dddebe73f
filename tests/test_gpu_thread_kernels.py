"""The one-cell-per-thread kernels that run where the cell groups do not: above
their hand-over counts, and for mechanisms that have no groups."""
import numpy as np
import pytest

from micm_b200 import Solver, micm_bench, synthetic
from micm_b200 import solver as sv
from micm_b200._native import check, lib
from micm_b200.mechanism import padded_cells
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
