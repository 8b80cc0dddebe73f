"""A job with one step size for all cells whose ranks run different forms of the
plain solve (cell groups, per-stage kernels: each rank chooses by its own number
of cells).  All ranks have to make the same number of exchanges, also where the
solve ends with the last attempt of a batch (8, then 16, 32 and 64 more)."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from micm_b200 import Solver, synthetic
from micm_b200._native import check, lib
from micm_b200.solver import RosenbrockSolverParameters
from gpu_helpers import make_state

pytestmark = pytest.mark.gpu
SHARDS = [40, 61]


class _DeviceArray:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (int(ptr), False),
                                         "version": 3, "strides": None}


def _dev(ptr, n):
    return torch.as_tensor(_DeviceArray(ptr, n), device="cuda")


def _solve(monkeypatch, blocked, max_steps):
    """Two ranks on two host threads, the exchange through the host: each rank's
    values and statistics, and its exchanges.  blocked: the ranks that run the
    per-stage kernels (the register-blocked schedules are theirs)."""
    mech = synthetic.synthetic_mechanism(60, 120, seed=601)
    inp = synthetic.cell_inputs(mech, sum(SHARDS), 5)
    states, streams, solvers, start = [], [], [], 0
    for rank, n in enumerate(SHARDS):
        params = RosenbrockSolverParameters.four_stage()
        params.max_number_of_steps = max_steps
        if blocked[rank]:
            monkeypatch.setenv("MICMB_BLOCKED_SCHEDULES", "1")
        else:
            monkeypatch.delenv("MICMB_BLOCKED_SCHEDULES", raising=False)
        solvers.append(Solver(mech, params, vector_length=32))
        states.append(make_state(solvers[rank], {k: v[start:start + n] for k, v in inp.items()}))
        solvers[rank].update_state_parameters(states[rank])
        streams.append(torch.cuda.Stream())
        check(lib().micmb_state_set_stream(states[rank].handle, ctypes.c_void_p(streams[rank].cuda_stream)))
        start += n
    torch.cuda.synchronize()
    barrier = threading.Barrier(2, timeout=10)
    slots, calls, results, errors = [0.0, 0.0], [0, 0], [None, None], []

    def make_exchange(rank):
        def exchange(send, recv, world, stream):
            calls[rank] += 1
            streams[rank].synchronize()
            slots[rank] = float(_dev(send, 1).cpu().item())
            barrier.wait()
            both = torch.tensor(slots, dtype=torch.float64)
            barrier.wait()
            with torch.cuda.stream(torch.cuda.ExternalStream(stream)):
                _dev(recv, 2).copy_(both)
            return 0
        return exchange

    def run(rank):
        try:
            torch.cuda.set_device(0)
            states[rank].set_global_exchange(make_exchange(rank), 2, sum(SHARDS))
            results[rank] = solvers[rank].solve(600.0, states[rank], method="plain", step_control="global")
        except Exception as e:  # reported below
            errors.append(e)
            barrier.abort()

    threads = [threading.Thread(target=run, args=(r,)) for r in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=300)
    assert not errors, (errors, calls)
    y = []
    for st in states:
        st.sync_outputs_to_host()
        y.append(st.concentrations())
    return np.concatenate(y), [(r.state, r.stats) for r in results], calls


# a solve stops after the first accepted step past max_steps: attempt 8 and 24 end a batch
@pytest.mark.parametrize("max_steps", [6, 7, 8, 23, 1000])
def test_ranks_on_different_kernels_make_the_same_exchanges(cuda_device, monkeypatch, max_steps):
    y_ref, r_ref, _ = _solve(monkeypatch, (False, False), max_steps)
    for blocked in ((False, True), (True, False), (True, True)):
        y, r, calls = _solve(monkeypatch, blocked, max_steps)
        assert calls[0] == calls[1]
        np.testing.assert_array_equal(y, y_ref)
        assert r == r_ref
    if max_steps in (7, 23):  # what this test is about
        assert r_ref[0][1]["number_of_steps"] == max_steps + 1
