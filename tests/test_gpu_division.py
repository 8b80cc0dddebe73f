"""The cell groups' division by a known reciprocal (group.cuh, divide_by) against
the divide, bit for bit: a linear solve with a diagonal matrix is one division per
value, and its operands can be uploaded."""
import itertools

import numpy as np
import pytest

from micm_b200 import Solver
from micm_b200 import solver as sv
from micm_b200._native import check, lib
from micm_b200.mechanism import Mechanism, arrhenius
from gpu_helpers import download_cols, upload_cols

pytestmark = pytest.mark.gpu


def _quotients(v, d):
    """v / d by a solve of one-entry rows, three per cell, on the GPU."""
    m = Mechanism(species=["A", "B", "C"], reactions=[], name="decay")
    for i in range(3):
        m.add(arrhenius(A=1.0), [i], [])
    solver = Solver(m, 3, vector_length=32)
    n = -(-len(v) // 3)
    st = solver.get_state(n)

    def cols(a):
        return np.concatenate([a, np.ones(3 * n - len(a))]).reshape(n, 3)
    upload_cols(st, sv.BUF_JACOBIAN, cols(d))
    upload_cols(st, sv.BUF_FORCING, cols(v))
    check(lib().micmb_linear_solve(solver.handle, st.handle))
    return download_cols(st, sv.BUF_FORCING, 3).ravel()[:len(v)]


def _compare(v, d):
    with np.errstate(all="ignore"):
        expected = v / d
    got = np.concatenate([_quotients(v[i:i + 90000], d[i:i + 90000]) for i in range(0, len(v), 90000)])
    number = ~np.isnan(expected)
    np.testing.assert_array_equal(np.isnan(got), ~number)
    np.testing.assert_array_equal(got[number].view(np.int64), expected[number].view(np.int64))


def test_special_values_and_exponent_borders(cuda_device):
    """Zeros, infinities, NaN, subnormals, all-ones significands, and both sides of
    2^-500 and 2^500, where the divide takes over."""
    x = [0.0, np.inf, np.nan, 5e-324, np.finfo(float).tiny, np.nextafter(np.finfo(float).tiny, 0), np.finfo(float).max]
    for e in (-1022, -501, -500, -499, -1, 0, 1, 499, 500, 501, 1023):
        p = 2.0 ** e
        x += [p, np.nextafter(p, 0), np.nextafter(p, np.inf), p * (1.0 + 1.0 / 3.0)]
    x = np.array(x + [-a for a in x])
    pairs = np.array(list(itertools.product(x, x)))
    _compare(np.ascontiguousarray(pairs[:, 0]), np.ascontiguousarray(pairs[:, 1]))


@pytest.mark.parametrize("kind", ["any", "normal", "halfway"])
def test_random_operands(cuda_device, kind):
    """Any bit pattern; operands of the range in use; quotients next to the middle
    of two neighbouring doubles."""
    rng = np.random.default_rng(12)
    n = 500000
    if kind == "any":
        v, d = (rng.integers(0, 1 << 64, n, dtype=np.uint64).view(np.float64) for _ in range(2))
    else:
        d = rng.uniform(1.0, 2.0, n)
        v = rng.uniform(1.0, 2.0, n)
        if kind == "halfway":
            # v = (a 53-bit quotient and a half ulp) d, rounded, and its neighbours
            q = rng.integers(1 << 52, 1 << 53, n)
            dm = (d * 2.0 ** 52).astype(np.int64)
            v = np.array([float((2 * int(a) + 1) * int(b)) for a, b in zip(q, dm)]) * 2.0 ** -106
            v = np.where(rng.integers(0, 3, n) == 0, np.nextafter(v, 0), v)
        scale = rng.integers(-400, 400, (2, n))
        v, d = np.ldexp(v, scale[0]), np.ldexp(d, scale[1])
        v *= rng.choice([-1.0, 1.0], n)
    _compare(v, d)
