"""The cell-group kernels' work lists, run on the host for one cell: bit for bit
the serial schedules, every element in range, no two item lanes on one element
without a synchronisation between them -- for every block shape, on mechanisms
from three species to 600, with long sums, empty rows and repeated reactants."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

from micm_b200 import micm_bench, synthetic
from micm_b200._abi import DescHolder, MechanismDesc
from micm_b200.mechanism import Mechanism, arrhenius

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "micm_b200", "csrc")
pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")


def repeated_reactants():
    m = Mechanism(species=["A", "B", "C", "D"], reactions=[], name="repeated")
    m.add(arrhenius(A=1.0), [0, 0], [(1, 2.0), (1, 0.5)])
    m.add(arrhenius(A=2.0), [1, 1, 1], [(0, 1.0), (2, 1.0)])
    m.add(arrhenius(A=3.0), [2], [(2, 1.0)])
    m.add(arrhenius(A=4.0), [], [(3, 1.0)])
    return m


MECHS = {"readme": synthetic.readme_mechanism, "repeated": repeated_reactants,
         "chapman": lambda: micm_bench.mechanism("chapman"), "ts1": lambda: micm_bench.mechanism("ts1"),
         "c60": synthetic.CONFIGS["c60_adjoint"]["mech"], "c210": synthetic.CONFIGS["c210"]["mech"],
         "c600": synthetic.CONFIGS["c600"]["mech"]}


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("group") / "group_lists.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-o", so,
                    os.path.join(ROOT, "tests", "cpp", "group_lists.cpp"), os.path.join(CSRC, "group.cpp"),
                    os.path.join(CSRC, "mechanism.cpp")], check=True)
    f = C.CDLL(so).check_group_lists
    f.restype, f.argtypes = C.c_int64, [C.POINTER(MechanismDesc)] + 3 * [C.c_int32]
    return f


@pytest.mark.parametrize("name", sorted(MECHS))
@pytest.mark.parametrize("G,W", [(1, 1), (1, 8), (2, 4), (4, 2), (8, 8), (16, 4), (32, 1), (32, 8)])
def test_work_lists_equal_the_serial_schedules(check, name, G, W):
    desc = DescHolder(MECHS[name]().flat())
    assert check(C.byref(desc.desc), G, W, 0) == 0


# the adjoint's backward sweep: transposed factors, contributions of 2 to 6 stages
@pytest.mark.parametrize("name", sorted(MECHS))
@pytest.mark.parametrize("G,W,stages", [(1, 8, 3), (4, 2, 6), (8, 8, 4), (32, 1, 2)])
def test_backward_sweep_work_lists(check, name, G, W, stages):
    desc = DescHolder(MECHS[name]().flat())
    assert check(C.byref(desc.desc), G, W, stages) == 0
