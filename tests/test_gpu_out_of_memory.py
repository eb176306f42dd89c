"""Calls whose device allocations fail, one after the other (the failure is made
on the host): the call reports it, and the next call is the one of a handle
that never ran out.
"""
import numpy as np
import pytest

from phybs_gb300 import _lib as L
from phybs_gb300 import meshes as M
from phybs_gb300.solver import DescentSolver, make_params

pytestmark = pytest.mark.gpu

TEST_FAIL_ALLOC = 1  # pbs_test_hook


@pytest.fixture(scope="module", autouse=True)
def built():
    from phybs_gb300.build import build
    build()


def _reshape(s):
    s.set_chunk_shape(128, 192, 128)
    s.step()


CALLS = {
    "step": lambda s: s.step(),
    "be": lambda s: s.backward_euler_step(),
    "pd": lambda s: s.pd_step(),
    "pbd": lambda s: s.pbd_step(),
    "shape": _reshape,
}


@pytest.mark.parametrize("call", CALLS)
def test_failed_allocation_leaves_the_handle_usable(call):
    m = M.box_mesh(5, 4, 7, edge=0.05, seed=1, young=1e5)
    p = make_params("gpu_reference", h=1 / 30, max_iters=16)
    f = CALLS[call]

    def solver():
        s = DescentSolver(m, params=p)
        if call == "shape":
            s.step()  # (a shape that fails leaves a layout that was in use)
        return s

    ref = solver()
    f(ref)
    f(ref)
    want = ref.positions()
    ref.close()
    failed = 0
    for k in range(1, 40):
        s = solver()
        L.lib().pbs_test_hook(s._h, TEST_FAIL_ALLOC, k)
        try:
            f(s)
        except L.PhybsError as e:
            assert e.code == L.PBS_E_OUT_OF_MEMORY
            failed += 1
            if call == "shape":  # the layout it had still steps
                s.step()
                s.reset()
                s.step()
            f(s)
        else:
            L.lib().pbs_test_hook(s._h, TEST_FAIL_ALLOC, 0)
            s.close()
            break
        f(s)
        assert np.array_equal(s.positions(), want), k
        s.close()
    assert 3 <= failed < 39
