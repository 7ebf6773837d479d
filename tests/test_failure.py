"""Failure handling without a GPU fault: a device wait that can never be
satisfied runs out of its bounded time, the kernel returns an error status
that the host reports (VLBA_ERR_TIMEOUT), and the context keeps working.
Host-side failures (invalid requests in a batch or a served stream) are
covered in test_batch.py and test_server.py."""

from __future__ import annotations

import numpy as np
import pytest

from visloc_ba import BaConfig, RobustKernel, synth
from visloc_ba import _abi


@pytest.mark.gpu
def test_a_wait_on_a_flag_nothing_sets_times_out_and_the_context_survives(solver):
    st, waited = solver.wait_probe(250.0)
    assert st == _abi.ERR_TIMEOUT
    assert 200.0 <= waited <= 2000.0
    p = synth.ring_problem(10, 300, seed=5)
    st, res = solver.optimize(p.copy(), BaConfig(max_iterations=5,
                                                 robust_kernel=RobustKernel.huber(1.0)))
    assert st == _abi.OK and res.final_cost < res.initial_cost


@pytest.mark.gpu
def test_a_team_without_one_of_its_blocks_times_out_and_solves_the_same_again(solver):
    """The other blocks of the team publish words under the next numbers and
    give up: a later solve must not take those for its own."""
    p = synth.ring_problem(200, 8000, seed=3)
    cfg = BaConfig(max_iterations=4, robust_kernel=RobustKernel.huber(1.0), max_pcg_iterations=60,
                   pcg_relative_tolerance=1e-6)
    assert solver.upload(p, cfg) == _abi.OK
    st, first = solver.solve_uploaded()
    assert st == _abi.OK
    before, after, again = p.copy(), p.copy(), p.copy()
    assert solver.download(before) == _abi.OK
    for _ in range(2):
        st, waited = solver.wait_probe(50.0)
        assert st == _abi.ERR_TIMEOUT and waited <= 2000.0
        assert "gave up" in solver.last_error()
    assert solver.download(after) == _abi.OK  # the state is left as it was
    st, second = solver.solve_uploaded()
    assert st == _abi.OK and second.final_cost == first.final_cost
    assert [i.pcg_iterations for i in second.iterations] == \
        [i.pcg_iterations for i in first.iterations]
    assert solver.download(again) == _abi.OK
    for q in (after, again):
        assert np.array_equal(before.pose_q, q.pose_q)
        assert np.array_equal(before.landmarks, q.landmarks)


def test_probe_limits_are_checked():
    lib = _abi.load_solver_library()
    import ctypes as C

    assert lib.visloc_ba_cuda_wait_probe(None, 10.0, C.byref(C.c_double())) == \
        _abi.ERR_INVALID_ARGUMENT
