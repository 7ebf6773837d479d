"""The PCG kernels of reduced systems that stay on the chip at the sizes where
one begins and ends, against the FP64 iteration they restate: the clusters
(at most 16 tile rows, 128 cameras), the teams of blocks (up to 576 densely
coupled cameras), and past them the persistent kernel."""

from __future__ import annotations

import numpy as np
import pytest

from visloc_ba import BaConfig, RobustKernel, synth

pytestmark = pytest.mark.gpu


def system(n, keep, seed):
    """A random SPD block system of n nodes, each pair coupled with
    probability `keep`, its condition number about 50."""
    rng = np.random.default_rng(seed)
    a, b = np.triu_indices(n, 1)
    on = rng.random(len(a)) <= keep
    a, b = a[on], b[on]
    ga, gb = (np.eye(6) + 0.3 * rng.standard_normal((len(a), 6, 6)) for _ in range(2))
    off = -(gb.transpose(0, 2, 1) @ ga)
    edges = np.stack([a, b], 1)
    diag = np.zeros((n, 6, 6))
    np.add.at(diag, a, ga.transpose(0, 2, 1) @ ga)
    np.add.at(diag, b, gb.transpose(0, 2, 1) @ gb)
    diag += np.eye(6) * (1.0 + 0.05 * np.trace(diag.mean(0)) / 6)
    return diag, edges.astype(np.uint32), off.astype(np.float32), rng.standard_normal((n, 6))


def dense(diag, edges, off):
    n = len(diag)
    S = np.zeros((n, 6, n, 6))
    S[np.arange(n), :, np.arange(n), :] = diag
    a, b = edges[:, 0], edges[:, 1]
    S[b, :, a, :] = off
    S[a, :, b, :] = off.transpose(0, 2, 1)
    return S.reshape(6 * n, 6 * n)


def pcg64(S, diag, rhs, tol, cap):
    n = len(diag)
    inv = np.linalg.inv(diag)
    prec = lambda r: np.einsum("nab,nb->na", inv, r.reshape(n, 6)).reshape(-1)  # noqa: E731
    b = rhs.reshape(-1)
    x, r = np.zeros_like(b), b.copy()
    z = prec(r)
    p, rz = z.copy(), r @ z
    for k in range(cap):
        q = S @ p
        alpha = rz / (p @ q)
        x += alpha * p
        r -= alpha * q
        if np.linalg.norm(r) <= tol * np.linalg.norm(b):
            return x, k + 1
        z = prec(r)
        new = r @ z
        p, rz = z + (new / rz) * p, new
    return x, cap


@pytest.mark.parametrize("n", [1, 2, 5, 8, 15, 16, 17, 31, 32, 33, 63, 64, 65, 71, 127, 128, 129, 151, 256,
                               330, 449, 490])
@pytest.mark.parametrize("keep", [1.0, 0.15])
def test_matches_the_fp64_iteration(solver, n, keep):
    diag, edges, off, rhs = system(n, keep, 7 * n)
    S = dense(diag, edges, off)
    x, it, rr = solver.reduced_solve(diag, edges, off, rhs, 1e-5, 300)
    ref, it_ref = pcg64(S, diag, rhs, 1e-5, 300)
    assert abs(it - it_ref) <= 1 and rr <= 1e-5
    # Both stop within 1e-5 |b| of the solution's residual: they differ by
    # at most twice that over the smallest eigenvalue, and FP32 rounding.
    lmin = np.linalg.eigvalsh(S)[0]
    bound = 2e-5 * np.linalg.norm(rhs) / lmin + 1e-5 * np.linalg.norm(ref)
    assert np.linalg.norm(x.reshape(-1) - ref) <= bound
    # A few iterations only: the iterates themselves, before rounding grows.
    if n >= 5:
        x3, it3, _ = solver.reduced_solve(diag, edges, off, rhs, 0.0, 3)
        ref3, _ = pcg64(S, diag, rhs, -1.0, 3)
        assert it3 == 3
        assert np.linalg.norm(x3.reshape(-1) - ref3) <= 1e-5 * np.linalg.norm(ref3)
    # The same bits on a repeated call.
    again, _, _ = solver.reduced_solve(diag, edges, off, rhs, 1e-5, 300)
    assert np.array_equal(again, x)


def kernel_of(s, problem, monkeypatch, capfd):
    """Which PCG kernel solves the problem: the persistent one alone fills the
    phase trace, and only a team has waits for the probe to run out."""
    with monkeypatch.context() as m:
        m.setenv("VLBA_TRACE_PCG", "1")
        capfd.readouterr()
        st, _ = s.optimize(problem.copy(), BaConfig(max_iterations=1, max_pcg_iterations=3))
        assert st == 0
        if "vlba pcg trace:" in capfd.readouterr().err:
            return "persistent"
    s.wait_probe(1.0)
    return "team" if "a bounded device wait" in s.last_error() else "cluster"


@pytest.mark.parametrize("cameras,kernel", [(128, "cluster"), (129, "team"), (576, "team"),
                                            (577, "persistent")])
def test_the_kernel_of_a_dense_system_follows_its_size(solver, cameras, kernel, monkeypatch, capfd):
    p = synth.ring_problem(cameras + 2, 40 * cameras, seed=cameras)  # two cameras are fixed
    assert kernel_of(solver, p, monkeypatch, capfd) == kernel


@pytest.mark.parametrize("n", [513, 520, 569, 576, 577, 584, 600])
def test_dense_systems_at_the_limit_of_the_teams(solver, n):
    """The largest layouts of a team (576 nodes: 36 parts a block, 20 of them in
    shared memory) and the first sizes of the persistent kernel."""
    diag, edges, off, rhs = system(n, 1.0, n)
    S = dense(diag, edges, off)
    x3, it3, _ = solver.reduced_solve(diag, edges, off, rhs, 0.0, 3)
    ref3, _ = pcg64(S, diag, rhs, -1.0, 3)
    assert it3 == 3
    assert np.linalg.norm(x3.reshape(-1) - ref3) <= 1e-5 * np.linalg.norm(ref3)
    x, it, rr = solver.reduced_solve(diag, edges, off, rhs, 1e-5, 300)
    _, it_ref = pcg64(S, diag, rhs, 1e-5, 300)
    assert abs(it - it_ref) <= 1 and rr <= 1e-5
    assert np.linalg.norm(S @ x.reshape(-1) - rhs.reshape(-1)) <= 2e-5 * np.linalg.norm(rhs)


@pytest.mark.parametrize("n", [3, 20, 50, 100, 140, 480, 600])
def test_stopping_rules(solver, n):
    """Zero right-hand side, iteration cap 0 and 1, non-positive curvature
    (x stays at the last iterate) and NaN: as the persistent kernel."""
    diag, edges, off, rhs = system(n, 0.5, n)
    x, it, _ = solver.reduced_solve(diag, edges, off, 0.0 * rhs, 1e-6, 50)
    assert it == 0 and not x.any()
    x, it, _ = solver.reduced_solve(diag, edges, off, rhs, 1e-6, 0)
    assert it == 0 and not x.any()
    x, it, _ = solver.reduced_solve(diag, edges, off, rhs, 1e-12, 1)
    assert it == 1 and x.any()
    # Indefinite beyond the block diagonal: large couplings.
    x, it, _ = solver.reduced_solve(diag, edges, 100.0 * off, rhs, 1e-6, 50)
    assert it < 50 and np.isfinite(x).all()
    bad = rhs.copy()
    bad[0, 0] = np.nan
    x, it, _ = solver.reduced_solve(diag, edges, off, bad, 1e-6, 50)
    assert it == 0 and not x.any()


@pytest.mark.parametrize("cameras", [12, 40, 60, 100, 150, 620])
def test_a_negative_tolerance_is_never_met(solver, cameras):
    """|r| <= tol |b| cannot hold for tol < 0: every kernel runs to the cap
    (with the square of the bound it held once |r| <= |b|)."""
    p = synth.ring_problem(cameras, 40 * cameras, seed=cameras)
    cfg = BaConfig(robust_kernel=RobustKernel.huber(1.0), max_pcg_iterations=9)
    cfg.pcg_relative_tolerance = -1.0
    never = solver.linear_step(p, cfg, 1e-3)
    assert never[2] == 9
    cfg.pcg_relative_tolerance = 0.0
    zero = solver.linear_step(p, cfg, 1e-3)
    assert zero[2] == 9 and np.array_equal(never[0], zero[0])


@pytest.mark.parametrize("band", [2, 9, 40, 60, 120])
def test_banded_team(solver, band):
    """A long chain (1,400 nodes, more tile rows than blocks at the widest
    team): each block reads its own stretch of columns.  The widest band fits
    no team."""
    n = 1400
    rng = np.random.default_rng(band)
    a = np.repeat(np.arange(n), band)
    b = a + np.tile(np.arange(1, band + 1), n)
    edges = np.stack([a, b], 1)[b < n]
    a, b = edges[:, 0], edges[:, 1]
    ga, gb = (np.eye(6) + 0.3 * rng.standard_normal((len(a), 6, 6)) for _ in range(2))
    off = -(gb.transpose(0, 2, 1) @ ga).astype(np.float32)
    diag = np.tile(np.eye(6) * 0.5, (n, 1, 1))
    np.add.at(diag, a, ga.transpose(0, 2, 1) @ ga)
    np.add.at(diag, b, gb.transpose(0, 2, 1) @ gb)
    rhs = rng.standard_normal((n, 6))
    x, it, _ = solver.reduced_solve(diag, edges, off, rhs, 0.0, 4)
    ref, _ = pcg64(dense(diag, edges, off), diag, rhs, -1.0, 4)
    assert it == 4
    assert np.linalg.norm(x.reshape(-1) - ref) <= 1e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("big", [False, True])
def test_teams_solve_the_same_alone_and_in_a_batch(solver, big):
    """Problems of the cluster and team kernels, and with `big` of the
    persistent one, in one batch (teams in two rounds): the bits of each
    solved alone."""
    probs = [synth.ring_problem(140, 6000, seed=1), synth.stereo_window(20, 800, seed=2),
             synth.ring_problem(200, 8000, seed=3), synth.ring_problem(300, 20000, seed=4),
             synth.street_loop(500, 20000, seed=5), synth.ring_problem(100, 4000, seed=6)]
    if big:
        probs[1:1] = [synth.ring_problem(610, 24400, seed=7)]
        probs.append(synth.ring_problem(700, 21000, seed=8))
    cfg = BaConfig(max_iterations=4, robust_kernel=RobustKernel.huber(1.0), max_pcg_iterations=60,
                   pcg_relative_tolerance=1e-6)
    alone = [p.copy() for p in probs]
    costs = []
    for p in alone:
        st, res = solver.optimize(p, cfg)
        assert st == 0
        costs.append(res.final_cost)
    for graph in (False, True):
        cfg.graph = graph
        batch = [p.copy() for p in probs]
        statuses, results = solver.batch_optimize(batch, cfg)
        assert statuses == [0] * len(probs)
        for a, b, c, r in zip(alone, batch, costs, results):
            assert r.final_cost == c
            assert np.array_equal(a.pose_q, b.pose_q) and np.array_equal(a.landmarks, b.landmarks)


def test_finished_problems_of_the_persistent_kernel_stay_out(solver):
    """Iteration caps apart: each kernel's problems end at their own iteration
    while the others go on, in either order."""
    probs = [synth.ring_problem(610, 24400, seed=7), synth.ring_problem(40, 2000, seed=2),
             synth.ring_problem(620, 24800, seed=9), synth.ring_problem(200, 8000, seed=3)]
    for caps in ((1, 4, 3, 2), (4, 1, 2, 3)):
        cfgs = [BaConfig(max_iterations=m, robust_kernel=RobustKernel.huber(1.0),
                         max_pcg_iterations=40, pcg_relative_tolerance=1e-6) for m in caps]
        batch = [p.copy() for p in probs]
        statuses, results = solver.batch_optimize(batch, cfgs)
        assert statuses == [0] * len(probs)
        for p, b, c, r in zip(probs, batch, cfgs, results):
            alone = p.copy()
            st, res = solver.optimize(alone, c)
            assert st == 0 and res.final_cost == r.final_cost
            assert [i.pcg_iterations for i in res.iterations] == [i.pcg_iterations for i in r.iterations]
            assert np.array_equal(alone.pose_q, b.pose_q) and np.array_equal(alone.landmarks, b.landmarks)


def test_each_round_of_teams_is_a_launch(solver):
    """A team's waits never cover another team's solve: two teams that do not
    fit the device together (112 blocks each) take a launch each."""
    one = synth.ring_problem(300, 20000, seed=4)
    cfg = BaConfig(max_iterations=2, robust_kernel=RobustKernel.huber(1.0), max_pcg_iterations=20)
    st, alone = solver.optimize(one.copy(), cfg)
    assert st == 0
    statuses, both = solver.batch_optimize([one.copy(), one.copy()], cfg)
    assert statuses == [0, 0]
    assert both[0].kernel_launches == alone.kernel_launches + 2
    assert both[0].final_cost == both[1].final_cost == alone.final_cost


def test_the_phase_trace_covers_the_persistent_kernel_only(solver, monkeypatch, capfd):
    """VLBA_TRACE_PCG prints what k_pcg measured, and nothing for systems that
    it does not solve (their trace memory holds nothing)."""
    monkeypatch.setenv("VLBA_TRACE_PCG", "1")
    cfg = BaConfig(max_iterations=2, max_pcg_iterations=12)
    small, big = synth.ring_problem(20, 800, seed=1), synth.ring_problem(620, 24800, seed=2)
    statuses, _ = solver.batch_optimize([small.copy(), synth.ring_problem(140, 5600, seed=3)], cfg)
    assert statuses == [0, 0] and capfd.readouterr().err == ""
    statuses, results = solver.batch_optimize([small.copy(), big.copy()], cfg)
    assert statuses == [0, 0]
    lines = [s for s in capfd.readouterr().err.splitlines() if s.startswith("vlba pcg trace:")]
    assert [int(s.split()[3]) for s in lines] == [i.pcg_iterations for i in results[1].iterations]
    assert all(0.0 < float(s.split()[-1]) < 1e4 for s in lines)


@pytest.mark.parametrize("cluster", [1, 8])
def test_without_large_clusters_the_teams_take_over(cluster, monkeypatch):
    """On a device that places no cluster of 16 (or 4) blocks, the systems
    those solve go to a team of blocks."""
    from visloc_ba.solver import CudaSolver

    monkeypatch.setenv("VLBA_MAX_CLUSTER", str(cluster))
    with CudaSolver(0) as s:
        for n in (17, 33, 40, 64, 65, 100, 128):
            diag, edges, off, rhs = system(n, 0.6, n)
            x, it, _ = s.reduced_solve(diag, edges, off, rhs, 0.0, 3)
            ref, _ = pcg64(dense(diag, edges, off), diag, rhs, -1.0, 3)
            assert it == 3
            assert np.linalg.norm(x.reshape(-1) - ref) <= 1e-5 * np.linalg.norm(ref)
