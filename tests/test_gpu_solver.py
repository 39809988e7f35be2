"""GPU parity of pgmres and JVIE_Solver against the oracle restatements of
pgmres.m / pgmres_iter.m / JVIE_Solver.m, the mixed-precision solve against
the FP64 solve, and the Mie-series sphere check (RUN_Sphere_VIE_MIE.m)."""
import numpy as np
import pytest

from oracle import mie
from oracle import vie_oracle as vo

pytestmark = pytest.mark.gpu
FREQ = 298e6


def dense(n, seed):
    rng = np.random.default_rng(seed)
    A = np.eye(n) * 3 + 0.4 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    return A, b


@pytest.mark.parametrize("restart,tol,maxit", [(10, 1e-10, 20), (5, 1e-6, 3), (50, 1e-12, 2)])
def test_pgmres_host_handles_match_oracle(restart, tol, maxit):
    import marie_gb300 as mg

    A, b = dense(60, restart)
    ref = vo.pgmres(lambda v: A @ v, b, restart, tol, maxit)
    out = mg.pgmres(lambda v: A @ v, b, restart, tol, maxit)
    assert out[1] == ref[1]
    assert out[3] == ref[3]
    np.testing.assert_allclose(out[4], ref[4], rtol=1e-8, atol=1e-14)
    np.testing.assert_allclose(out[0], ref[0], rtol=1e-9, atol=1e-12)
    assert abs(out[2] - ref[2]) <= 1e-9 * max(ref[2], 1e-12) + 1e-15


def test_pgmres_preconditioners_and_x0(cuda):
    import torch

    import marie_gb300 as mg

    A, b = dense(50, 4)
    P = np.diag(1.0 / np.diag(A))
    Pt = torch.from_numpy(P).to(cuda)
    At = torch.from_numpy(A).to(cuda)
    x0 = np.full(50, 0.1 + 0.2j)
    for kw in (dict(R1=lambda v: P @ v), dict(L1=lambda v: P @ v), dict(L1=lambda v: P @ v, R2=lambda v: P @ v)):
        ref = vo.pgmres(lambda v: A @ v, b, 8, 1e-9, 10, x0=x0, **kw)
        out = mg.pgmres(lambda v: A @ v, b, 8, 1e-9, 10, x0=x0, **kw)
        assert out[3] == ref[3] and out[1] == ref[1]
        np.testing.assert_allclose(out[4], ref[4], rtol=1e-8, atol=1e-14)
        np.testing.assert_allclose(out[0], ref[0], rtol=1e-8)
    # device handles on a device right-hand side
    bt = torch.from_numpy(b).to(cuda)
    out = mg.pgmres(lambda v: At @ v, bt, 8, 1e-9, 10, R1=lambda v: Pt @ v)
    ref = vo.pgmres(lambda v: A @ v, b, 8, 1e-9, 10, R1=lambda v: P @ v)
    assert out[0].is_cuda
    np.testing.assert_allclose(out[0].cpu().numpy(), ref[0], rtol=1e-8)


def sphere_problem(L, dx, radius, eps_r=50.0, sigma=0.5):
    r = vo.grid(L, L, L, dx)
    er = np.ones((L, L, L), complex)
    er[np.sum(r * r, axis=3) < radius**2] = eps_r - 1j * sigma / (vo.EPS0 * 2 * np.pi * FREQ)
    em = vo.EMconstants(FREQ)
    E, _ = vo.PlaneWave_Excitation(r, [0, 0, em["ko"]], em["omega_mu"], [1, 0, 0])
    return r, np.asfortranarray(er), np.asfortranarray(E)


@pytest.mark.parametrize("form,precond", [(2, 0), (1, 0), (1, "R"), (2, "L")])
def test_jvie_solver_matches_oracle(form, precond):
    import marie_gb300 as mg

    L, dx = 8, 5e-3
    r, er, E = sphere_problem(L, dx, 0.018)
    fN = vo.getOPERATORS(r, FREQ)
    ref = vo.JVIE_Solver(E, er, r, FREQ, fN, tol=1e-10, form=form, precond=precond, inner_it=20, solver="G")
    op = mg.Operator.from_array(fN)
    out = mg.JVIE_Solver(E, er, r, FREQ, op, tol=1e-10, form=form, precond=precond, inner_it=20, solver="G")
    assert out[1] == ref[1] == 0
    assert out[3] == ref[3]
    np.testing.assert_allclose(out[4], ref[4], rtol=1e-6, atol=1e-13)
    assert np.max(np.abs(out[0] - ref[0])) < 1e-8 * np.max(np.abs(ref[0]))


@pytest.mark.parametrize("restart", [31, 33, 65, 127])
def test_rotations_and_back_substitution_past_a_warp(restart):
    """The Givens step composes the previous rotations over 32 lanes a round
    and the back-substitution holds up to four rows a lane: restarts around and
    past 32 and 64 against the oracle, on a sphere that takes over 65 steps and
    is far from exhausting its Krylov space (an operator perturbed by 2e-15
    moves the oracle's residuals by at most 8e-11 and its fields by 2e-13:
    1e-8 and 1e-10 here, and the last estimate equals the true residual to the
    same digits)."""
    import marie_gb300 as mg

    L, dx = 12, 5e-3
    r, er, E = sphere_problem(L, dx, 0.028, eps_r=3000.0, sigma=0.02)
    fN = vo.getOPERATORS(r, FREQ)
    kw = dict(tol=1e-6, inner_it=restart, solver="G")
    ref = vo.JVIE_Solver(E, er, r, FREQ, fN, **kw)
    out = mg.JVIE_Solver(E, er, r, FREQ, mg.Operator.from_array(fN), **kw)
    assert out[1] == ref[1] == 0 and out[3] == ref[3] and len(ref[4]) > 65
    np.testing.assert_allclose(out[4], ref[4], rtol=1e-8)
    assert abs(out[4][-1] / out[2] - 1) < 1e-8
    assert np.max(np.abs(out[0] - ref[0])) < 1e-10 * np.max(np.abs(ref[0]))


def test_restart_cycles_run_in_one_graph_launch():
    """After the first restart cycle, the remaining cycles of a GMRES call run
    in one graph launch (a conditional WHILE node whose body is one cycle and
    its device-side close); the solve matches the oracle's as before."""
    import marie_gb300 as mg

    L, dx = 8, 5e-3
    r, er, E = sphere_problem(L, dx, 0.018)
    fN = vo.getOPERATORS(r, FREQ)
    ref = vo.JVIE_Solver(E, er, r, FREQ, fN, tol=1e-10, inner_it=10, solver="G")
    lib = mg.load()
    n0 = lib.marie_graph_loops()
    out = mg.JVIE_Solver(E, er, r, FREQ, mg.Operator.from_array(fN), tol=1e-10, inner_it=10, solver="G")
    assert ref[3][1] > 2  # several restart cycles
    assert lib.marie_graph_loops() > n0
    assert out[1] == ref[1] == 0 and out[3] == ref[3]
    np.testing.assert_allclose(out[4], ref[4], rtol=1e-6, atol=1e-13)


@pytest.mark.parametrize("precision,precond", [("fp64", 0), ("fp64", "R"), ("mixed", 0)])
def test_batched_excitations_match_single_solves(precision, precond):
    """Several excitations of one body in one lockstep batch give the same
    fields and iteration counts as one-at-a-time solves (c3 structure)."""
    import marie_gb300 as mg

    L, dx = 8, 5e-3
    r, er, E1 = sphere_problem(L, dx, 0.018)
    em = vo.EMconstants(FREQ)
    E2, _ = vo.PlaneWave_Excitation(r, [0, 0, em["ko"]], em["omega_mu"], [0, 1, 0])
    E3 = vo.Dipole_Excitation(r, em["ko"], np.array([[0, 0, 1.0]]), np.array([[0.05, 0.0, 0.01]]))
    Eb = np.asfortranarray(np.stack([E1, E2, E3], axis=4))
    op = mg.Operator.assemble(L, L, L, dx, FREQ, precision=precision, nrhs_max=3)
    Jb, flags, relres, iters, _ = mg.JVIE_Solver_batch(Eb, er, r, FREQ, op, tol=1e-8, precond=precond,
                                                      inner_it=15)
    for e in range(3):
        Js, fs, rs, its, _, _ = mg.JVIE_Solver(np.asfortranarray(Eb[..., e]), er, r, FREQ, op, tol=1e-8,
                                               precond=precond, inner_it=15, solver="G")
        assert flags[e] == fs == 0
        if precision == "fp64":
            assert list(iters[e]) == list(its)
            assert np.max(np.abs(Jb[..., e] - Js)) <= 1e-9 * np.max(np.abs(Js))
        else:
            # each system of the batch refines with its own inner tolerances,
            # so it takes the single solve's steps: the same bits
            assert list(iters[e]) == list(its) and relres[e] == rs <= 1e-8
            np.testing.assert_array_equal(Jb[..., e], Js)
    if precision == "fp64":
        fN = op.to_array()
        for e in range(3):
            ref = vo.JVIE_Solver(np.asfortranarray(Eb[..., e]), er, r, FREQ, fN, tol=1e-8, precond=precond,
                                 inner_it=15, solver="G")
            assert ref[3] == list(iters[e])
            assert np.max(np.abs(Jb[..., e] - ref[0])) < 1e-7 * np.max(np.abs(ref[0]))


@pytest.mark.parametrize("precision,precond", [("fp64", 0), ("fp64", "R"), ("mixed", 0), ("mixed", "L")])
def test_batch_in_two_groups_gives_the_same_bits(precision, precond):
    """Two groups of excitations on two streams (one group's Gram-Schmidt
    beside the other's matvec) give bit for bit the fields, iteration counts
    and residual histories of the one-group lockstep batch, with an uneven
    split (3 excitations: 2 + 1) and restart cycles in the conditional graph."""
    import marie_gb300 as mg

    L, dx = 12, 5e-3
    r, er, E1 = sphere_problem(L, dx, 0.025)
    em = vo.EMconstants(FREQ)
    E2, _ = vo.PlaneWave_Excitation(r, [0, 0, em["ko"]], em["omega_mu"], [0, 1, 0])
    E3 = vo.Dipole_Excitation(r, em["ko"], np.array([[0, 0, 1.0]]), np.array([[0.06, 0.0, 0.01]]))
    Eb = np.asfortranarray(np.stack([E1, E2, E3], axis=4))
    op = mg.Operator.assemble(L, L, L, dx, FREQ, precision=precision, nrhs_max=3)
    kw = dict(tol=1e-9, precond=precond, inner_it=8)
    op.set_batch_groups(1)
    one = mg.JVIE_Solver_batch(Eb, er, r, FREQ, op, **kw)
    lib = mg.load()
    n0 = lib.marie_graph_loops()
    op.set_batch_groups(2)
    two = mg.JVIE_Solver_batch(Eb, er, r, FREQ, op, **kw)
    assert lib.marie_graph_loops() > n0
    np.testing.assert_array_equal(two[0], one[0])
    assert list(map(list, two[3])) == list(map(list, one[3]))
    np.testing.assert_array_equal(two[2], one[2])
    assert np.all(np.asarray(two[1]) == 0)
    op.set_batch_groups(1)
    again = mg.JVIE_Solver_batch(Eb, er, r, FREQ, op, **kw)
    np.testing.assert_array_equal(again[0], one[0])
    with pytest.raises(mg.MarieError):
        op.set_batch_groups(3)
    op.close()


@pytest.mark.parametrize("basis,precond,groups", [("fp64", 0, 2), ("fp64", "R", 1), ("fp32", "L", 2),
                                                  ("fp64", "L", 1)])
def test_graph_refinement_matches_host_driven(basis, precond, groups):
    """The mixed-precision refinement as one graph launch (nested conditional
    WHILE nodes, the device deciding every step) gives bit for bit the
    fields, flags, iteration counts and residual histories of the
    host-driven refinement, for a batch and for a single excitation."""
    import marie_gb300 as mg

    L, dx = 12, 5e-3
    r, er, E1 = sphere_problem(L, dx, 0.025, eps_r=80.0, sigma=1.0)
    em = vo.EMconstants(FREQ)
    E2, _ = vo.PlaneWave_Excitation(r, [0, 0, em["ko"]], em["omega_mu"], [0, 1, 0])
    E3 = vo.Dipole_Excitation(r, em["ko"], np.array([[0, 0, 1.0]]), np.array([[0.06, 0.0, 0.01]]))
    Eb = np.asfortranarray(np.stack([E1, E2, E3], axis=4))
    op = mg.Operator.assemble(L, L, L, dx, FREQ, precision="mixed", nrhs_max=3)
    op.set_inner_precision(basis).set_batch_groups(groups).set_inner_restart(6)
    kw = dict(tol=1e-9, precond=precond, inner_it=30)
    lib = mg.load()
    res = {}
    for graph in (False, True):
        op.set_graph_refinement(graph)
        n0 = lib.marie_graph_loops()
        batch = mg.JVIE_Solver_batch(Eb, er, r, FREQ, op, **kw)
        single = mg.JVIE_Solver(np.asfortranarray(E2), er, r, FREQ, op, solver="G", **kw)
        res[graph] = (batch, single, lib.marie_graph_loops() - n0)
    (bh, sh, _), (bg, sg, loops) = res[False], res[True]
    assert loops >= 2  # the batch and the single solve each ran as one graph launch
    np.testing.assert_array_equal(bg[0], bh[0])
    assert list(map(list, bg[3])) == list(map(list, bh[3]))
    np.testing.assert_array_equal(bg[2], bh[2])
    assert list(bg[1]) == list(bh[1]) == [0, 0, 0]
    np.testing.assert_array_equal(sg[0], sh[0])
    assert sg[1] == sh[1] == 0 and list(sg[3]) == list(sh[3]) and sg[2] == sh[2]
    np.testing.assert_array_equal(np.asarray(sg[4]), np.asarray(sh[4]))
    assert len(sg[4]) > 10
    op.close()


def test_uneven_bodies_solved_concurrently():
    """Three bodies of different grid sizes with two dipole excitations each
    (c3 structure at test sizes) give the same fields as separate solves."""
    import marie_gb300 as mg
    from marie_gb300 import phantoms

    em = vo.EMconstants(FREQ)
    bodies, singles = [], []
    for seed, L in ((1, 12), (2, 16), (3, 24)):
        dx = 2e-3
        r, er, _ = phantoms.ellipsoids(L, L, L, dx, 3, seed, FREQ)
        pos = phantoms.dipole_ring(0.6 * L * dx, [0.0, 0.25 * L * dx], 1)
        Es = [vo.Dipole_Excitation(r, em["ko"], np.array([[0, 0, 1.0]]), p[None]) for p in pos]
        Eb = np.asfortranarray(np.stack(Es, axis=4))
        op = mg.Operator.assemble(L, L, L, dx, FREQ, precision="mixed", nrhs_max=2)
        bodies.append((Eb, er, r, op))
        singles.append([mg.JVIE_Solver(np.asfortranarray(E), er, r, FREQ, op, tol=1e-7, solver="G")[0] for E in Es])
    res, t = mg.JVIE_Solver_bodies(bodies, FREQ, tol=1e-7)
    for (Je, flag, relres, it), ref in zip(res, singles):
        assert np.all(flag == 0) and np.all(relres <= 1e-7)
        for e in range(2):
            assert np.linalg.norm(Je[..., e] - ref[e]) <= 1e-5 * np.linalg.norm(ref[e])


def test_uneven_bodies_in_one_graph_launch():
    """The refinements of three bodies of different grid sizes run as ONE
    graph launch (their loops are independent branches of one graph) and
    give bit for bit each body's own batched solve."""
    import marie_gb300 as mg
    from marie_gb300 import phantoms

    em = vo.EMconstants(FREQ)
    bodies = []
    for seed, L in ((1, 12), (2, 16), (3, 24)):
        r, er, _ = phantoms.ellipsoids(L, L, L, 2e-3, 3, seed, FREQ)
        pos = phantoms.dipole_ring(0.6 * L * 2e-3, [0.0, 0.25 * L * 2e-3], 1)
        Eb = np.asfortranarray(np.stack([vo.Dipole_Excitation(r, em["ko"], np.array([[0, 0, 1.0]]), p[None])
                                         for p in pos], axis=4))
        op = mg.Operator.assemble(L, L, L, 2e-3, FREQ, precision="mixed", nrhs_max=2)
        op.set_inner_restart(8)
        bodies.append((Eb, er, r, op))
    lib = mg.load()
    alone = [mg.JVIE_Solver_batch(Eb, er, r, FREQ, op, tol=1e-8) for Eb, er, r, op in bodies]
    n0 = lib.marie_graph_loops()
    res, _ = mg.JVIE_Solver_bodies(bodies, FREQ, tol=1e-8)
    assert lib.marie_graph_loops() == n0 + 1  # one launch for all three bodies
    for (Je, flg, rel, it), ref in zip(res, alone):
        np.testing.assert_array_equal(Je, ref[0])
        assert list(flg) == list(ref[1]) == [0, 0]
        np.testing.assert_array_equal(rel, ref[2])
        assert list(map(list, it)) == list(map(list, ref[3]))
    # one plan driven from the host: the bodies go back to one host thread
    # each (no shared launch), with the same bits
    bodies[1][3].set_graph_refinement(False)
    n1 = lib.marie_graph_loops()
    res2, _ = mg.JVIE_Solver_bodies(bodies, FREQ, tol=1e-8)
    assert lib.marie_graph_loops() == n1 + 2  # bodies 0 and 2 launch their own graphs
    for (Je, flg, rel, it), ref in zip(res2, alone):
        np.testing.assert_array_equal(Je, ref[0])
        np.testing.assert_array_equal(rel, ref[2])
    for b in bodies:
        b[3].close()


def test_mixed_precision_solve_matches_fp64():
    import marie_gb300 as mg

    L, dx = 16, 5e-3
    r, er, E = sphere_problem(L, dx, 0.035)
    op64 = mg.Operator.assemble(L, L, L, dx, FREQ, precision="fp64")
    opm = mg.Operator.assemble(L, L, L, dx, FREQ, precision="mixed")
    J64, f64, rr64, it64, _, _ = mg.JVIE_Solver(E, er, r, FREQ, op64, tol=1e-6, solver="G")
    Jm, fm, rrm, itm, resm, _ = mg.JVIE_Solver(E, er, r, FREQ, opm, tol=1e-6, solver="G")
    assert f64 == 0 and fm == 0 and rrm <= 1e-6
    # both solutions satisfy the FP64 system to 1e-6: fields agree to ~cond * tol
    assert np.linalg.norm(Jm - J64) / np.linalg.norm(J64) < 2e-5


@pytest.mark.parametrize("precond", [0, "L", "R"])
def test_mixed_inner_basis_fp32_and_fp64(precond):
    """The inner GMRES of the mixed-precision refinement with an FP32 Krylov
    basis (the default) and with an FP64 one: both reach the FP64 residual bar
    and give the FP64 solve's field to the same accuracy, with every
    preconditioner side (form 1, where the preconditioner is not the identity).
    32^3 has fused x+y passes (64^3 FFT grid)."""
    import marie_gb300 as mg

    L, dx = 32, 2.5e-3
    r, er, E = sphere_problem(L, dx, 0.035)
    op64 = mg.Operator.assemble(L, L, L, dx, FREQ, precision="fp64")
    opm = mg.Operator.assemble(L, L, L, dx, FREQ, precision="mixed")
    J64 = mg.JVIE_Solver(E, er, r, FREQ, op64, tol=1e-8, form=1, precond=precond, inner_it=20, solver="G")[0]
    errs = {}
    # the FP32 basis runs the matvec on FP32 vectors: fused x+y passes and the
    # five-pass form
    for inner, fuse in (("fp64", 1), ("fp32", 1), ("fp32", 0)):
        opm.set_inner_precision(inner).set_schedule(fuse, 0, 0)
        Jm, fm, rrm, itm, resm, _ = mg.JVIE_Solver(E, er, r, FREQ, opm, tol=1e-8, form=1, precond=precond,
                                                   inner_it=20, solver="G")
        assert fm == 0 and rrm <= 1e-8, (inner, fuse, rrm)
        assert resm[-1] == pytest.approx(rrm)
        errs[(inner, fuse)] = np.linalg.norm(Jm - J64) / np.linalg.norm(J64)
    assert all(e < 1e-6 for e in errs.values()), errs


def test_inner_settings_validated():
    import marie_gb300 as mg

    op = mg.Operator(8, 8, 8, precision="mixed")
    op.set_inner_precision("fp64").set_inner_precision("fp32").set_inner_restart(0).set_inner_restart(127)
    with pytest.raises(mg.MarieError):
        op.set_inner_restart(128)
    with pytest.raises(mg.MarieError):
        op.set_inner_restart(-1)
    with pytest.raises(KeyError):
        op.set_inner_precision("fp16")


def mie_error(L, dx, R, precision="fp64"):
    import marie_gb300 as mg

    r, er, E = sphere_problem(L, dx, R)
    op = mg.Operator.assemble(L, L, L, dx, FREQ, precision=precision)
    Je, flag, relres, it, resvec, _ = mg.JVIE_Solver(E, er, r, FREQ, op, tol=1e-6, solver="G")
    assert flag == 0
    Et = mg.E_field_Nop(Je, op, dx**3, FREQ, E)
    rad = np.sqrt(np.sum(r * r, axis=3))
    core = rad < R - 0.01  # away from the staircased surface
    Em = mie.MIE_SERIES(r[core][:, None, None, :], R, 50.0, 0.5, FREQ)[:, 0, 0, :]
    return np.linalg.norm(Et[core] - Em) / np.linalg.norm(Em)


def test_mie_sphere_c1_and_refinement():
    """The sphere of RUN_Sphere_VIE_MIE.m at the c1 sizes: r = 7.5 cm, eps_r = 50,
    sigma = 0.5 S/m, 298 MHz, x-polarised +z plane wave.  The reference compares
    with the Mie series visually.  Here the relative L2 error of the total field
    more than 1 cm inside the surface is bounded at 5 mm (32^3, the staircased
    sphere carries a first-order discretisation error) and must shrink when the
    voxel size is halved (2.5 mm, 64^3), as the discretisation converges."""
    e5 = mie_error(32, 5e-3, 0.075)
    e25 = mie_error(64, 2.5e-3, 0.075, precision="mixed")
    assert e5 < 0.35, e5
    assert e25 < 0.65 * e5, (e5, e25)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_solves_while_their_passes_are_timed(precision):
    """With marie_plan_profile on, a solve of several restart cycles (the graph
    forms otherwise), a batch and two bodies together run their products one by
    one: the same bits, and every product counted."""
    import ctypes as C

    import marie_gb300 as mg

    L, dx = 16, 5e-3
    r, er, E = sphere_problem(L, dx, 0.035)
    E2 = np.asfortranarray(np.stack([E, 2j * E], axis=4))
    ops = [mg.Operator.assemble(L, L, L, dx, FREQ, precision=precision, nrhs_max=2) for _ in range(2)]
    op = ops[0]

    def calls():
        one = mg.JVIE_Solver(E, er, r, FREQ, op, tol=1e-8, inner_it=5, solver="G")
        two = mg.JVIE_Solver_batch(E2, er, r, FREQ, op, tol=1e-8, inner_it=5)
        both = mg.JVIE_Solver_bodies([(E2, er, r, o) for o in ops], FREQ, tol=1e-8, inner_it=5)[0]
        return one[0], one[3], two[0], list(map(list, two[3])), both[0][0], both[1][0]

    ref = calls()
    ms, n = (C.c_double * 5)(), C.c_int64()
    timed = lambda on: op.lib.marie_plan_profile(op.plan, on, ms, C.byref(n))
    timed(1)
    out = calls()
    timed(0)
    for a, b in zip(out, ref):
        np.testing.assert_array_equal(np.asarray(a), np.asarray(b))
    assert n.value > 3 * 10 and min(ms) >= 0 and ms[2] > 0
    for o in ops:
        o.close()
