"""The J-VIE solve as the coil solvers' inner solver: fVIEsolver_Assembly.m
(crop, operator cache, tau3, Scoord) and jvie2solver.m (BiCGSTAB with an
initial guess) against the oracle restatement."""
import numpy as np
import pytest

from oracle import vie_oracle as vo

pytestmark = pytest.mark.gpu
FREQ = 298e6


def body(L, dx, region):
    """RHBM dict on an L^3 grid: a lossy block (region = index slices) in air."""
    r = vo.grid(L, L, L, dx)
    eps = np.ones((L, L, L))
    sig = np.zeros((L, L, L))
    eps[region] = 45.0
    sig[region] = 0.6
    inner = tuple(slice(s.start + 1, s.stop - 1) for s in region)
    eps[inner] = 70.0
    return {"r": r, "epsilon_r": np.asfortranarray(eps), "sigma_e": np.asfortranarray(sig), "fN": None,
            "freqfN": None}


def incident(R, Scoord, tau3):
    """tau3 .* E_inc at the non-air voxels (the coil solvers' right-hand side)."""
    em = vo.EMconstants(FREQ)
    E, _ = vo.PlaneWave_Excitation(R["r"], [0, 0, em["ko"]], em["omega_mu"], [1, 0.5, 0])
    nonair = np.flatnonzero(np.abs(R["epsilon_r"].reshape(-1, order="F") - 1) > 0)
    Es = np.concatenate([E[..., c].reshape(-1, order="F")[nonair] for c in range(3)])
    return tau3 * Es


@pytest.mark.parametrize("region", [
    (slice(4, 14), slice(4, 14), slice(4, 14)),
    (slice(5, 14), slice(3, 12), slice(6, 15)),
])
def test_fviesolver_matches_oracle(region):
    import marie_gb300 as mg

    R = body(20, 5e-3, region)
    solver, Gram, tau3, Scoord, op = mg.fVIEsolver_Assembly(R, FREQ)
    rsolver, rGram, rtau3, rScoord, (re_r, ridx, rfN) = vo.fVIEsolver_Assembly(R, FREQ)
    # the reference's crop (the oracle), extended with air to the next FFT size
    assert re_r.shape[0] < 20 and (op.L, op.M, op.N) == tuple(mg.supported_size(n) for n in re_r.shape)
    assert Gram == rGram
    np.testing.assert_allclose(tau3, rtau3, rtol=1e-15)
    np.testing.assert_array_equal(Scoord, rScoord)
    b = incident(R, Scoord, tau3)
    x, flag, relres, it = rsolver(b, 1e-8)
    xs = solver(b, 1e-8)
    assert flag == 0
    assert np.linalg.norm(xs - x) <= 1e-6 * np.linalg.norm(x)


def test_jvie2solver_initial_guess_and_zero_rhs(cuda):
    import torch

    import marie_gb300 as mg

    R = body(16, 5e-3, (slice(3, 11), slice(4, 12), slice(2, 10)))
    solver, Gram, tau3, Scoord, op = mg.fVIEsolver_Assembly(R, FREQ)
    rsolver, _, _, _, (re_r, ridx, rfN) = vo.fVIEsolver_Assembly(R, FREQ)
    b = incident(R, Scoord, tau3)
    # the low-level entry with the cropped body's data: iterations and flags as the oracle
    e_r = np.ones((op.L, op.M, op.N), complex, order="F")
    e_r[:re_r.shape[0], :re_r.shape[1], :re_r.shape[2]] = re_r
    nd = e_r.size
    idxS = np.flatnonzero(np.abs(e_r.reshape(-1, order="F") - 1) > 1e-12)
    idx = np.concatenate([idxS, nd + idxS, 2 * nd + idxS]).astype(np.int64) + 1
    Mr, Mc = np.asfortranarray(e_r / e_r), np.asfortranarray((e_r - 1) / e_r)
    x, flag, relres, it, _ = mg.jvie2solver(b, op, idx, Mr, Mc, Gram, 1e-9)
    rx, rflag, rrelres, rit = rsolver(b, 1e-9)
    assert flag == rflag == 0 and abs(it - rit) <= 1.0, (it, rit)
    assert np.linalg.norm(x - rx) <= 1e-6 * np.linalg.norm(rx)
    # starting from the solution: converged at once
    x2, flag2, relres2, it2, _ = mg.jvie2solver(b, op, idx, Mr, Mc, Gram, 1e-6, Vini=x)
    assert flag2 == 0 and it2 == 0 and relres2 <= 1e-6
    # an all-zero right-hand side is returned as the solution
    z, fz, rz, iz, _ = mg.jvie2solver(np.zeros_like(b), op, idx, Mr, Mc, Gram, 1e-6)
    assert not np.any(z) and fz == 0 and iz == 0
    # device vectors in place
    bd = torch.from_numpy(b).to(cuda)
    xd = solver(bd, 1e-9)
    assert xd.is_cuda and np.linalg.norm(xd.cpu().numpy() - rx) <= 1e-6 * np.linalg.norm(rx)


def scattered(L, dx, precision, seed=3, keep=0.5):
    """jvie2solver's arguments for scattered lossy voxels on an L^3 grid."""
    import marie_gb300 as mg

    rng = np.random.default_rng(seed)
    er = np.ones((L, L, L), complex)
    er[rng.random(er.shape) < keep] = 40.0 - 25.0j
    er = np.asfortranarray(er)
    idxS = np.flatnonzero(np.abs(er.reshape(-1, order="F") - 1) > 1e-12) + 1
    idx = np.concatenate([idxS, er.size + idxS, 2 * er.size + idxS]).astype(np.int64)
    b = (rng.standard_normal(idx.size) + 1j * rng.standard_normal(idx.size)) * dx**3
    op = mg.Operator.assemble(L, L, L, dx, FREQ, precision=precision)
    return op, idx, np.asfortranarray(er / er), np.asfortranarray((er - 1) / er), dx**3, b, rng


def products_of(op, call):
    """call() and the products the plan ran in it."""
    import ctypes as C

    ms, n = (C.c_double * 5)(), C.c_int64()
    op.lib.marie_plan_profile(op.plan, 1, ms, C.byref(n))
    try:
        out = call()
    finally:
        op.lib.marie_plan_profile(op.plan, 0, ms, C.byref(n))
    return out, n.value


def test_jvie2solver_products_stay_in_proportion_and_within_max_it(cuda):
    """A solve that starts near the solution takes a few products, not the
    closing cycle's ten as well, and max_it bounds the products.  BiCGSTAB takes
    two per iteration, one for the start's residual and up to five
    confirmations; the closing cycle at most a quarter of the iterations'."""
    import marie_gb300 as mg

    op, idx, Mr, Mc, Gram, b, rng = scattered(12, 5e-3, "fp64")
    solve = lambda tol, **k: mg.jvie2solver(b, op, idx, Mr, Mc, Gram, tol, **k)
    x = solve(1e-12)[0]
    near = x + 1e-6 * np.linalg.norm(x) / np.sqrt(x.size) * (rng.standard_normal(x.size) + 1j * rng.standard_normal(x.size))
    (_, flag, relres, it, _), n = products_of(op, lambda: solve(2e-7, Vini=near))
    assert flag == 0 and relres <= 2e-7 and 0 < it <= 6, (it, relres)
    assert n <= 2.5 * it + 6, (n, it)
    (_, flag, _, it, _), n = products_of(op, lambda: solve(1e-6))
    assert flag == 0 and n <= 2.5 * it + 6, (n, it)
    most = int(np.ceil(it))
    (_, flag, _, it, _), n = products_of(op, lambda: solve(1e-6, max_it=most))
    assert flag == 0 and it <= most and n <= 2 * most + 6, (n, it)
    op.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("tol", [1e-2, 1e-4, 1e-7])
def test_jvie2solver_relres_is_the_returned_vectors(precision, tol, cuda):
    """relres is ||b - A x|| / ||b|| of the vector that is returned, cold and
    from a start near the solution; the two products' roundings move it by 1e-13
    at most."""
    import marie_gb300 as mg

    op, idx, Mr, Mc, Gram, b, rng = scattered(12, 5e-3, precision)
    cold = mg.jvie2solver(b, op, idx, Mr, Mc, Gram, tol)
    x0 = cold[0] * (1 + 30 * tol * rng.standard_normal(b.size))
    for x, flag, relres, it, _ in (cold, mg.jvie2solver(b, op, idx, Mr, Mc, Gram, tol, Vini=x0)):
        res = np.linalg.norm(b - mg.mv_AN(x, op, Mr, Mc, Gram, "notransp", idx)) / np.linalg.norm(b)
        assert flag == 0 and relres <= tol
        assert abs(relres - res) <= 1e-13
    op.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("voxels", [1, 2])
def test_jvie2solver_of_a_few_dofs(precision, voxels, cuda):
    """Three and six unknowns: the Krylov space is exhausted before any closing
    step, and the result stands."""
    import marie_gb300 as mg

    op, idx, Mr, Mc, Gram, b, _ = scattered(8, 5e-3, precision)
    part = np.concatenate([idx[c * len(idx) // 3:][:voxels] for c in range(3)])
    rhs = b[:part.size]
    x, flag, relres, it, _ = mg.jvie2solver(rhs, op, part, Mr, Mc, Gram, 1e-10)
    res = np.linalg.norm(rhs - mg.mv_AN(x, op, Mr, Mc, Gram, "notransp", part)) / np.linalg.norm(rhs)
    assert flag == 0 and relres <= 1e-10 and res <= 1.01e-10
    op.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_jvie2solver_allocation_failures_leave_a_converged_result(precision, cuda):
    """An allocation that fails in the solve is MARIE_ENOMEM; one that fails in
    the closing cycle leaves BiCGSTAB's result."""
    import marie_gb300 as mg

    op, idx, Mr, Mc, Gram, b, _ = scattered(12, 5e-3, precision)
    solve = lambda: mg.jvie2solver(b, op, idx, Mr, Mc, Gram, 1e-6)
    ref = solve()
    lib, stood, past = mg.load(), 0, 0
    for nth in range(1, 80):
        lib.marie_inject_alloc_failure(nth)
        try:
            x, flag, relres, it, _ = solve()
        except mg.MarieError as e:
            assert e.code == -2
            continue
        finally:
            lib.marie_inject_alloc_failure(0)
        assert flag == 0 and relres <= 1e-6 and it == ref[3]
        same = np.array_equal(x, ref[0])
        stood, past = stood + (not same), past + same
    assert stood > 0 and past > 0  # some fell into the closing cycle, some came after the last allocation
    op.close()
