"""The plan-bound mv_AN as the operator of pgmres / pgmresDR / bicgstab (the C
ABI's NULL operator) against the oracle with the same mv_AN handle."""
import ctypes as C

import numpy as np
import pytest

from oracle import vie_oracle as vo

pytestmark = pytest.mark.gpu
FREQ = 298e6


def system(L=8, dx=5e-3, radius=0.018):
    r = vo.grid(L, L, L, dx)
    er = np.ones((L, L, L), complex)
    er[np.sum(r * r, axis=3) < radius**2] = 50.0 - 30.0j
    er = np.asfortranarray(er)
    V = L * L * L
    idxS = np.flatnonzero(np.abs(er.reshape(-1, order="F") - 1) > 1e-12)
    idx = (np.concatenate([idxS, V + idxS, 2 * V + idxS]) + 1).astype(np.int64)
    Mr = np.asfortranarray(er / er)
    Mc = np.asfortranarray((er - 1) / er)
    fN = vo.getOPERATORS(r, FREQ)
    rng = np.random.default_rng(3)
    b = rng.standard_normal(idx.size) + 1j * rng.standard_normal(idx.size)
    return fN, Mr, Mc, dx**3, idx, b


@pytest.mark.parametrize("transp", ["notransp", "transp"])
def test_bound_mv_AN_in_krylov_solvers(transp):
    import marie_gb300 as mg

    fN, Mr, Mc, Gram, idx, b = system()
    op = mg.Operator.from_array(fN).bind_mv_AN(Mr, Mc, Gram, transp, idx)
    A = lambda v: vo.mv_AN(v, fN, Mr, Mc, Gram, transp, idx)
    ref = vo.pgmres(A, b, 10, 1e-10, 20)
    out = mg.pgmres(op, b, 10, 1e-10, 20)
    assert out[1] == ref[1] == 0 and out[3] == ref[3]
    np.testing.assert_allclose(out[4], ref[4], rtol=1e-6, atol=1e-14)
    assert np.linalg.norm(out[0] - ref[0]) <= 1e-8 * np.linalg.norm(ref[0])
    refb = vo.bicgstab(A, b, 1e-10, 200)
    outb = mg.bicgstab(op, b, 1e-10, 200)
    # BiCGSTAB's path follows the rounding of the FFTs (cuFFT-free device
    # transforms here, pocketfft in the oracle): same answer, counts close
    assert outb[1] == refb[1] == 0 and abs(outb[3] - refb[3]) <= 0.1 * refb[3] + 2
    assert np.linalg.norm(outb[0] - refb[0]) <= 1e-7 * np.linalg.norm(refb[0])
    refd = vo.pgmresDR(A, b, 10, 1e-10, 20, 3)
    outd = mg.pgmresDR(op, b, 10, 1e-10, 20, 3)
    assert outd[1] == refd[1] == 0 and outd[3] == refd[3]
    assert np.linalg.norm(outd[0] - refd[0]) <= 1e-8 * np.linalg.norm(refd[0])


def test_null_operator_needs_a_binding(cuda):
    import marie_gb300 as mg

    fN, Mr, Mc, Gram, idx, b = system()
    op = mg.Operator.from_array(fN)
    with pytest.raises(mg.MarieError):
        mg.pgmres(op, b, 10, 1e-8, 5)
    op.bind_mv_AN(Mr, Mc, Gram, "notransp", idx)
    with pytest.raises(mg.MarieError):
        mg.pgmres(op, b[:-3], 10, 1e-8, 5)
    with pytest.raises(ValueError):
        op.bind_mv_AN(Mr, Mc, Gram, "both", idx)


@pytest.mark.parametrize("transp", ["notransp", "transp"])
def test_apply_bound_mv_AN(cuda, transp):
    """marie_plan_apply_mv_AN: the bound mv_AN without a per-call DOF map; FP64
    gives the bits of marie_mv_AN, FP32 (epilogue in FP32 too) meets the FP32
    bar against the oracle; host and device vectors, two right-hand sides."""
    import torch

    import marie_gb300 as mg

    fN, Mr, Mc, Gram, idx, b = system(L=16, dx=3e-3, radius=0.02)
    rng = np.random.default_rng(8)
    J = np.asfortranarray(rng.standard_normal((idx.size, 2)) + 1j * rng.standard_normal((idx.size, 2)))
    op = mg.Operator.from_array(fN, precision="mixed", nrhs_max=2).bind_mv_AN(Mr, Mc, Gram, transp, idx)
    ref = np.stack([vo.mv_AN(J[:, c], fN, Mr, Mc, Gram, transp, idx) for c in range(2)], axis=1)
    scale = np.max(np.abs(ref))
    out64 = op.apply_mv_AN(J, "fp64")
    np.testing.assert_array_equal(out64, mg.mv_AN(J, op, Mr, Mc, Gram, transp, idx, precision="fp64"))
    assert np.max(np.abs(out64 - ref)) / scale < 1e-12
    out32 = op.apply_mv_AN(J, "fp32")
    assert np.max(np.abs(out32 - ref)) / scale < 1e-5
    Jd = torch.from_numpy(J[:, 0].copy()).to(cuda)
    outd = op.apply_mv_AN(Jd, "fp32")
    assert outd.is_cuda
    np.testing.assert_array_equal(outd.cpu().numpy(), out32[:, 0])
    op.close()


def _off_centre_body(shape, lo, size, dx=4e-3, seed=5):
    """A box of scattered non-air voxels inside a larger grid of air."""
    rng = np.random.default_rng(seed)
    r = vo.grid(*shape, dx)
    er = np.ones(shape, complex)
    part = er[tuple(slice(a, a + s) for a, s in zip(lo, size))]
    part[rng.random(size) < 0.7] = 30.0 - 20.0j
    part[0, 0, 0] = part[-1, -1, -1] = 12.0 - 3.0j
    return r, np.asfortranarray(er)


# grids above the crop's smallest size; boxes at an edge, in the middle and
# one voxel above a supported size; one, two and three axes shrink
CROPS = [((48, 32, 40), (0, 3, 20), (17, 8, 20)), ((32, 96, 12), (5, 40, 0), (27, 33, 12)),
         ((40, 32, 32), (12, 9, 11), (9, 23, 21))]


@pytest.mark.parametrize("shape,lo,size", CROPS)
@pytest.mark.parametrize("transp", ["notransp", "transp"])
def test_bound_product_on_the_bodys_box(cuda, shape, lo, size, transp):
    """A body that leaves most of its grid empty: the bound product, run on the
    smallest grid that holds the body, against the unbound one on the whole
    grid; 1e-13 of the largest value in FP64 (the smaller spectrum carries a
    few roundings of its own), the FP32 bar in FP32, two columns."""
    import marie_gb300 as mg

    r, er = _off_centre_body(shape, lo, size)
    op = mg.Operator.assemble(*shape, 4e-3, FREQ, precision="mixed", nrhs_max=2)
    V = er.size
    idxS = np.flatnonzero(np.abs(er.reshape(-1, order="F") - 1) > 1e-12) + 1
    idx = np.concatenate([idxS, V + idxS, 2 * V + idxS]).astype(np.int64)
    Mr, Mc = np.asfortranarray(er / er), np.asfortranarray((er - 1) / er)
    rng = np.random.default_rng(2)
    J = np.asfortranarray(rng.standard_normal((idx.size, 2)) + 1j * rng.standard_normal((idx.size, 2)))
    ref = mg.mv_AN(J, op, Mr, Mc, 4e-3**3, transp, idx)
    op.bind_mv_AN(Mr, Mc, 4e-3**3, transp, idx)
    scale = np.max(np.abs(ref))
    assert np.max(np.abs(op.apply_mv_AN(J, "fp64") - ref)) < 1e-13 * scale
    assert np.max(np.abs(op.apply_mv_AN(J, "fp32") - ref)) < 1e-5 * scale
    # another operator in the plan: the bound DOFs follow it
    other = mg.Operator.assemble(*shape, 4e-3, 0.5 * FREQ)
    fN = other.to_array()
    mg._lib.check(op.lib.marie_set_operator(op.plan, C.c_void_p(fN.ctypes.data), *fN.shape[:3]))
    ref = mg.mv_AN(J, op, Mr, Mc, 4e-3**3, transp, idx)
    assert np.max(np.abs(op.apply_mv_AN(J, "fp64") - ref)) < 1e-13 * np.max(np.abs(ref))
    op.close()


@pytest.mark.parametrize("shape,lo,size", CROPS[:2])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_solves_on_the_bodys_box(cuda, shape, lo, size, precision):
    """JVIE_Solver ('G', 'B'), the batch, jvie2solver and the gradient of a body
    in a mostly empty grid against the same calls on a grid cut around it by
    hand: the same flags, and fields equal to the solves' tolerance (1e-9,
    times a condition of up to 1e3); two bodies in turn on one plan."""
    import marie_gb300 as mg
    from marie_gb300.autograd import adjoint_gradient

    dx, em = 4e-3, vo.EMconstants(FREQ)
    small = [mg.supported_size(s) for s in size]
    cut = tuple(slice(min(a, n - s), min(a, n - s) + s) for a, n, s in zip(lo, shape, small))
    op = mg.Operator.assemble(*shape, dx, FREQ, precision=precision, nrhs_max=2)
    ref_op = mg.Operator.assemble(*small, dx, FREQ, precision=precision, nrhs_max=2)

    def calls(op, r, er, E):
        E2 = np.asfortranarray(np.stack([E, 1j * E[..., ::-1]], axis=4))
        V = er.size
        idxS = np.flatnonzero(np.abs(er.reshape(-1, order="F") - 1) > 1e-12) + 1
        idx = np.concatenate([idxS, V + idxS, 2 * V + idxS]).astype(np.int64)
        Mr, Mc = np.asfortranarray(er / er), np.asfortranarray((er - 1) / er)
        yield mg.JVIE_Solver(E, er, r, FREQ, op, tol=1e-9, solver="G")[:2]
        yield mg.JVIE_Solver(E, er, r, FREQ, op, tol=1e-9, solver="B")[:2]
        yield mg.JVIE_Solver_batch(E2, er, r, FREQ, op, tol=1e-9)[:2]
        b = E.reshape(-1, order="F")[idx - 1] * dx**3
        yield mg.jvie2solver(b, op, idx, Mr, Mc, dx**3, 1e-9)[:2]
        g = adjoint_gradient(op, E, er, dx, FREQ, "power", tol=1e-9)
        yield g[1], g[3]

    for k in range(2):
        r, er = _off_centre_body(shape, lo, [s - 2 * k for s in size], seed=5 + k)
        E = np.asfortranarray(vo.PlaneWave_Excitation(r, [0, 0, em["ko"]], em["omega_mu"], [1, 0, 0])[0])
        f = lambda a: np.asfortranarray(a[cut])
        for (x, fx), (y, fy) in zip(calls(op, r, er, E), calls(ref_op, f(r), f(er), f(E))):
            assert np.all(np.asarray(fx) == 0) and np.all(np.asarray(fy) == 0)
            inside = x[cut] if x.ndim > 1 else x
            assert np.linalg.norm(inside - y) <= 1e-6 * np.linalg.norm(y)
            assert np.count_nonzero(inside) == np.count_nonzero(x)  # nothing outside the body
    op.close()
    ref_op.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape,lo,size", [((12, 12, 20), (2, 4, 5), (8, 8, 12)), ((40, 24, 40), (0, 3, 0), (40, 20, 40)),
                                           ((40, 40, 24), (0, 0, 4), (40, 40, 20)),
                                           ((32, 32, 48), (0, 0, 3), (32, 32, 40))])
def test_solves_on_the_bodys_rows_and_planes(cuda, shape, lo, size, precision):
    """Grids that are not cut to the body's box (small, or filled to more than
    0.8): the passes run over the box's rows and planes of the whole grid, the
    last shape with the fused x+y passes in FP32.  Against a grid that is the
    box, as above."""
    import marie_gb300 as mg

    dx, em = 4e-3, vo.EMconstants(FREQ)
    cut = tuple(slice(a, a + s) for a, s in zip(lo, size))
    r, er = _off_centre_body(shape, lo, size)
    E = np.asfortranarray(vo.PlaneWave_Excitation(r, [0, 0, em["ko"]], em["omega_mu"], [1, 0, 0])[0])
    out = []
    for grid, c in ((shape, (slice(None),) * 3), (size, cut)):
        op = mg.Operator.assemble(*grid, dx, FREQ, precision=precision)
        ec, Ec, rc = (np.asfortranarray(a[c]) for a in (er, E, r))
        J, flag = mg.JVIE_Solver(Ec, ec, rc, FREQ, op, tol=1e-9, solver="G")[:2]
        V = ec.size
        idxS = np.flatnonzero(np.abs(ec.reshape(-1, order="F") - 1) > 1e-12) + 1
        idx = np.concatenate([idxS, V + idxS, 2 * V + idxS]).astype(np.int64)
        b = Ec.reshape(-1, order="F")[idx - 1] * dx**3
        x, flag2 = mg.jvie2solver(b, op, idx, np.asfortranarray(ec / ec), np.asfortranarray((ec - 1) / ec), dx**3, 1e-9)[:2]
        assert flag == 0 and flag2 == 0
        out.append((J if grid == size else J[cut], x, np.count_nonzero(J)))
        op.close()
    (J, x, nz), (Jr, xr, nzr) = out
    assert nz == nzr
    assert np.linalg.norm(J - Jr) <= 1e-6 * np.linalg.norm(Jr)
    assert np.linalg.norm(x - xr) <= 1e-6 * np.linalg.norm(xr)


def _bound_operator(shape, precision, dx=4e-3, seed=5, keep=0.6, box=None, cls_args=()):
    import marie_gb300 as mg

    lo, size = box or ((0, 0, 0), shape)
    er = np.ones(shape, complex, order="F")
    part = er[tuple(slice(a, a + s) for a, s in zip(lo, size))]
    part[np.random.default_rng(seed).random(size) < keep] = 30.0 - 20.0j
    part[0, 0, 0] = part[-1, -1, -1] = 12.0 - 3.0j
    idxS = np.flatnonzero(np.abs(er.reshape(-1, order="F") - 1) > 1e-12) + 1
    idx = np.concatenate([idxS, er.size + idxS, 2 * er.size + idxS]).astype(np.int64)
    op = mg.Operator.assemble(*shape, dx, FREQ, precision=precision, nrhs_max=2)
    return op, er, idx


@pytest.mark.parametrize("shape", [(8, 12, 16), (20, 20, 8), (48, 48, 4), (64, 64, 8), (16, 96, 8)])
@pytest.mark.parametrize("transp", ["notransp", "transp"])
def test_fp32_products_keep_the_diagonal_term_in_fp64(cuda, shape, transp):
    """Grids without fused passes: FP32 arithmetic is the circulant's, the
    diagonal Gram Mr J of FP64 vectors is FP64's.  With Mc = 0 it is all there
    is: one complex product, three roundings (Gram Mr: one more)."""
    op, er, idx = _bound_operator(shape, "mixed")
    rng = np.random.default_rng(1)
    J = rng.standard_normal(idx.size) + 1j * rng.standard_normal(idx.size)
    Mr = np.asfortranarray(1 + 40 * rng.random(shape) - 20j * rng.random(shape))
    op.bind_mv_AN(Mr, np.zeros(shape, complex, order="F"), 0.37, transp, idx)
    m = Mr.reshape(-1, order="F")[(idx - 1) % Mr.size]
    ref = 0.37 * (m if transp == "notransp" else np.conj(m)) * J
    out = op.apply_mv_AN(J, "fp32")
    assert np.max(np.abs(out - ref) / np.abs(ref)) <= 1e-15
    op.close()


def _launches(op, call):
    import torch

    torch.cuda.synchronize()
    n0 = op.lib.marie_launch_count()
    out = call()
    torch.cuda.synchronize()
    return out, op.lib.marie_launch_count() - n0


@pytest.mark.parametrize("how", ["autotune", "schedule"])
def test_a_schedule_without_choice_leaves_the_box_its_fused_passes(cuda, how):
    """A 48 x 48 grid has no fused x+y passes, so tuning it chooses nothing; the
    64 x 64 transforms of a 32 x 32 body in it keep theirs: three passes a
    product, before and after."""
    shape = (48, 48, 16)
    op, er, idx = _bound_operator(shape, "mixed", box=((5, 9, 0), (32, 32, 16)))
    op.bind_mv_AN(np.asfortranarray(er / er), np.asfortranarray((er - 1) / er), 4e-3**3, "notransp", idx)
    rng = np.random.default_rng(4)
    J = rng.standard_normal(idx.size) + 1j * rng.standard_normal(idx.size)
    op.apply_mv_AN(J, "fp32")
    ref, before = _launches(op, lambda: op.apply_mv_AN(J, "fp32"))
    if how == "autotune":
        chosen, cands = op.autotune()
        assert chosen == (0, 0, 0) and len(cands) == 1
    else:
        op.set_schedule(0, 0, 0)
    out, after = _launches(op, lambda: op.apply_mv_AN(J, "fp32"))
    assert before == after == 3
    np.testing.assert_array_equal(out, ref)
    op.close()


def test_schedule_of_a_grid_with_fused_passes_holds_on_its_box(cuda):
    """On a grid that has fused passes the schedule is a choice, for the box cut
    from it along z as well; the products agree to the FP32 bar."""
    op, er, idx = _bound_operator((32, 32, 48), "mixed", box=((0, 0, 3), (32, 32, 20)))
    op.bind_mv_AN(np.asfortranarray(er / er), np.asfortranarray((er - 1) / er), 4e-3**3, "notransp", idx)
    rng = np.random.default_rng(4)
    J = rng.standard_normal(idx.size) + 1j * rng.standard_normal(idx.size)
    ref = op.apply_mv_AN(J, "fp64")
    for fuse, passes in ((1, 3), (0, 5), (1, 3)):
        op.set_schedule(fuse, 0, 0)
        out, n = _launches(op, lambda: op.apply_mv_AN(J, "fp32"))
        assert n == passes and np.max(np.abs(out - ref)) < 1e-5 * np.max(np.abs(ref))
    op.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_solves_without_memory_for_the_box(cuda, precision):
    """Whatever allocation of a solve fails once the caller's buffers are there,
    the box's operator or one beside it, the solve takes the whole grid."""
    import torch

    import marie_gb300 as mg
    from marie_gb300.autograd import adjoint_gradient

    shape, lo, size = CROPS[0]
    r, er = _off_centre_body(shape, lo, size)
    em = vo.EMconstants(FREQ)
    E = vo.PlaneWave_Excitation(r, [0, 0, em["ko"]], em["omega_mu"], [1, 0, 0])[0]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a.transpose())).to(cuda).permute(*reversed(range(a.ndim)))
    Ed, erd = dev(E), dev(er)
    op = mg.Operator.assemble(*shape, 4e-3, FREQ, precision=precision)
    idxS = torch.nonzero((erd.permute(2, 1, 0).reshape(-1) - 1).abs() > 1e-12)[:, 0] + 1
    idx = torch.cat([idxS + c * erd.numel() for c in range(3)])
    b = Ed.permute(3, 2, 1, 0).reshape(-1)[idx - 1] * 4e-3**3
    Mr, Mc = erd / erd, (erd - 1) / erd
    torch.cuda.synchronize()

    def gradient():
        F, g, _, flags, _ = adjoint_gradient(op, Ed, erd, 4e-3, FREQ, "power", tol=1e-8)
        return g, max(flags)

    for solve in (lambda: mg.JVIE_Solver(Ed, erd, r, FREQ, op, tol=1e-8, solver="G")[:2],
                  lambda: mg.JVIE_Solver(Ed, erd, r, FREQ, op, tol=1e-8, solver="B")[:2],
                  lambda: mg.jvie2solver(b, op, idx, Mr, Mc, 4e-3**3, 1e-8)[:2], gradient):
        ref, _ = solve()
        torch.cuda.synchronize()
        for nth in (2, 3, 6, 9, 12, 16, 22, 30):
            solve()
            op.lib.marie_inject_alloc_failure(nth)
            try:
                x, flag = solve()
            finally:
                op.lib.marie_inject_alloc_failure(0)
            assert flag == 0
            assert float((x - ref).norm()) <= 1e-5 * float(ref.norm())
            torch.cuda.synchronize()
    op.close()


@pytest.mark.parametrize("nth", [1, 2, 3, 4, 5])
def test_binding_and_first_solve_without_memory_for_the_box(cuda, nth):
    """On a fresh plan the nth allocation from the bind on fails: the bind falls
    back to the whole grid or reports MARIE_ENOMEM, and the products are right."""
    import torch

    import marie_gb300 as mg

    shape, lo, size = CROPS[0]
    op, er, idx = _bound_operator(shape, "mixed", box=(lo, size))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a.transpose())).to(cuda).permute(*reversed(range(a.ndim)))
    Mr, Mc, idx_d = dev(er / er), dev((er - 1) / er), torch.from_numpy(idx).to(cuda)
    rng = np.random.default_rng(3)
    J = torch.from_numpy(rng.standard_normal(idx.size) + 1j * rng.standard_normal(idx.size)).to(cuda)
    torch.cuda.synchronize()
    ref = mg.mv_AN(J, op, Mr, Mc, 4e-3**3, "notransp", idx_d)
    op.lib.marie_inject_alloc_failure(nth)
    try:
        op.bind_mv_AN(Mr, Mc, 4e-3**3, "notransp", idx_d)
    except mg.MarieError as e:
        assert e.code == -2
        op.lib.marie_inject_alloc_failure(0)
        op.bind_mv_AN(Mr, Mc, 4e-3**3, "notransp", idx_d)
    finally:
        op.lib.marie_inject_alloc_failure(0)
    assert float((op.apply_mv_AN(J, "fp64") - ref).abs().max()) < 1e-13 * float(ref.abs().max())
    op.close()


def test_bodies_on_their_boxes_in_one_launch(cuda):
    """Two bodies on grids that are cut to their boxes, solved in one graph
    launch, give bit for bit their own batches."""
    import marie_gb300 as mg

    em = vo.EMconstants(FREQ)
    bodies = []
    for shape, lo, size in CROPS[:2]:
        r, er = _off_centre_body(shape, lo, size)
        E = vo.PlaneWave_Excitation(r, [0, 0, em["ko"]], em["omega_mu"], [1, 0, 0])[0]
        op = mg.Operator.assemble(*shape, 4e-3, FREQ, precision="mixed", nrhs_max=2)
        bodies.append((np.asfortranarray(np.stack([E, 1j * E[..., ::-1]], axis=4)), er, r, op))
    alone = [mg.JVIE_Solver_batch(E, er, r, FREQ, op, tol=1e-7) for E, er, r, op in bodies]
    n0 = bodies[0][3].lib.marie_graph_loops()
    res, _ = mg.JVIE_Solver_bodies(bodies, FREQ, tol=1e-7)
    assert bodies[0][3].lib.marie_graph_loops() == n0 + 1
    for (J, flag, relres, it), ref in zip(res, alone):
        np.testing.assert_array_equal(J, ref[0])
        assert list(flag) == [0, 0] and np.all(relres <= 1e-7)
    for b in bodies:
        b[3].close()


@pytest.mark.parametrize("name", ["apply", "mv_AN", "mv_L", "E_field", "mv_K", "H_field", "pgmres", "pgmresDR",
                                  "bicgstab", "solve", "batch", "inner", "gradient", "scat"])
def test_calls_beside_a_boxs_operator_without_memory(cuda, name):
    """Beside the operator of a box, which a bound mv_AN or a solve left on the
    plan, the nth allocation of a call fails: the plan gives that operator back
    and the call runs as it does without one.  Host arrays, so the calls' own
    buffers are among the allocations.  Products and fields on either grid agree
    to 1e-13, solves to their tolerance times a condition of up to 1e3."""
    import marie_gb300 as mg
    from marie_gb300.autograd import adjoint_gradient

    shape, lo, size = CROPS[0]
    dx = 4e-3
    r, er = _off_centre_body(shape, lo, size)
    op = mg.Operator.assemble(*shape, dx, FREQ, precision="fp64", nrhs_max=2).assemble_k(dx, FREQ)
    em = vo.EMconstants(FREQ)
    E = np.asfortranarray(vo.PlaneWave_Excitation(r, [0, 0, em["ko"]], em["omega_mu"], [1, 0, 0])[0])
    idxS = np.flatnonzero(np.abs(er.reshape(-1, order="F") - 1) > 1e-12) + 1
    idx = np.concatenate([idxS, er.size + idxS, 2 * er.size + idxS]).astype(np.int64)
    Mr, Mc = np.asfortranarray(er / er), np.asfortranarray((er - 1) / er)
    rng = np.random.default_rng(8)
    J = rng.standard_normal(idx.size) + 1j * rng.standard_normal(idx.size)
    F = np.asfortranarray(rng.standard_normal(E.shape) + 1j * rng.standard_normal(E.shape))
    b = E.reshape(-1, order="F")[idx - 1] * dx**3
    E2 = np.asfortranarray(np.stack([E, 1j * E], axis=4))
    eps, sig = np.asfortranarray(er.real), np.asfortranarray(-er.imag * 2 * np.pi * FREQ * 8.854e-12)
    calls = {
        "apply": lambda: op.apply_mv_AN(J, "fp64"),
        "mv_AN": lambda: mg.mv_AN(J, op, Mr, Mc, dx**3, "notransp", idx),
        "mv_L": lambda: mg.mv_L(J, op, r, dx**3, idx),
        "E_field": lambda: mg.E_field_Nop(F, op, dx**3, FREQ, E),
        "mv_K": lambda: mg.mv_K(J, op, r, idx),
        "H_field": lambda: mg.H_field_Kop(F, op, dx**3, E),
        "pgmres": lambda: mg.pgmres(op, b, 30, 1e-8, 20)[0],
        "pgmresDR": lambda: mg.pgmresDR(op, b, 30, 1e-8, 20, 4)[0],
        "bicgstab": lambda: mg.bicgstab(op, b, 1e-8, 400)[0],
        "solve": lambda: mg.JVIE_Solver(E, er, r, FREQ, op, tol=1e-8)[0],
        "batch": lambda: mg.JVIE_Solver_batch(E2, er, r, FREQ, op, tol=1e-8)[0],
        "inner": lambda: mg.jvie2solver(b, op, idx, Mr, Mc, dx**3, 1e-8)[0],
        "gradient": lambda: adjoint_gradient(op, E, er, dx, FREQ, "power", tol=1e-8)[1],
        "scat": lambda: mg.Scat_Solver(E, None, FREQ, r, eps, sig, np.ones(shape, order="F"), tol=1e-8, fN=op)[0],
    }
    call = calls[name]
    bind = lambda: op.bind_mv_AN(Mr, Mc, dx**3, "notransp", idx)
    bind()
    ref = np.asarray(call())
    tol = 1e-13 if name in ("apply", "mv_AN", "mv_L", "E_field", "mv_K", "H_field") else 1e-5
    for nth in (1, 2, 3, 5, 8):
        bind()
        op.lib.marie_inject_alloc_failure(nth)
        try:
            out = np.asarray(call())
        finally:
            op.lib.marie_inject_alloc_failure(0)
        assert np.max(np.abs(out - ref)) <= tol * np.max(np.abs(ref))
    op.close()


def test_a_bound_box_given_back_leaves_the_whole_grids_product(cuda):
    """After a solve that found no memory the bound product runs on the whole grid
    (bit for bit the product that per-pass timing runs there) until it is bound
    again."""
    import marie_gb300 as mg

    shape, lo, size = CROPS[0]
    op, er, idx = _bound_operator(shape, "fp64", box=(lo, size))
    bind = lambda: op.bind_mv_AN(np.asfortranarray(er / er), np.asfortranarray((er - 1) / er), 4e-3**3, "notransp", idx)
    bind()
    rng = np.random.default_rng(6)
    J = rng.standard_normal(idx.size) + 1j * rng.standard_normal(idx.size)
    on_box = op.apply_mv_AN(J, "fp64")
    op.lib.marie_plan_profile(op.plan, 1, None, None)
    whole = op.apply_mv_AN(J, "fp64")
    op.lib.marie_plan_profile(op.plan, 0, None, None)
    assert np.any(on_box != whole)
    r = vo.grid(*shape, 4e-3)
    em = vo.EMconstants(FREQ)
    E = np.asfortranarray(vo.PlaneWave_Excitation(r, [0, 0, em["ko"]], em["omega_mu"], [1, 0, 0])[0])
    op.lib.marie_inject_alloc_failure(6)
    try:
        assert mg.JVIE_Solver(E, er, r, FREQ, op, tol=1e-6)[1] == 0
    finally:
        op.lib.marie_inject_alloc_failure(0)
    np.testing.assert_array_equal(op.apply_mv_AN(J, "fp64"), whole)
    bind()
    np.testing.assert_array_equal(op.apply_mv_AN(J, "fp64"), on_box)
    op.close()
