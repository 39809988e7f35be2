"""The calls whose speed is measured, one or more for each part of the J-VIE path:

  mv_AN      one product with the system operator, coefficients and DOF list passed per call
  apply      the same product bound to the plan once (a Krylov loop of the user's own)
  e_field    total electric field of a current (every voxel is a DOF)
  h_field    total magnetic field of a current (the K operator)
  operators  getOPERATORS: assembly of the operator's spectrum for one frequency
  solve      JVIE_Solver, one excitation
  batch      JVIE_Solver_batch, several dipoles around one body
  inner      jvie2solver, the inner solve of the coil solvers (BiCGSTAB, the reference's default)
  gradient   the adjoint gradient of the absorbed power

Grids, resolutions and materials are those of the repository's benchmark configurations (32^3 sphere at 5 mm, 64^3 at
3 mm, 128^3 and 256 x 192 x 160 at 2 mm, 298 MHz, ellipsoid phantoms) and of its tests; draw() spreads them over the
grid sizes that the transforms take.

An FP32 product and a solve to a tolerance are right to about 1e-6, so the program keeps what they return in single
precision; FP64 products, fields and operators are kept as they come.

exact() is written in plain torch on 64-bit values: the operator from its definition (face-pair quadratures), padded
FFTs for the products and a long GMRES for the systems.
"""
import math

import numpy as np
import torch

import marie_gb300 as mg
from marie_gb300.autograd import adjoint_gradient

MU0 = 4e-7 * math.pi
C0 = 299792458.0
EPS0 = 1.0 / (C0 * C0 * MU0)
FREQ = 298e6
SIZES = (8, 12, 16, 20, 24, 32, 40, 48, 64, 80, 96, 128, 160, 192, 256)

# iterations (products) a solve cannot do without, as the reference arithmetic takes them, and rounded; for work() only
PRODUCTS = {"solve": 220, "batch": 160, "inner": 160, "gradient": 340}


def listed():
    def case(name, kind, grid, dx_mm, precision, **more):
        L, M, N = grid
        return {"name": name, "kind": kind, "L": L, "M": M, "N": N, "dx_mm": dx_mm, "precision": precision,
                "body": "ellipsoids", "transp": False, "nrhs": 1, "tol": 1e-6, **more}

    return [
        # the smallest call: one product on a coarse, uneven grid, where launches and the DOF list's set-up count
        case("mv_AN_12x8x20", "mv_AN", (12, 8, 20), 10, "fp64"),
        # four columns at once through the adjoint in FP32 (a block of coil modes on a coarse body)
        case("mv_AN_64x4_fp32_T", "mv_AN", (64, 64, 64), 3, "fp32", transp=True, nrhs=4),
        # an FP64 product on an uneven grid, as an FP64 Krylov loop does it once per step
        case("apply_96x80x64", "apply", (96, 80, 64), 2, "fp64"),
        # the product of the headline workload's inner iterations
        case("apply_128_fp32", "apply", (128, 128, 128), 2, "fp32"),
        # the largest grid, adjoint product in FP32 (sensitivities of a whole-body model)
        case("apply_256x192x160_fp32_T", "apply", (256, 192, 160), 2, "fp32", transp=True),
        # B1 map of a solved current
        case("h_field_48x40x64", "h_field", (48, 40, 64), 3, "fp64"),
        # a new frequency: the operator is assembled before any solve
        case("operators_96", "operators", (96, 96, 96), 2, "fp64"),
        # the analytic check's size: a small solve in the reference's arithmetic
        case("solve_32_sphere", "solve", (32, 32, 32), 5, "fp64", body="sphere"),
        # the headline workload: one plane wave, FP32 products refined in FP64
        case("solve_128_mixed", "solve", (128, 128, 128), 2, "mixed"),
        # eight dipoles around one body, solved together
        case("batch_64x8_mixed", "batch", (64, 64, 64), 3, "mixed", nrhs=8),
        # one inner solve of a coil solver
        case("inner_48", "inner", (48, 48, 48), 4, "fp64"),
        # one step of a material fit: two solves and the gradient, at the gradient entry point's own tolerance
        case("gradient_64_mixed", "gradient", (64, 64, 64), 3, "mixed", tol=1e-8),
    ]


def draw(rng):
    # (kind, weight, most voxels): a drawn case costs no more than the largest listed one of its kind
    kinds = (("mv_AN", 3, 96 ** 3), ("apply", 3, 160 * 128 * 128), ("e_field", 1, 96 ** 3), ("h_field", 1, 96 ** 3),
             ("operators", 2, 80 ** 3), ("solve", 2, 80 ** 3), ("batch", 1, 48 ** 3), ("inner", 1, 48 ** 3),
             ("gradient", 1, 48 ** 3))
    kind, _, most = rng.choices(kinds, [k[1] for k in kinds])[0]
    while True:
        target = math.exp(rng.uniform(math.log(8 * 8 * 8), math.log(most)))
        side = target ** (1 / 3)
        L, M, N = (min(SIZES, key=lambda s: abs(math.log(s / (side * math.exp(rng.uniform(-0.5, 0.5)))))) for _ in "xyz")
        if L * M * N <= most:
            break
    precision = rng.choice(("fp64", "mixed") if kind in ("solve", "batch", "inner", "gradient") else
                           ("fp64",) if kind == "operators" else ("fp64", "fp32"))
    solves = kind in ("solve", "batch", "inner", "gradient")
    return {"kind": kind, "L": L, "M": M, "N": N, "dx_mm": rng.choice((2, 3, 4, 5) if solves else (2, 3, 5, 8)),
            "precision": precision, "body": rng.choice(("ellipsoids", "ellipsoids", "sphere")),
            "transp": kind in ("mv_AN", "apply") and rng.random() < 0.5,
            "nrhs": rng.randint(2, 6) if kind == "batch" else rng.choice((1, 1, 2, 3)) if kind in ("mv_AN", "apply") else 1,
            "tol": 1e-8 if kind == "gradient" else rng.choice((1e-4, 1e-6)) if solves else 1e-6}


# ---------------------------------------------------------------------------------------------------------------------
# what a program has in hand: bodies, excitations, operators
# ---------------------------------------------------------------------------------------------------------------------
def _rng(seed):
    return np.random.default_rng(seed), torch.Generator(device="cuda").manual_seed(seed)


def _lines(case):
    """Voxel centres along each axis, centred on the origin."""
    dx = case["dx_mm"] * 1e-3
    return [(torch.arange(n, dtype=torch.float64, device="cuda") - (n - 1) / 2) * dx
            for n in (case["L"], case["M"], case["N"])]


def _outer(case):
    """Semi-axes of the body: 20 x 15 x 25 cm, shrunk to fit the grid."""
    dx = case["dx_mm"] * 1e-3
    axes = np.array([0.10, 0.075, 0.125])
    span = np.array([case["L"], case["M"], case["N"]]) * dx
    if case["body"] == "sphere":
        return np.full(3, min(0.075, 0.47 * span.min()))
    return axes * min(1.0, float(np.min(0.95 * span / (2 * axes))))


def _body(case, seed):
    """(eps_r, sigma), each N x M x L in memory (x fastest): a lossy body in air."""
    g, _ = _rng(seed)
    x, y, z = _lines(case)
    axes = _outer(case)

    def inside(c, a):
        return (((z - c[2]) / a[2]) ** 2)[:, None, None] + (((y - c[1]) / a[1]) ** 2)[:, None] + ((x - c[0]) / a[0]) ** 2 < 1

    body = inside((0, 0, 0), axes)
    eps = torch.ones_like(body, dtype=torch.float64)
    sig = torch.zeros_like(eps)
    if case["body"] == "sphere":
        eps[body], sig[body] = g.uniform(40, 60), g.uniform(0.4, 0.6)
        return eps, sig
    eps[body], sig[body] = g.uniform(5, 80), g.uniform(0.02, 2)
    scale = axes[0] / 0.10
    for _ in range(12):
        c = g.normal(size=3)
        c *= axes * g.uniform() ** (1 / 3) / np.linalg.norm(c)
        m = inside(c, g.uniform(0.01, 0.10, 3) * scale) & body
        eps[m], sig[m] = g.uniform(5, 80), g.uniform(0.02, 2)
    return eps, sig


def _permittivity(eps, sig):
    return torch.complex(eps, -sig / (EPS0 * 2 * math.pi * FREQ))


def _columns(t):
    """The column-major view (x first) of an array held x fastest."""
    return t.permute(*range(t.dim() - 1, -1, -1))


def _excitation(case, seed):
    """Incident fields, nrhs x 3 x N x M x L: a plane wave along z, or dipoles on a ring around the body."""
    g, _ = _rng(seed + 1)
    x, y, z = _lines(case)
    k = 2 * math.pi * FREQ / C0
    if case["kind"] != "batch":
        pol = g.uniform(0, math.pi)
        wave = torch.polar(torch.ones_like(z), -k * z)[:, None, None].expand(len(z), len(y), len(x))
        return torch.stack([math.cos(pol) * wave, math.sin(pol) * wave, 0 * wave])[None].contiguous()
    fields = []
    for i in range(case["nrhs"]):
        phi, h = 2 * math.pi * i / case["nrhs"] + g.uniform(0, 0.3), g.uniform(-0.05, 0.05)
        d = (z[:, None, None] - h, (y - 0.25 * math.sin(phi))[:, None], x - 0.25 * math.cos(phi))
        R = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
        green = torch.polar(1 / R, -k * R) * (-1j * 2 * math.pi * FREQ * MU0 / (4 * math.pi))
        a = 1 - 1j / (k * R) - 1 / (k * R) ** 2
        b = (3 / (k * R) ** 2 + 3j / (k * R) - 1) * d[0] / R
        fields.append(torch.stack([green * b * d[2] / R, green * b * d[1] / R, green * (a + b * d[0] / R)]))
    return torch.stack(fields)


def _noise(seed, *shape):
    _, g = _rng(seed + 2)
    return torch.randn(*shape, dtype=torch.complex128, generator=g, device="cuda")


def _currents(case, seed, scale):
    """A current on every voxel and an incident field of a size that the current's own field does not vanish beside."""
    J, F = (_noise(seed + i, 3, case["N"], case["M"], case["L"]) for i in (0, 10))
    return J, scale * F


def _dofs(er):
    """1-based positions of the body's unknowns in the (x, y, z, component) array."""
    v = torch.nonzero((er.reshape(-1) - 1).abs() > 1e-12)[:, 0]
    return torch.cat([v + c * er.numel() + 1 for c in range(3)])


def _grid_points(case):
    x, y, z = (t.cpu().numpy() for t in _lines(case))
    r = np.empty((len(x), len(y), len(z), 3), order="F")
    r[..., 0], r[..., 1], r[..., 2] = x[:, None, None], y[:, None], z
    return r


def _assembly_inputs(case, seed):
    """Frequency of the 'operators' cases: between 1.5 T and 7 T proton imaging."""
    g, _ = _rng(seed)
    return float(g.uniform(64e6, 300e6))


def prepare(case, seed):
    kind, dx = case["kind"], case["dx_mm"] * 1e-3
    s = {"case": case, "kept": None}
    if kind == "operators":
        s["r"] = _columns(torch.from_numpy(np.ascontiguousarray(_grid_points(case).T)).cuda())
        s["freq"] = _assembly_inputs(case, seed)
        return s
    held = "mixed" if case["precision"] in ("fp32", "mixed") else "fp64"
    if kind == "h_field":
        s["op"] = mg.Operator.from_array_k(_columns(_spectrum_k(case)), precision=held)
        s["J"], s["H"] = (_columns(v) for v in _currents(case, seed, dx))
        return s
    s["op"] = mg.Operator.from_array(_columns(_spectrum(case)), precision=held, nrhs_max=case["nrhs"])
    if kind == "e_field":
        s["J"], s["E"] = (_columns(v) for v in _currents(case, seed, 1.0))
        return s
    eps, sig = _body(case, seed)
    er = _permittivity(eps, sig)
    s["er"], s["r"] = _columns(er), _grid_points(case)
    if kind in ("solve", "batch", "gradient"):
        E = _excitation(case, seed)
        s["E"] = _columns(E if kind == "batch" else E[0])
        return s
    s["Mr"], s["Mc"] = _columns(torch.ones_like(er)), _columns((er - 1) / er)
    s["idx"] = _dofs(er)
    n = len(s["idx"])
    s["J"] = _noise(seed, n) if case["nrhs"] == 1 else _columns(_noise(seed, case["nrhs"], n))
    if kind == "inner":
        s["J"] *= dx ** 3
    if kind == "apply":
        s["op"].bind_mv_AN(s["Mr"], s["Mc"], dx ** 3, "transp" if case["transp"] else "notransp", s["idx"])
    return s


def run(s):
    case = s["case"]
    kind, dx, prec = case["kind"], case["dx_mm"] * 1e-3, case["precision"]
    if kind == "operators":
        return mg.getOPERATORS(s["r"], s["freq"], "N")
    if kind == "mv_AN":
        out = mg.mv_AN(s["J"], s["op"], s["Mr"], s["Mc"], dx ** 3, "transp" if case["transp"] else "notransp", s["idx"],
                       precision=prec)
    elif kind == "apply":
        out = s["op"].apply_mv_AN(s["J"], precision=prec)
    elif kind == "e_field":
        out = mg.E_field_Nop(s["J"], s["op"], dx ** 3, FREQ, s["E"], precision=prec)
    elif kind == "h_field":
        out = mg.H_field_Kop(s["J"], s["op"], dx ** 3, s["H"], precision=prec)
    elif kind == "gradient":
        F, d_eps, d_sig, flags, _ = adjoint_gradient(s["op"], s["E"], s["er"], dx, FREQ, "power", tol=case["tol"])
        s["kept"] = (d_eps, d_sig)
        return {"F": F, "d_eps": d_eps.float(), "d_sigma": d_sig.float(), "flags": list(flags)}
    else:
        if kind == "solve":
            out, flag = mg.JVIE_Solver(s["E"], s["er"], s["r"], FREQ, s["op"], tol=case["tol"], solver="G")[:2]
        elif kind == "batch":
            out, flag = mg.JVIE_Solver_batch(s["E"], s["er"], s["r"], FREQ, s["op"], tol=case["tol"])[:2]
        else:
            out, flag = mg.jvie2solver(s["J"], s["op"], s["idx"], s["Mr"], s["Mc"], dx ** 3, case["tol"])[:2]
        s["kept"] = out  # the library writes it on a stream of its own: it stays while the conversion below reads it
        return {"J": out.to(torch.complex64), "flag": flag}
    if prec == "fp64":
        return out
    s["kept"] = out
    return out.to(torch.complex64)


def work(case):
    """Every input read once and every output written once, and the flops of zero-padded radix-2 transforms, the 3 x 3
    products and the diagonal terms; for a solve, as many products as the system needs (PRODUCTS)."""
    kind, nrhs = case["kind"], case["nrhs"]
    L, M, N = case["L"], case["M"], case["N"]
    V, octant = L * M * N, (L + 1) * (M + 1) * (N + 1)
    q = 3 if kind == "h_field" else 6
    if kind == "operators":
        # per offset six face-pair integrals (parallel and crossed squares for each axis) of 4^4 point pairs; the FFTs
        return {"bytes": 24 * V + 16.0 * 6 * 8 * V, "flops": 6 * 256 * 40.0 * V + 5.0 * 6 * 8 * V * math.log2(8 * V)}
    n = 3 * V if kind in ("e_field", "h_field") else 4 * math.pi * np.prod(_outer(case)) / (case["dx_mm"] * 1e-3) ** 3
    fft = 30 * (2 * V * math.log2(2 * L) + 4 * V * math.log2(2 * M) + 8 * V * math.log2(2 * N))
    flops = nrhs * (fft + 528 * V)
    spectrum = octant * q * (16 if case["precision"] == "fp64" else 8)
    if kind in ("mv_AN", "apply"):
        return {"bytes": float(spectrum + n * (32 * nrhs + 8 + (32 / 3 if kind == "mv_AN" else 32))), "flops": float(flops)}
    if kind in ("e_field", "h_field"):
        return {"bytes": float(spectrum + 48 * n), "flops": float(flops)}
    times = PRODUCTS[kind]
    return {"bytes": times * float(spectrum + 32 * n * nrhs), "flops": times * float(flops)}


# ---------------------------------------------------------------------------------------------------------------------
# the operators from their definition, in plain torch
# ---------------------------------------------------------------------------------------------------------------------
def _rule(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return (x + 1) / 2, w / 2


def _differences(n):
    """Values u_i - u_k of an n-point rule and their summed weights."""
    u, w = _rule(n)
    d, at = np.unique(np.round(u[:, None] - u, 13).ravel(), return_inverse=True)
    return d, np.bincount(at.ravel(), (w[:, None] * w).ravel())


def _sum(k, dx, bases, rules):
    """sum of w exp(-j k R)/R over the rules' points, at every combination of integer base offsets (x, y, z)."""
    bases = [torch.as_tensor(b, dtype=torch.float64, device="cuda") for b in bases]
    pts = np.array(np.meshgrid(*[r[0] for r in rules], indexing="ij")).reshape(3, -1)
    wts = np.prod(np.array(np.meshgrid(*[r[1] for r in rules], indexing="ij")).reshape(3, -1), axis=0)
    pts, wts = torch.from_numpy(pts).cuda(), torch.from_numpy(wts).cuda()
    cells = math.prod(len(b) for b in bases)
    step = max(1, (1 << 25) // cells)
    re = torch.zeros([len(b) for b in bases[::-1]], dtype=torch.float64, device="cuda")
    im = torch.zeros_like(re)
    for i in range(0, len(wts), step):
        x, y, z = (((b[None] + p[:, None]) * dx) ** 2 for b, p in zip(bases, pts[:, i:i + step]))
        R = torch.sqrt(x[:, None, None, :] + y[:, None, :, None] + z[:, :, None, None])
        w = wts[i:i + step, None, None, None] / R
        R *= k
        re += (w * torch.cos(R)).sum(0)
        im -= (w * torch.sin(R)).sum(0)
    return torch.complex(re, im)


def _toeplitz_block(dims, dx, k, n, sing=None):
    """Entries xx xy xz yy yz zz for offsets 0 .. dims - 1 with an n-point rule per direction; sing: the integrals over
    touching squares (same, edge in plane, edge across, vertex in plane, vertex across)."""
    both, (u, w) = _differences(n), _rule(n)
    scale = dx ** 4 / (4 * math.pi)

    def axis_of(t, a, i):
        return t.movedim(2 - a, 0)[i]

    D = []
    for a in range(3):  # squares normal to axis a, planes -1 .. dims apart: second difference over the two sides
        bases = [np.arange(d) for d in dims]
        bases[a] = np.arange(-1, dims[a] + 1)
        rules = [both] * 3
        rules[a] = (np.zeros(1), np.ones(1))
        f = scale * _sum(k, dx, bases, rules)
        if sing is not None:
            g = f.movedim(2 - a, 0)[1]
            g[0, 0], g[0, 1], g[1, 0], g[1, 1] = (sing[i] / (4 * math.pi) for i in (0, 1, 1, 3))
        f = f.movedim(2 - a, 0)
        D.append((2 * f[1:-1] - f[2:] - f[:-2]).movedim(0, 2 - a))

    def cross(p, q):  # observation squares normal to q, source squares normal to p
        c = 3 - p - q
        bases = [np.arange(d) for d in dims]
        bases[q], bases[p] = np.arange(dims[q] + 1), np.arange(-1, dims[p])
        rules = [both] * 3
        rules[q], rules[p] = (-u, w), (u, w)
        f = (scale * _sum(k, dx, bases, rules)).permute(2 - c, 2 - q, 2 - p)
        if sing is not None:
            f[0, :2, :2], f[1, :2, :2] = sing[2] / (4 * math.pi), sing[4] / (4 * math.pi)
        g = -(f[:, 1:, :-1] + f[:, :-1, 1:] - f[:, :-1, :-1] - f[:, 1:, 1:])
        return g.permute(*np.argsort([2 - c, 2 - q, 2 - p]).tolist())

    return torch.stack([D[1] + D[2], cross(0, 1), cross(0, 2), D[0] + D[2], cross(1, 2), D[0] + D[1]])


def _touching(dx, k):
    """Integrals of exp(-j k R)/R over touching squares: relative coordinates, the point singularity taken out by
    mapping each pyramid of a cell to a cube."""
    x, w = _rule(40)

    def green(R):
        return np.exp(-1j * k * R) / R

    def corner(weight, dim):  # a cell with the singular corner at the origin
        total = 0
        s, *t = np.meshgrid(*[x] * dim, indexing="ij")
        ws = np.prod(np.meshgrid(*[w] * dim, indexing="ij"), axis=0)
        for lead in range(dim):
            c = [dx * s * v for v in t]
            c.insert(lead, dx * s)
            total = total + np.sum(ws * dx * (dx * s) ** (dim - 1) * weight(*c) * green(np.sqrt(sum(v * v for v in c))))
        return total

    def away(shift, weight):  # a cell that does not touch it
        c = np.meshgrid(*[dx * (x + m) for m in shift], indexing="ij")
        ws = np.prod(np.meshgrid(*[w * dx] * len(shift), indexing="ij"), axis=0)
        return np.sum(ws * weight(*c) * green(np.sqrt(sum(v * v for v in c))))

    a = dx
    same = 4 * corner(lambda p, q: (a - p) * (a - q), 2)
    edge = 2 * (corner(lambda p, q: p * (a - q), 2) + away((1, 0), lambda p, q: (2 * a - p) * (a - q)))
    edge_across = 2 * corner(lambda p, q, t: a - t, 3)
    vertex = (corner(lambda p, q: p * q, 2) + 2 * away((1, 0), lambda p, q: (2 * a - p) * q)
              + away((1, 1), lambda p, q: (2 * a - p) * (2 * a - q)))
    vertex_across = corner(lambda p, q, t: t, 3) + away((0, 0, 1), lambda p, q, t: 2 * a - t)
    return [complex(v) for v in (same, edge, edge_across, vertex, vertex_across)]


def _circulant(T, odd):
    """FFT of the circulant of T (components x N x M x L); odd[c]: the axes along which component c is odd."""
    Q, N, M, L = T.shape
    C = torch.zeros(Q, 2 * N, 2 * M, 2 * L, dtype=torch.complex128, device="cuda")
    C[:, :N, :M, :L] = T
    sign = [torch.tensor([-1.0 if a in o else 1.0 for o in odd], dtype=torch.float64, device="cuda")[:, None, None, None]
            for a in range(3)]
    C[:, :, :, L + 1:] = sign[0] * C[:, :, :, 1:L].flip(3)
    C[:, :, M + 1:] = sign[1] * C[:, :, 1:M].flip(2)
    C[:, N + 1:] = sign[2] * C[:, 1:N].flip(1)
    for c in range(Q):
        C[c] = torch.fft.fftn(C[c])
    return C


def _spectrum(case):
    """fN, 6 x 2N x 2M x 2L: 4 points per direction, 10 within five voxels, 20 within two."""
    dx, k = case["dx_mm"] * 1e-3, 2 * math.pi * FREQ / C0
    dims = (case["L"], case["M"], case["N"])
    T = _toeplitz_block(dims, dx, k, 4)
    for reach, n, sing in ((5, 10, None), (2, 20, _touching(dx, k))):
        T[:, :reach, :reach, :reach] = _toeplitz_block((reach,) * 3, dx, k, n, sing)
    return _circulant(T, ((), (0, 1), (0, 2), (), (1, 2), ()))


def _spectrum_k(case):
    """fK, 3 x 2N x 2M x 2L: the curl of the Green's function at voxel distances, zero at the voxel itself."""
    dx, k = case["dx_mm"] * 1e-3, 2 * math.pi * FREQ / C0
    x, y, z = (torch.arange(n, dtype=torch.float64, device="cuda") * dx for n in (case["L"], case["M"], case["N"]))
    d = torch.stack(torch.meshgrid(z, y, x, indexing="ij")[::-1])
    R = torch.sqrt((d * d).sum(0))
    R[0, 0, 0] = dx
    g = torch.polar(dx ** 6 / (4 * math.pi * R ** 3), -k * R) * (1 + 1j * k * R)
    return _circulant(-g * d, ((0,), (1,), (2,)))


# ---------------------------------------------------------------------------------------------------------------------
# products and solves in plain torch
# ---------------------------------------------------------------------------------------------------------------------
def _product(fN, J):
    """N J on the grid for J 3 x N x M x L."""
    _, N, M, L = J.shape
    X = [torch.fft.fftn(J[c], s=(2 * N, 2 * M, 2 * L)) for c in range(3)]
    out = []
    for rows in ((0, 1, 2), (1, 3, 4), (2, 4, 5)):
        y = fN[rows[0]] * X[0]
        y += fN[rows[1]] * X[1]
        y += fN[rows[2]] * X[2]
        out.append(torch.fft.ifftn(y)[:N, :M, :L])
    return torch.stack(out)


def _curl(fK, J):
    _, N, M, L = J.shape
    X = [torch.fft.fftn(J[c], s=(2 * N, 2 * M, 2 * L)) for c in range(3)]
    return torch.stack([torch.fft.ifftn(fK[b] * X[c] - fK[c] * X[b])[:N, :M, :L] for b, c in ((2, 1), (0, 2), (1, 0))])


def _system(fN, er, idx, dx):
    """x -> dx^3 x - Mc N x on the DOFs idx (0-based), Mc = (er - 1)/er."""
    V = er.numel()
    Mc = ((er - 1) / er).reshape(-1)[idx % V]
    J = torch.zeros(3, *er.shape, dtype=torch.complex128, device="cuda")

    def apply(x):
        J.view(-1)[idx] = x
        return dx ** 3 * x - Mc * _product(fN, J).reshape(-1)[idx]

    return apply


def _gmres(A, b, tol=1e-11, m=60):
    x, nb = torch.zeros_like(b), torch.linalg.norm(b)
    for _ in range(200):
        r = b - A(x)
        beta = torch.linalg.norm(r)
        if beta <= tol * nb:
            break
        V = torch.empty(m + 1, len(b), dtype=b.dtype, device=b.device)
        H = torch.zeros(m + 1, m, dtype=b.dtype, device=b.device)
        V[0] = r / beta
        for k in range(m):
            w = A(V[k])
            for _ in range(2):
                h = V[:k + 1].conj() @ w
                w = w - h @ V[:k + 1]
                H[:k + 1, k] += h
            H[k + 1, k] = torch.linalg.norm(w)
            V[k + 1] = w / H[k + 1, k]
        e = torch.zeros(m + 1, 1, dtype=b.dtype)
        e[0, 0] = beta.cpu()
        y = torch.linalg.lstsq(H.cpu(), e).solution[:, 0].to(b.device)
        x = x + y @ V[:m]
    return x


def exact(case, seed):
    kind, dx = case["kind"], case["dx_mm"] * 1e-3
    if kind == "operators":
        return None  # the default quadrature of the touching squares has an error of its own that is part of the result
    if kind == "h_field":
        J, H = _currents(case, seed, dx)
        return _columns(H + _curl(_spectrum_k(case), J) / dx ** 3)
    fN = _spectrum(case)
    omega_eps0 = 2 * math.pi * FREQ * EPS0
    if kind == "e_field":
        J, E = _currents(case, seed, 1.0)
        return _columns(E + (_product(fN, J) - dx ** 3 * J) / (1j * omega_eps0 * dx ** 3))
    eps, sig = _body(case, seed)
    er = _permittivity(eps, sig)
    idx = _dofs(er) - 1
    V = er.numel()
    A = _system(fN, er, idx, dx)
    ed = er.reshape(-1)[idx % V]
    if kind in ("mv_AN", "apply"):
        J = _noise(seed, case["nrhs"], len(idx)) if case["nrhs"] > 1 else _noise(seed, len(idx))[None]
        if not case["transp"]:
            out = torch.stack([A(x) for x in J])
        else:  # the Hermitian adjoint: N is symmetric
            g = torch.zeros(3, *er.shape, dtype=torch.complex128, device="cuda")
            out = []
            for x in J:
                g.view(-1)[idx] = ((ed - 1) / ed) * x.conj()
                out.append(dx ** 3 * x - _product(fN, g).reshape(-1)[idx].conj())
            out = torch.stack(out)
        return out[0] if case["nrhs"] == 1 else _columns(out)
    if kind == "inner":
        return {"J": _gmres(A, _noise(seed, len(idx)) * dx ** 3), "flag": None}
    source = dx ** 3 * 1j * omega_eps0 * (ed - 1) / ed
    fields = _excitation(case, seed)
    currents = [_gmres(A, source * E.reshape(-1)[idx]) for E in fields]
    if kind == "gradient":
        J = currents[0]
        E = J / (1j * omega_eps0 * (ed - 1))
        s = sig.reshape(-1)[idx % V]
        lam = _gmres(A, 0.5 * s * E.conj() / ed)
        g = torch.zeros(3, *er.shape, dtype=torch.complex128, device="cuda")
        g.view(-1)[idx] = lam
        q = dx ** 3 * lam - _product(fN, g).reshape(-1)[idx]
        each = (q * E).reshape(3, -1).sum(0)
        d_eps, d_sig = torch.zeros_like(eps), torch.zeros_like(eps)
        at = idx[:len(idx) // 3]
        d_eps.view(-1)[at] = -2 * each.real
        d_sig.view(-1)[at] = -2 * each.imag / omega_eps0 + 0.5 * (E.abs() ** 2).reshape(3, -1).sum(0)
        return {"F": float((0.5 * s * E.abs() ** 2).sum()), "d_eps": _columns(d_eps), "d_sigma": _columns(d_sig),
                "flags": None}
    out = torch.zeros(len(fields), 3, *er.shape, dtype=torch.complex128, device="cuda")
    for o, x in zip(out, currents):
        o.view(-1)[idx] = x
    return {"J": _columns(out if kind == "batch" else out[0]), "flag": None}
