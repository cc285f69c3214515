"""Measured workloads of the library: what its users have it compute, through
its public Python entry points.

Kinds of case
    call          a whole solver call on host data (mesh, options, sources in;
                  currents out): assembly, factorization, refined solve
    assemble      the system matrix into device memory
    factor_solve  factorization of an assembled matrix and a refined solve
    solve         one more refined solve with factors that are kept
    gradient      far-field objective of a SIE-GSTC surface and its gradient
                  with respect to the per-face parameters (torch autograd)
    fields        near fields and the far-field pattern of solved currents

A case is plain values only; prepare() makes its inputs from a seed (a rotated
mesh, a frequency within 1 % of the nominal one, sources, tensors). exact()
gives the same results in 64 bits from torch alone; the float roundings in it
are those of the scalars the formulation defines in float (wavenumber, medium
constants, quadrature rule, extraction threshold, mass scales).
"""

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "sie-gstc-2026_b200"))

import sieb200  # noqa: E402

C0 = 299792458.0
PI = math.pi
C128 = torch.complex128


# ------------------------------------------------------------------- cases
def listed():
    return [
        # A first look at a small scatterer, or one step of a parameter study
        # over small bodies: latency of a whole call.
        dict(name="pec_call_small", kind="call", form="pec", mesh="sphere", n=2, m=0, ka=2.0, rule=5, columns=1,
             method="mixed_ir"),
        # The 1280-face conducting sphere (1920 edges), 7-point rule, one
        # plane wave, ka = 2 pi: the bench's PEC workload as one call.
        dict(name="pec_call", kind="call", form="pec", mesh="sphere", n=8, m=0, ka=2 * PI, rule=5, columns=1,
             method="mixed_ir"),
        # A small surface solved for several excitations at once.
        dict(name="gstc_call_batch", kind="call", form="gstc", mesh="sphere", n=4, m=0, ka=2.5, rule=7, columns=8,
             method="mixed_ir"),
        # The dielectric sphere of the bench (2000 faces, N = 6000) at the
        # solvers' default rule.
        dict(name="pmchwt_assemble", kind="assemble", form="pmchwt", mesh="sphere", n=10, m=0, ka=PI, rule=17),
        # The bench's 2880-face SIE-GSTC sphere (N = 17280), default rule.
        dict(name="gstc_assemble", kind="assemble", form="gstc", mesh="sphere", n=12, m=0, ka=2 * PI, rule=17),
        # Rotated testing (N-Mueller) on an odd mesh with a 13-point rule.
        dict(name="muller_assemble", kind="assemble", form="muller", mesh="spindle", n=17, m=29, ka=3.0, rule=7),
        # The headline solve: mixed-precision factorization and refined solve
        # of the N = 6000 dielectric sphere, one right-hand side.
        dict(name="pmchwt_factor_solve", kind="factor_solve", form="pmchwt", mesh="sphere", n=10, m=0, ka=PI, rule=4,
             columns=1, method="mixed_ir"),
        # The library's FP64 LU at an ordinary size.
        dict(name="fp64_factor_solve", kind="factor_solve", form="pmchwt", mesh="sphere", n=7, m=0, ka=2.5, rule=4,
             columns=3, method="lu_fp64"),
        # 64 plane waves on the N = 17280 SIE-GSTC sphere, as one batch.
        dict(name="gstc_factor_solve_64", kind="factor_solve", form="gstc", mesh="sphere", n=12, m=0, ka=2 * PI,
             rule=4, columns=64, method="mixed_ir"),
        # One more excitation with the factors at hand.
        dict(name="gstc_solve", kind="solve", form="gstc", mesh="sphere", n=8, m=0, ka=4.0, rule=4, columns=1,
             method="mixed_ir"),
        # One step of adjoint synthesis on a circular-arc spindle (N = 20,880).
        dict(name="spindle_gradient", kind="gradient", form="gstc", mesh="spindle", n=30, m=60, ka=3.0, rule=5),
        # A two-plane near-field cut (720 points, partly within a tenth of a
        # wavelength of the surface) and the radiation pattern on the
        # 91 x 181 grid that directivity is integrated on.
        dict(name="fields", kind="fields", form="pmchwt", mesh="sphere", n=10, m=0, ka=PI, rule=17, points=720,
             directions=16471),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "assemble", "assemble", "factor_solve", "solve", "gradient", "fields"])
    mesh = "spindle" if kind == "gradient" else rng.choice(["sphere", "sphere", "spindle"])
    case = dict(kind=kind, form="", mesh=mesh, n=0, m=0, ka=round(rng.uniform(1.5, 6.5), 4), rule=0)

    def size(faces_lo, faces_hi):
        faces = _log_int(rng, faces_lo, faces_hi)
        if mesh == "sphere":
            case["n"] = max(1, int(math.sqrt(faces / 20.0)))
        else:
            case["n"] = max(3, int(math.sqrt(faces / 4.0)))
            case["m"] = max(4, faces // (2 * (case["n"] - 1)))

    if kind == "call":
        case["form"] = rng.choice(["pec", "pmchwt", "gstc"])
        size(60, 1300 if case["form"] == "pec" else 500)
        case["rule"] = rng.choice([3, 4, 5, 7, 8])
        case["columns"] = _log_int(rng, 1, 16) if case["form"] == "gstc" else 1
        case["method"] = rng.choice(["mixed_ir", "mixed_ir", "lu_fp64"])
    elif kind == "assemble":
        case["form"] = rng.choice(["pec", "pmchwt", "gstc", "n_pmchwt", "muller"])
        case["rule"] = rng.choice([3, 4, 5, 6, 7, 9, 12, 14, 17])
        size(100, 2800 if case["rule"] <= 9 else 1500)
    elif kind in ("factor_solve", "solve"):
        case["form"] = rng.choice(["pec", "pmchwt", "gstc"])
        case["method"] = rng.choice(["mixed_ir", "mixed_ir", "lu_fp64"])
        most = {"pec": 2600, "pmchwt": 2600, "gstc": 2000}[case["form"]]
        size(80, most if case["method"] == "mixed_ir" else 800)
        case["rule"] = 4
        case["columns"] = rng.choice([1, 1, 2, _log_int(rng, 3, 64)])
    elif kind == "gradient":
        case["form"] = "gstc"
        size(300, 3300)
        case["rule"] = rng.choice([4, 5, 7])
    else:
        case["form"] = "pmchwt"
        size(300, 2000)
        case["rule"] = rng.choice([4, 5, 8, 17])
        case["points"] = _log_int(rng, 20, 720)
        case["directions"] = _log_int(rng, 181, 16000)
    return case


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=8)
def _unit_mesh(kind, n, m):
    if kind == "sphere":
        return sieb200.geodesic_sphere(1.0, n)
    return sieb200.revolved_spindle(1.0, 60.0, n_axial=n, n_azimuth=m)


def _mesh(case, rng):
    """The case's mesh in a random orientation, radius (half length) 1 m."""
    base = _unit_mesh(case["mesh"], case["n"], case["m"])
    q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
    if np.linalg.det(q) < 0:
        q[:, 0] = -q[:, 0]
    return sieb200.MeshData(np.ascontiguousarray(base.vertices @ q.T), base.faces, base.edges, base.faces_edges)


def _options(case, rng):
    f = case["ka"] * C0 / (2 * PI) * (1.0 + 0.01 * rng.uniform(-1.0, 1.0))
    common = dict(frequency_hz=f, quadrature_rule=case["rule"], solver=case.get("method", "mixed_ir"))
    if case["form"] == "pec":
        return sieb200.PecOptions(**common)
    if case["form"] == "gstc":
        return sieb200.GstcSieOptions(**common)
    formulation = {"pmchwt": "T_PMCHWT", "n_pmchwt": "N_PMCHWT", "muller": "N_Muller"}[case["form"]]
    return sieb200.DielectricOptions(interior=sieb200.IsotropicMedium(4.0, 1.0), formulation=formulation, **common)


def _waves(case, rng):
    """Plane waves from random directions with random transverse polarisations."""
    out = []
    for _ in range(case.get("columns", 1)):
        k = rng.standard_normal(3)
        k /= np.linalg.norm(k)
        e = np.cross(k, rng.standard_normal(3))
        e /= np.linalg.norm(e)
        e -= k * (k @ e)
        out.append(sieb200.PlaneWaveExcitation(electric_amplitude=tuple(e), propagation_direction=tuple(k)))
    return out


def _records(nf, rng):
    """Reciprocal 4x4 maps [[Y, K], [-K^T, Z]] with complex random entries, and
    their inverses: 32 complex values per face."""
    def c(*shape):
        return rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape)
    y, z, k = c(nf, 2, 2), c(nf, 2, 2), 0.5 * c(nf, 2, 2)
    y = (y + y.transpose(0, 2, 1)) / 2 + 2 * np.eye(2)
    z = (z + z.transpose(0, 2, 1)) / 2 + 2 * np.eye(2)
    maps = np.concatenate([np.concatenate([y, k], 2), np.concatenate([-k.transpose(0, 2, 1), z], 2)], 1)
    return np.concatenate([maps.reshape(nf, 16), np.linalg.inv(maps).reshape(nf, 16)], 1)


def _omega_parameters(nf, rng):
    """Lossless omega parameters (B, X, chi) per face, away from singular maps."""
    p = rng.uniform(-2, 2, (3, nf))
    while True:
        bad = np.abs(p[2] ** 2 - p[0] * p[1]) < 1.0
        if not bad.any():
            return p
        p[:, bad] = rng.uniform(-2, 2, (3, int(bad.sum())))


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    mesh = _mesh(case, rng)
    opts = _options(case, rng)
    s = dict(case=case, mesh=mesh, opts=opts, tensors=None, ctx=sieb200.default_context())
    kind = case["kind"]
    if case["form"] == "gstc" and kind != "gradient":
        s["tensors"] = _records(mesh.num_faces, rng)
    if kind != "fields":
        s["waves"] = _waves(case, rng)
    n = _sizes(case)[2]
    if kind == "assemble":
        s["Z"] = torch.empty((n, n), dtype=C128, device="cuda")
    elif kind in ("factor_solve", "solve"):
        s["Z"] = torch.empty((n, n), dtype=C128, device="cuda")  # column-major: Z[c] is column c
        s["ctx"].synchronize()
        torch.cuda.synchronize()
        sieb200.assemble_matrix_device(mesh, opts, s["Z"].data_ptr(), tensors=s["tensors"])
        s["B"] = torch.from_numpy(np.ascontiguousarray(sieb200.assemble_rhs(mesh, opts, s["waves"]).T)).cuda()
        s["X"] = torch.empty_like(s["B"])
        s["stream"] = torch.cuda.ExternalStream(s["ctx"].stream)
        s["solver"] = sieb200.DenseLuSolver(n, case["method"])
        if kind == "solve":
            s["solver"].factorize(s["Z"].data_ptr())
    elif kind == "gradient":
        s["params"] = [torch.tensor(v, device="cuda") for v in _omega_parameters(mesh.num_faces, rng)]
        s["b"] = torch.from_numpy(sieb200.assemble_rhs(mesh, opts, s["waves"])[:, 0].copy()).cuda()
        s["objective"] = sieb200.FarFieldConeObjective(mesh, opts, half_angle_deg=10.0)
    elif kind == "fields":
        ne = mesh.num_edges
        s["J"] = rng.standard_normal(ne) + 1j * rng.standard_normal(ne)
        s["M"] = 377.0 * (rng.standard_normal(ne) + 1j * rng.standard_normal(ne))
        half = (case["points"] + 1) // 2
        t = np.arange(case["points"]) * (2 * PI / half)
        ring = np.stack([np.sin(t), np.zeros_like(t), np.cos(t)], 1)
        ring[half:] = ring[half:, [1, 0, 2]]
        s["points"] = np.ascontiguousarray(ring * np.where(np.arange(case["points"]) % 2, 1.1, 3.0)[:, None])
        th = np.arccos(rng.uniform(-1, 1, case["directions"]))
        ph = rng.uniform(0, 2 * PI, case["directions"])
        s["frames"] = sieb200.spherical_frames(th, ph)
    return s


# -------------------------------------------------------------------- pass
def run(s):
    case, mesh, opts = s["case"], s["mesh"], s["opts"]
    kind = case["kind"]
    if kind == "call":
        if case["form"] == "pec":
            return sieb200.solve_pec_dense(mesh, opts, s["waves"][0]).currents
        if case["form"] == "pmchwt":
            return sieb200.solve_dielectric_dense(mesh, opts, s["waves"][0]).currents
        cases = [sieb200.GstcExcitationCase(exterior=w) for w in s["waves"]]
        return [r.currents for r in sieb200.solve_gstc_dense_batch(mesh, s["tensors"], opts, cases)]
    if kind == "assemble":
        sieb200.assemble_matrix_device(mesh, opts, s["Z"].data_ptr(), tensors=s["tensors"])
        return s["Z"]
    if kind in ("factor_solve", "solve"):
        with torch.cuda.stream(s["stream"]):
            s["X"].copy_(s["B"])
        if kind == "factor_solve":
            s["solver"].factorize(s["Z"].data_ptr())
        s["solver"].solve(s["X"].data_ptr(), nrhs=case["columns"])
        return s["X"]
    if kind == "gradient":
        params = [p.detach().requires_grad_(True) for p in s["params"]]
        x = sieb200.gstc_solve(sieb200.omega_records(*params), s["b"], mesh, opts, tolerance=1e-12)
        objective = s["objective"](x)
        objective.backward()
        return [objective.detach(), x.detach()] + [p.grad for p in params]
    e, h = sieb200.evaluate_surface_integral_fields(mesh, s["J"], s["M"], s["points"], opts.frequency_hz,
                                                    quadrature_rule=case["rule"])
    f = sieb200.far_field(mesh, s["J"], s["M"], 2 * PI * opts.frequency_hz / C0, 376.730313668, *s["frames"])
    return [e, h, *f]


# -------------------------------------------------------------------- work
def _sizes(case):
    if case["mesh"] == "sphere":
        faces = 20 * case["n"] ** 2
    else:
        faces = 2 * case["m"] * (case["n"] - 1)
    edges = 3 * faces // 2
    return faces, edges, {"pec": 1, "gstc": 4}.get(case["form"], 2) * edges


def _points_of(rule):
    return [1, 3, 4, 6, 7, 12, 13, 16, 19, 25, 27, 33, 37, 42, 48, 52, 61, 70, 73, 79][rule - 1]


def work(case):
    """One pass: operands read once, results written once; the additions and
    multiplications of the method (a Green kernel value with its share of the
    moments counted 50, LU 8/3 n^3, 8 n^2 per solved column and product)."""
    faces, edges, n = _sizes(case)
    q = _points_of(case["rule"])
    media = 2 if case["form"] in ("pmchwt", "n_pmchwt", "muller") else 1
    quadrature = 50.0 * media * faces * (faces + 1) / 2 * q * q
    matrix = 16.0 * n * n
    cols = case.get("columns", 1)
    lu = 8.0 / 3.0 * n ** 3
    column = 2 * 8.0 * n * n
    records = 512.0 * faces if case["form"] == "gstc" else 0.0
    kind = case["kind"]
    if kind == "call":
        return {"bytes": 2 * matrix + 16.0 * n * cols + records, "flops": quadrature + lu + cols * column}
    if kind == "assemble":
        return {"bytes": matrix + records + 72.0 * edges, "flops": quadrature}
    if kind == "factor_solve":
        return {"bytes": matrix + 32.0 * n * cols, "flops": lu + cols * column}
    if kind == "solve":
        return {"bytes": matrix + 32.0 * n * cols, "flops": cols * column}
    if kind == "gradient":
        return {"bytes": 2 * matrix + 2 * records + 48.0 * n, "flops": quadrature + lu + 2 * column}
    return {"bytes": 32.0 * edges + 216.0 * case["points"] + 112.0 * case["directions"],
            "flops": 60.0 * case["points"] * faces * q + 56.0 * case["directions"] * faces * 7}


# --------------------------------------------------- the same in 64 bits
def _f32(x):
    return float(np.float32(x))


def _f32t(t):
    return t.to(torch.float32).to(torch.float64)


def _rule(rule):
    """Points and weights of the Dunavant rule (single precision by definition)."""
    q = _points_of(rule)
    pts, w = np.zeros(2 * q, np.float32), np.zeros(q, np.float32)
    sieb200.lib().sieb200_quadrature_rule(rule, pts.ctypes.data, w.ctypes.data)
    return torch.from_numpy(pts.reshape(q, 2).astype(np.float64)).cuda(), torch.from_numpy(w.astype(np.float64)).cuda()


class _Faces:
    """Geometry of every face on the device: vertices, centroid, free vertices
    of the local edges (a, a + 1), signed edge lengths, area, rule points."""

    def __init__(self, mesh, rule):
        f = torch.from_numpy(mesh.faces.astype(np.int64)).cuda()
        v = torch.from_numpy(np.asarray(mesh.vertices)).cuda()[f]
        self.v, self.fe, self.ne = v, torch.from_numpy(mesh.faces_edges.astype(np.int64)).cuda(), mesh.num_edges
        self.c = v.mean(1)
        self.fv = v[:, [2, 0, 1]]
        nxt = [1, 2, 0]
        sign = torch.where(f > f[:, nxt], 1.0, -1.0).to(torch.float64)
        self.len = sign * (v[:, nxt] - v).norm(dim=2)
        self.normal = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
        self.area = 0.5 * self.normal.norm(dim=1)
        self.normal = self.normal / self.normal.norm(dim=1, keepdim=True)
        self.pts, self.w = _rule(rule)
        xi, eta = self.pts[:, 0], self.pts[:, 1]
        bary = torch.stack([1.0 - xi - eta, xi, eta], 1)
        self.r = torch.einsum("qa,fac->fqc", bary, v)
        self.count, self.q = v.shape[0], self.w.numel()


def _scalars(case, opts):
    omega = 2.0 * PI * opts.frequency_hz
    mu0, ep0 = opts.vacuum_permeability, opts.vacuum_permittivity
    out = dict(omega=omega, mu0=_f32(mu0), ep0=_f32(ep0), omf=_f32(omega))
    media = [opts.exterior] if case["form"] == "pec" else [opts.interior, opts.exterior]
    out["k"] = [_f32(omega * math.sqrt(m.relative_permeability * mu0 * m.relative_permittivity * ep0)) for m in media]
    out["mu"] = [_f32(_f32(m.relative_permeability) * out["mu0"]) for m in media]
    out["ep"] = [_f32(_f32(m.relative_permittivity) * out["ep0"]) for m in media]
    out["eta"] = float(np.sqrt(np.float32(out["mu0"]) / np.float32(out["ep0"])))
    out["threshold"] = _f32(opts.singularity_threshold_lambda0 / (math.sqrt(mu0 * ep0) * opts.frequency_hz))
    return out


def _potentials(r, tri, normal):
    """Integrals over triangles (Wilton et al., IEEE T-AP 32, 1984) seen from
    points r (..., 3): 1/R, (r' - r_pi)/R, 1/R^3, (r' - r_pi)/R^3 and the
    projection r_pi of r into the plane."""
    d = ((r - tri[..., 0, :]) * normal).sum(-1)
    r_pi = r - normal * d[..., None]
    ad = d.abs()
    i1, i3 = torch.zeros_like(d), torch.zeros_like(d)
    v1, v3 = torch.zeros_like(r), torch.zeros_like(r)
    for e in range(3):
        a, b = tri[..., e, :], tri[..., (e + 1) % 3, :]
        t = (b - a) / (b - a).norm(dim=-1, keepdim=True)
        u = torch.linalg.cross(t, normal.expand_as(t))
        s = ((a - r_pi) * u).sum(-1)
        p0 = s.abs()
        lp, lm = ((b - r_pi) * t).sum(-1), ((a - r_pi) * t).sum(-1)
        r0 = p0 * p0 + ad * ad
        rp, rm = (r0 + lp * lp).sqrt(), (r0 + lm * lm).sqrt()
        log = torch.where(lp + lm > 0, ((rp + lp) / (rm + lm)).log(), ((rm - lm) / (rp - lp)).log())
        beta = torch.atan2(p0 * lp, r0 + ad * rp) - torch.atan2(p0 * lm, r0 + ad * rm)
        side = torch.where(s >= 0, 1.0, -1.0)
        i1 = i1 + torch.where(p0 > 1e-9, side * (p0 * log - ad * beta), torch.zeros_like(p0))
        v1 = v1 + 0.5 * u * (r0 * log + lp * rp - lm * rm)[..., None]
        flat = -(lp / (p0 * (p0 * p0 + lp * lp).sqrt()) - lm / (p0 * (p0 * p0 + lm * lm).sqrt()))
        flat = torch.where(p0 > 1e-9, flat, torch.zeros_like(p0))
        i3 = i3 + side * torch.where(ad > 1e-6, beta / ad, flat)
        v3 = v3 - u * log[..., None]
    return i1, v1, i3, v3, r_pi


def _kernels(dist, k, extracted):
    """G and g (gradient factor) of exp(-j k R)/(4 pi R), or the same without
    the terms that are integrated in closed form."""
    if not extracted:
        phase = torch.polar(torch.ones_like(dist), -k * dist)
        green = phase / (4 * PI * dist)
        return green, green * torch.complex(1.0 / dist, torch.full_like(dist, k)) / dist
    c, s = torch.cos(k * dist), torch.sin(k * dist)
    zero = dist < 1e-9
    safe = torch.where(zero, torch.ones_like(dist), dist)
    green = torch.complex((c - 1.0) / safe, -s / safe) / (4 * PI)
    i2, i3 = safe ** -2, safe ** -3
    g = (torch.complex(i3, k * i2) * torch.complex(c, -s) - (i3 + 0.5 * k * k / safe)) / (4 * PI)
    green = torch.where(zero, torch.full_like(green, complex(0.0, -k / (4 * PI))), green)
    return green, torch.where(zero, torch.zeros_like(g), g)


def _expand(F, mg, mt, m, n, k):
    """3 x 3 blocks TL and TK of face pairs from the kernel's moments
    mg, mt [..., 4, 4] (1, x, y, z about the centroids, test then source)."""
    a, b = (F.fv[m] - F.c[m][:, None]).to(C128), (F.fv[n] - F.c[n][:, None]).to(C128)
    scale = F.len[m][:, :, None] * F.len[n][:, None, :]

    def second(mom):  # [pair, j, i, 3, 3]: sum of K (p - A_j)_c (q - B_i)_d
        return (mom[:, None, None, 1:, 1:] - mom[:, None, None, 1:, :1] * b[:, None, :, None, :]
                - mom[:, None, None, :1, 1:] * a[:, :, None, :, None]
                + mom[:, None, None, :1, :1] * a[:, :, None, :, None] * b[:, None, :, None, :])
    tl = scale * (0.25 * second(mg).diagonal(dim1=-2, dim2=-1).sum(-1) - mg[:, None, None, 0, 0] / k ** 2)
    w = second(mt)
    cross = torch.stack([w[..., 1, 2] - w[..., 2, 1], w[..., 2, 0] - w[..., 0, 2], w[..., 0, 1] - w[..., 1, 0]], -1)
    d = (F.fv[m][:, :, None] - F.fv[n][:, None, :]).to(C128)
    tk = 0.25 * scale * (cross * d).sum(-1)
    return tl, torch.where((m == n)[:, None, None], torch.zeros_like(tk), tk)


def _calderon(F, k, threshold, with_tk):
    """TL and TK of one wavenumber between all edges (E x E)."""
    nf, q = F.count, F.q
    local = F.r - F.c[:, None]
    mono = (torch.cat([torch.ones_like(local[..., :1]), local], 2) * F.w[None, :, None]).to(C128)
    near = _f32t((F.c[:, None] - F.c[None]).norm(dim=2)) < threshold
    blocks = [torch.zeros((nf, nf, 3, 3), dtype=C128, device="cuda") for _ in range(2 if with_tk else 1)]
    flat_r = F.r.reshape(nf * q, 3)
    step = max(1, int(6e7 // (nf * q * q)))
    every = torch.arange(nf, device="cuda")
    for m0 in range(0, nf, step):
        m = every[m0:m0 + step]
        p = F.r[m].reshape(-1, 3)
        dist = sum((p[:, None, c] - flat_r[None, :, c]) ** 2 for c in range(3)).sqrt()
        green, g = _kernels(torch.where(dist < 1e-12, torch.ones_like(dist), dist), k, False)
        mom = []
        for kernel in ((green, g) if with_tk else (green,)):
            over_q = torch.bmm(kernel.view(-1, nf, q).permute(1, 0, 2), mono).view(nf, len(m), q, 4)
            mom.append(torch.einsum("nmqb,mqa->mnab", over_q, mono[m]).reshape(-1, 4, 4))
        del dist, green, g
        mi, ni = m.repeat_interleave(nf), every.repeat(len(m))
        got = _expand(F, mom[0], mom[-1], mi, ni, k)
        for o, x in zip(blocks, got):
            o[m] = x.view(len(m), nf, 3, 3)
    pairs = near.nonzero()
    step = max(1, int(3e7 // (q * q)))
    for s in range(0, len(pairs), step):
        m, n = pairs[s:s + step, 0], pairs[s:s + step, 1]
        dist = (F.r[m][:, :, None] - F.r[n][:, None, :]).norm(dim=3)
        mom = [torch.einsum("xpq,xpa,xqb->xab", kk, mono[m], mono[n]) for kk in _kernels(dist, k, True)]
        tl, tk = _expand(F, mom[0], mom[1], m, n, k)
        r, fv = F.r[m], F.fv[n]
        i1, v1, i3, v3, r_pi = _potentials(r, F.v[n][:, None], F.normal[n][:, None])
        scale = F.len[m][:, :, None] * F.len[n][:, None, :] / (4 * PI * F.area[n])[:, None, None]
        rho = r[:, :, None] - F.fv[m][:, None]                       # [pair, p, j, 3]
        arm = r_pi[:, :, None] - fv[:, None]                         # [pair, p, i, 3]
        psi = v1[:, :, None] + arm * i1[..., None, None]
        stat = 0.25 * torch.einsum("xpjc,xpic->xpji", rho, psi) - (i1 / k ** 2)[:, :, None, None]
        tl = tl + scale * torch.einsum("xpji,p->xji", stat, F.w)
        comb = v3[:, :, None] + arm * i3[..., None, None] + psi * _f32(_f32(k * k) * 0.5)
        ups = -torch.linalg.cross(r[:, :, None] - fv[:, None], comb)
        curl = 0.25 * scale * torch.einsum("xpjc,xpic,p->xji", rho, ups, F.w)
        tk = tk + torch.where((m == n)[:, None, None], torch.zeros_like(curl), curl)
        for o, x in zip(blocks, (tl, tk)):
            o[m, n] = x
    return [_to_edges(F, b.permute(0, 2, 1, 3).reshape(3 * nf, 3 * nf)) for b in blocks]


def _to_edges(F, block):
    ids = F.fe.reshape(-1)
    rows = torch.zeros((F.ne, block.shape[1]), dtype=C128, device="cuda").index_add(0, ids, block)
    return torch.zeros((F.ne, F.ne), dtype=C128, device="cuda").index_add(1, ids, rows)


def _mass(F, records, sc):
    """Jump-condition blocks between all edges, 4 x 4 regions (linear in records)."""
    e1 = F.v[:, 1] - F.v[:, 0]
    u = e1 / e1.norm(dim=1, keepdim=True)
    w = torch.linalg.cross(F.normal, u)
    frame = torch.stack([u, w], 1).to(C128)                          # [F, 2, 3]
    y = records.view(-1, 2, 2, 2, 2, 2).permute(0, 1, 2, 4, 3, 5)    # [F, Y/Z, block row, block col, 2, 2]
    t = torch.einsum("fszxab,fac,fbd->fszxcd", y, frame, frame)
    n = _f32t(F.normal)
    zero = torch.zeros_like(n[:, 0])
    cross = torch.stack([zero, -n[:, 2], n[:, 1], n[:, 2], zero, -n[:, 0], -n[:, 1], n[:, 0], zero],
                        1).view(-1, 3, 3).to(C128)
    perp = -torch.einsum("fac,fzxcd,fdb->fzxab", cross, t[:, 0], cross)
    t = torch.stack([perp, t[:, 1]], 1)
    rho = (F.r[:, :, None] - F.fv[:, None]).to(C128)                 # [F, q, 3, 3]
    sl = _f32t(_f32t(1.0 / (4.0 * _f32t(F.area)))[:, None] * _f32t(F.len))
    scale = _f32t(sl[:, :, None] * _f32t(F.len)[:, None, :])
    m = torch.einsum("fqjc,fszxcd,fqid,q->fszxji", rho, t, rho, F.w.to(C128)) * scale[:, None, None, None]
    yy, zz = 0.125 * m[:, 0], 0.5 * m[:, 1]
    (yee, yem), (yme, ymm) = [[yy[:, a, b] for b in range(2)] for a in range(2)]
    (zee, zem), (zme, zmm) = [[zz[:, a, b] for b in range(2)] for a in range(2)]
    e, e2 = sc["eta"], _f32(sc["eta"] * sc["eta"])
    ap, am, bp, bm = zee + ymm, zee - ymm, e * (zem + yme), e * (zem - yme)
    cp, cm, dp, dm = e * (zme + yem), e * (zme - yem), e2 * (zmm + yee), e2 * (zmm - yee)
    return [[ap, bm, am, bp], [cm, dp, cp, dm], [am, bp, ap, bm], [cp, dm, cm, dp]]


def _add_mass(F, Z, records, sc):
    """Z (row-major N x N) plus the jump-condition blocks."""
    blocks = _mass(F, records, sc)
    rows = F.fe[:, :, None].expand(-1, 3, 3).reshape(-1)
    cols = F.fe[:, None, :].expand(-1, 3, 3).reshape(-1)
    idx = torch.cat([(rows + r * F.ne) * Z.shape[1] + cols + c * F.ne for r in range(4) for c in range(4)])
    val = torch.cat([blocks[r][c].reshape(-1) for r in range(4) for c in range(4)])
    return Z.reshape(-1).index_add(0, idx, val).view(Z.shape)


def _matrix(case, mesh, opts, tensors, F=None):
    """The system matrix, row-major (Z[i, j])."""
    F = F or _Faces(mesh, case["rule"])
    sc = _scalars(case, opts)
    with_tk = case["form"] != "pec"
    by_k = {k: _calderon(F, k, sc["threshold"], with_tk) for k in dict.fromkeys(sc["k"])}
    if case["form"] == "pec":
        return 1j * float(np.float32(sc["omf"]) * np.float32(opts.exterior.relative_permeability)
                          * np.float32(sc["mu0"])) * by_k[sc["k"][0]][0]
    (l1, k1), (l2, k2) = by_k[sc["k"][0]], by_k[sc["k"][1]]
    om, eta = sc["omf"], sc["eta"]
    ne = F.ne
    if case["form"] == "pmchwt":
        jm = eta * (k1 + k2)
        jj = 1j * om * (sc["mu"][0] * l1 + sc["mu"][1] * l2)
        mm = 1j * om * _f32(eta * eta) * (sc["ep"][0] * l1 + sc["ep"][1] * l2)
        return torch.cat([torch.cat([jj, jm], 1), torch.cat([-jm, mm], 1)], 0)
    Z = torch.zeros((4 * ne, 4 * ne), dtype=C128, device="cuda")
    for r, (tl, tk) in enumerate(((l1, k1), (l2, k2))):
        a, b, c = 2 * r * ne, (2 * r + 1) * ne, (2 * r + 2) * ne
        Z[a:b, a:b] = 1j * om * sc["mu"][r] * tl
        Z[a:b, b:c] = eta * tk
        Z[b:c, a:b] = -eta * tk
        Z[b:c, b:c] = 1j * om * eta * eta * sc["ep"][r] * tl
    return _add_mass(F, Z, torch.as_tensor(tensors, dtype=C128).cuda(), sc)


def _rhs(case, mesh, opts, waves):
    F = _Faces(mesh, case["rule"])
    mu, ep = opts.vacuum_permeability, opts.vacuum_permittivity
    k, eta = 2 * PI * opts.frequency_hz * math.sqrt(mu * ep), math.sqrt(mu / ep)
    rho = (F.r[:, :, None] - F.fv[:, None]) * F.w[None, :, None, None] * (0.5 * _f32t(F.len))[:, None, :, None]
    cols = []
    for wave in waves:
        d = np.array(wave.propagation_direction)
        d = d / np.linalg.norm(d)
        e = np.array(wave.electric_amplitude)
        phase = torch.polar(torch.ones_like(F.r[..., 0]), -k * (F.r @ torch.from_numpy(d).cuda()))
        tested = []
        for vec in (e, np.cross(d, e) / eta):
            val = torch.einsum("fqjc,c,fq->fj", rho.to(C128), torch.from_numpy(vec).to(C128).cuda(), phase)
            tested.append(torch.zeros(F.ne, dtype=C128, device="cuda").index_add(0, F.fe.reshape(-1), val.reshape(-1)))
        ve, vh = tested
        if case["form"] == "pec":
            cols.append(ve)
        elif case["form"] == "pmchwt":
            cols.append(torch.cat([ve, eta * vh]))
        else:
            eta0 = math.sqrt(_f32(mu) / _f32(ep))
            cols.append(torch.cat([torch.zeros_like(ve), torch.zeros_like(ve), ve, eta0 * vh]))
    return torch.stack(cols, 1)


def _exact_fields(case, s):
    mesh, opts = s["mesh"], s["opts"]
    F = _Faces(mesh, case["rule"])
    mu, ep = sieb200.farfield.VACUUM_PERMEABILITY, sieb200.farfield.VACUUM_PERMITTIVITY
    omega = 2 * PI * opts.frequency_hz
    k = _f32(omega * math.sqrt(mu * ep))
    inv_k2 = float(np.float32(1) / (np.float32(k) * np.float32(k)))
    threshold = float(np.float32(0.1) * np.float32(2 * float(np.float32(PI)) / (omega * math.sqrt(mu * ep))))
    obs = torch.from_numpy(s["points"]).cuda()
    jc, mc = (torch.from_numpy(s[x]).cuda()[F.fe] for x in "JM")     # [F, 3]
    near = _f32t((obs[:, None] - F.c[None]).norm(dim=2)) < threshold
    E = torch.zeros((len(obs), 3), dtype=C128, device="cuda")
    H = torch.zeros_like(E)
    rho = F.r[:, :, None] - F.fv[:, None]                            # [F, q, i, 3]
    el = _f32t(F.len)
    for p in range(len(obs)):
        R = obs[p] - F.r
        dist = R.norm(dim=2)
        gs, ks = _kernels(dist, k, False)
        gr, kr = _kernels(dist, k, True)
        G, g = torch.where(near[p][:, None], gr, gs), torch.where(near[p][:, None], kr, ks)
        # the gradient is -g R for the outgoing kernel; L and K use +g R
        gv = g[..., None] * R
        wl = F.w[None, :, None, None] * el[:, None, :, None]
        L = ((0.5 * G[..., None, None] * rho - inv_k2 * gv[:, :, None]) * wl).sum(1)
        K = (0.5 * torch.linalg.cross(rho.to(C128), gv[:, :, None].expand(-1, -1, 3, -1)) * wl).sum(1)
        idx = near[p].nonzero()[:, 0]
        if len(idx):
            r = obs[p].expand(len(idx), 3)
            i1, v1, i3, v3, r_pi = _potentials(r, F.v[idx], F.normal[idx])
            arm, rf = r_pi[:, None] - F.fv[idx], r[:, None] - F.fv[idx]
            psi = v1[:, None] + arm * i1[:, None, None]
            phi3 = v3[:, None] + arm * i3[:, None, None]
            lin = psi - 0.5 * rf * i1[:, None, None] + (phi3 - rf * i3[:, None, None]) * inv_k2
            ups = -torch.linalg.cross(rf, phi3 + psi * _f32(_f32(k * k) * 0.5))
            base = _f32t(1.0 / _f32t(_f32t(8.0 * torch.tensor(_f32(PI))) * _f32t(F.area[idx])))
            ls = _f32t(el[idx] * base[:, None])[..., None]
            L[idx] += 2.0 * lin * ls
            K[idx] += ups * ls
        E[p] = (1j * omega * mu * jc[..., None] * L + mc[..., None] * K).sum((0, 1))
        H[p] = (-jc[..., None] * K + 1j * omega * ep * mc[..., None] * L).sum((0, 1))
    return [E, H, *_far(mesh, s["J"], s["M"], 2 * PI * opts.frequency_hz / C0, 376.730313668, s["frames"])]


def _far_samples(mesh):
    """Points of the 7-point rule and, per point, the RWG values of the face's
    three local edges (area integrals)."""
    F = _Faces(mesh, 1)
    s15 = math.sqrt(15.0)
    a, b = (6 - s15) / 21, (6 + s15) / 21
    nodes = [(1 / 3, 1 / 3)] + [t for x in (a, b) for t in ((x, x), (1 - 2 * x, x), (x, 1 - 2 * x))]
    w = torch.tensor([0.225] + [(155 - s15) / 1200] * 3 + [(155 + s15) / 1200] * 3, dtype=torch.float64).cuda()
    bary = torch.tensor([(1 - x - y, x, y) for x, y in nodes], dtype=torch.float64).cuda()
    r = torch.einsum("qa,fac->fqc", bary, F.v)
    rho = (r[:, :, None] - F.fv[:, None]) * w[None, :, None, None] * (0.5 * F.len)[:, None, :, None]
    return F, r, rho


def _far(mesh, j, m, k0, eta0, frames):
    F, r, rho = _far_samples(mesh)
    rh, th, ph = (torch.from_numpy(x).cuda() for x in frames)
    cur = [torch.einsum("fqic,fi->fqc", rho.to(C128), torch.as_tensor(x).cuda()[F.fe]).reshape(-1, 3) for x in (j, m)]
    vec = [[], []]
    for a in range(0, len(rh), 2048):
        phase = torch.polar(torch.ones((), dtype=torch.float64, device="cuda"), k0 * (rh[a:a + 2048] @ r.reshape(-1, 3).T))
        for x, c in zip(vec, cur):
            x.append(phase @ c)
    n, l = (torch.cat(x) for x in vec)
    nt, np_, lt, lp = (n * th).sum(1), (n * ph).sum(1), (l * th).sum(1), (l * ph).sum(1)
    c = -1j * k0 / (4 * PI)
    ft, fp = c * (eta0 * nt + lp), c * (eta0 * np_ - lt)
    return ft, fp, (ft.abs() ** 2 + fp.abs() ** 2) / (2 * eta0)


def _exact_gradient(case, s):
    mesh, opts = s["mesh"], s["opts"]
    F, sc = _Faces(mesh, case["rule"]), _scalars(case, opts)
    zero = np.zeros((mesh.num_faces, 32), dtype=np.complex128)
    Z = _matrix(case, mesh, opts, zero, F)
    params = [p.detach().clone().requires_grad_(True) for p in s["params"]]
    B, X, chi = params
    z = torch.zeros_like(B)
    jb, jx, c, o = torch.complex(z, B), torch.complex(z, X), torch.complex(chi, z), torch.complex(z, z)
    maps = torch.stack([jb, o, o, c, o, jb, -c, o, o, c, jx, o, -c, o, o, jx], 1).view(-1, 4, 4)
    records = torch.cat([maps.reshape(-1, 16), torch.linalg.inv(maps).reshape(-1, 16)], 1)
    b = s["b"]
    blocks = _mass(F, records, sc)
    with torch.no_grad():
        lu = torch.linalg.lu_factor(_add_mass(F, Z, records, sc))
        del Z
        x = torch.linalg.lu_solve(*lu, b[:, None])[:, 0]
    x.requires_grad_(True)
    eta0 = math.sqrt(opts.vacuum_permeability / opts.vacuum_permittivity)
    k0, ne = 2 * PI * opts.frequency_hz / C0, F.ne
    # Gauss-Legendre in cos(theta) x uniform phi over the 10 degree cone about +z
    c0 = math.cos(math.radians(10.0))
    node, wt = np.polynomial.legendre.leggauss(8)
    t, p = np.meshgrid(np.arccos(0.5 * (1 - c0) * node + 0.5 * (1 + c0)), (np.arange(16) + 0.5) * (2 * PI / 16),
                       indexing="ij")
    wt = torch.from_numpy(np.repeat(0.5 * (1 - c0) * wt * (2 * PI / 16), 16)).cuda()
    t, p = t.ravel(), p.ravel()
    frames = (np.stack([np.sin(t) * np.cos(p), np.sin(t) * np.sin(p), np.cos(t)], 1),
              np.stack([np.cos(t) * np.cos(p), np.cos(t) * np.sin(p), -np.sin(t)], 1),
              np.stack([-np.sin(p), np.cos(p), np.zeros_like(p)], 1))
    objective = (wt * _far(mesh, x[2 * ne:3 * ne], x[3 * ne:] * eta0, k0, eta0, frames)[2]).sum()
    objective.backward()
    lam = torch.linalg.lu_solve(*lu, x.grad[:, None], adjoint=True)[:, 0]
    # dL = -Re(lambda^H dZ x), and only the jump-condition blocks depend on the records
    xs, ls = x.detach().view(4, ne)[:, F.fe], lam.view(4, ne)[:, F.fe].conj()
    form = sum((torch.einsum("fj,fji,fi->", ls[r], blocks[r][q], xs[q])) for r in range(4) for q in range(4))
    grads = torch.autograd.grad(-form.real, params)
    return [objective.detach(), x.detach(), *grads]


def exact(case, seed):
    if case["form"] in ("muller", "n_pmchwt"):
        return None
    s = prepare(case, seed)
    torch.cuda.synchronize()
    mesh, opts, kind = s["mesh"], s["opts"], case["kind"]
    if kind == "fields":
        return _exact_fields(case, s)
    if kind == "gradient":
        return _exact_gradient(case, s)
    if kind == "assemble":
        del s["Z"]
        return _matrix(case, mesh, opts, s["tensors"]).T.contiguous()
    if kind in ("factor_solve", "solve"):
        return torch.linalg.solve(s["Z"].T, s["B"].T).T.contiguous()
    x = torch.linalg.solve(_matrix(case, mesh, opts, s["tensors"]), _rhs(case, mesh, opts, s["waves"]))
    eta0 = math.sqrt(opts.vacuum_permeability / opts.vacuum_permittivity)
    for odd in range(1, x.shape[0] // mesh.num_edges, 2):
        x[odd * mesh.num_edges:(odd + 1) * mesh.num_edges] *= eta0
    cols = [c.contiguous().cpu().numpy() for c in x.T]
    return cols if case["form"] == "gstc" else cols[0]
