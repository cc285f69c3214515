"""The regular quadrature pass: lane splits, pair layouts, slabs and phases at
the edges of its dispatch, and the far-field and surface-field sums that share
its phase factors, against the oracle."""

import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

C0 = 299792458.0


def _mesh(name):
    import sieb200
    return {"ico20": lambda: sieb200.icosphere(0.5, 0), "geo180": lambda: sieb200.geodesic_sphere(0.5, 3),
            "geo500": lambda: sieb200.geodesic_sphere(0.5, 5),
            "spindle90": lambda: sieb200.revolved_spindle(0.6, 60.0, n_axial=6, n_azimuth=9)}[name]()


def _options(form, rule, freq, eps_in, eps_out=1.0):
    import sieb200
    medium = sieb200.IsotropicMedium
    if form in ("pec", "n_mfie"):
        name, variant = ("TEfie", 0) if form == "pec" else ("NMfie", 2)
        return sieb200.PecOptions(frequency_hz=freq, quadrature_rule=rule, formulation=name), 0, variant
    if form == "gstc":
        return sieb200.GstcSieOptions(frequency_hz=freq, quadrature_rule=rule, interior=medium(eps_in, 1.0),
                                      exterior=medium(eps_out, 1.0)), 2, 0
    name, variant = {"pmchwt": ("T_PMCHWT", 0), "n_pmchwt": ("N_PMCHWT", 1), "muller": ("N_Muller", 2)}[form]
    return sieb200.DielectricOptions(frequency_hz=freq, quadrature_rule=rule, formulation=name,
                                     interior=medium(eps_in, 1.0), exterior=medium(eps_out, 1.0)), 1, variant


def _oracle(mesh, kind, variant, rule, opts, eps_in, eps_out=1.0, tensors=None):
    eps = (eps_in, eps_out) if kind else (1.0, 1.0)
    s = O.kernel_scalars(kind, opts.frequency_hz, eps_r=eps)
    return O.assemble(O.oracle(), kind, mesh, rule, s, tensors=tensors, variant=variant)


def _tensors(nf):
    rng = np.random.default_rng(nf)
    t = rng.standard_normal((nf, 32)) + 1j * rng.standard_normal((nf, 32))
    return np.ascontiguousarray(t)


@pytest.mark.parametrize("form", ["pec", "pmchwt", "gstc", "n_pmchwt", "muller"])
@pytest.mark.parametrize("rule", [1, 2, 5, 8, 20])
@pytest.mark.parametrize("name", ["ico20", "geo180", "spindle90"])
@pytest.mark.parametrize("same", [False, True])
def test_assembly_layouts(form, rule, name, same, gpu_ctx):
    """Every pair layout (one wavenumber, two, two equal, TK summed) with 1 to
    79 rule points, and so with 1 to 32 lanes per pair."""
    import sieb200
    mesh = _mesh(name)
    eps_in = 1.0 if same else 2.56
    opts, kind, variant = _options(form, rule, 0.6 * C0, eps_in)
    t = _tensors(mesh.num_faces) if kind == 2 else None
    Z = sieb200.assemble_matrix(mesh, opts, tensors=t, ctx=gpu_ctx)
    Zo = _oracle(mesh, kind, variant, rule, opts, eps_in, tensors=t)
    assert np.abs(Z - Zo).max() <= 1e-12 * np.abs(Zo).max()


ULP = 2.0 ** -53  # relative rounding of one FP64 operation


@pytest.mark.parametrize("k_extent", [9.0e6, 4.0e7])
def test_assembly_large_phase(k_extent, gpu_ctx):
    """Phases up to the step number's limit, and past it (sincos). The bound
    is the rounding of R (some four operations here, three in the oracle) and of the
    oracle's k R, 8 in all, times the largest phase, and twice that."""
    import sieb200
    mesh = _mesh("ico20")
    extent = np.ptp(np.asarray(mesh.vertices), axis=0)
    k = k_extent / extent.sum()
    opts, kind, variant = _options("pec", 5, k * C0 / (2 * math.pi), 1.0)
    Z = sieb200.assemble_matrix(mesh, opts, ctx=gpu_ctx)
    Zo = _oracle(mesh, kind, variant, 5, opts, 1.0)
    assert np.abs(Z - Zo).max() <= 16 * ULP * k * np.linalg.norm(extent) * np.abs(Zo).max()


# Face-pair values of 16 bytes per edge pair; the workspace holds 8 GB of them.
_SLABS = {"pec": (20, 1, 1.0), "pmchwt": (15, 3, 4.0), "gstc": (17, 2, 1.0), "gstc_two_media": (14, 4, 2.56),
          "n_pmchwt": (14, 4, 4.0), "muller": (14, 4, 4.0), "n_mfie": (20, 1, 1.0)}


@pytest.mark.parametrize("form", list(_SLABS))
def test_assembly_two_slabs(form, gpu_ctx):
    """Two slabs of test faces (with RWG testing pairs inside a slab are evaluated
    once and mirrored, pairs across slabs twice; the second slab is added
    to Z): rows of faces around the slab boundary and elsewhere, for every pair layout."""
    import torch
    import sieb200
    level, values, eps_in = _SLABS[form]
    mesh = sieb200.geodesic_sphere(1.0, level)
    nf = mesh.num_faces
    slab = (8 << 30) // (16 * 9 * values * nf)
    assert nf / 2 < slab < nf
    opts, kind, variant = _options("gstc" if form.startswith("gstc") else form, 1, 1.5 * C0, eps_in)
    t = _tensors(nf) if kind == 2 else None
    n = (1, 2, 4)[kind] * mesh.num_edges
    Z = torch.empty((n, n), dtype=torch.complex128, device="cuda")  # Z[c] is column c
    torch.cuda.synchronize()
    sieb200.assemble_matrix_device(mesh, opts, Z.data_ptr(), tensors=t, ctx=gpu_ctx)
    edge = np.unique(mesh.faces_edges[[0, nf // 3, slab - 10, slab - 1, slab, min(nf - 2, slab + 10), nf - 1]])
    rows = (edge[None, :] + mesh.num_edges * np.arange(n // mesh.num_edges)[:, None]).ravel()
    s = O.kernel_scalars(kind, opts.frequency_hz, eps_r=(eps_in, 1.0) if kind else (1.0, 1.0))
    Zo = O.assemble_rows(O.oracle(), kind, mesh, 1, s, rows, tensors=t, variant=variant)
    Zg = Z[:, torch.from_numpy(rows).cuda()].cpu().numpy().T
    assert np.abs(Zg - Zo).max() <= 1e-12 * np.abs(Zo).max()
    # the product without Z: the same values summed in another order, n of them
    x = np.random.default_rng(level).standard_normal(n) + 0j
    y = sieb200.matvec_matrix_free(mesh, opts, x, tensors=t, ctx=gpu_ctx)
    ref = (Z.T @ torch.from_numpy(x).cuda()).cpu().numpy()
    assert np.linalg.norm(y - ref) <= 1e-12 * np.linalg.norm(ref)


@pytest.mark.parametrize("rule", [1, 5, 17])
@pytest.mark.parametrize("name", ["ico20", "geo180"])
@pytest.mark.parametrize("points", [1, 130])
def test_surface_fields_near_and_far(rule, name, points, gpu_ctx):
    """Few and many near faces per warp, with and without magnetic currents."""
    import sieb200
    mesh = _mesh(name)
    rng = np.random.default_rng(rule)
    p = rng.standard_normal((points, 3))
    p *= (np.where(np.arange(points) % 3, 0.52, 1.7) / np.linalg.norm(p, axis=1))[:, None]
    j, m = (rng.standard_normal(mesh.num_edges) + 1j * rng.standard_normal(mesh.num_edges) for _ in range(2))
    for mc in (m, None):
        E, H = sieb200.evaluate_surface_integral_fields(mesh, j, mc, p, 0.4 * C0, quadrature_rule=rule, ctx=gpu_ctx)
        Eo, Ho = O.surface_fields(O.oracle(), mesh, j, mc, p, 0.4 * C0, rule=rule)
        assert np.abs(E - Eo).max() <= 1e-12 * np.abs(Eo).max()
        assert np.abs(H - Ho).max() <= 1e-12 * np.abs(Ho).max()


@pytest.mark.parametrize("limit", [0.99, 4.0])
@pytest.mark.parametrize("name", ["ico20", "geo180"])
def test_surface_fields_large_phase(name, limit, gpu_ctx):
    """Phases just below the step number's limit, as the call estimates them, and past it
    (sincos): eight roundings of the phase, as in the assembly, four times over
    for sums of as good as random phases, whose total is smaller than their terms."""
    import sieb200
    mesh = _mesh(name)
    rng = np.random.default_rng(7)
    p = rng.standard_normal((9, 3))
    p *= (np.where(np.arange(9) % 3, 0.52, 1.7) / np.linalg.norm(p, axis=1))[:, None]
    j, m = (rng.standard_normal(mesh.num_edges) + 1j * rng.standard_normal(mesh.num_edges) for _ in range(2))
    phase = limit * 1e7
    freq = phase / (4 * max(np.abs(p).max(), np.abs(mesh.vertices).max())) * C0 / (2 * math.pi)
    E, H = sieb200.evaluate_surface_integral_fields(mesh, j, m, p, freq, quadrature_rule=5, ctx=gpu_ctx)
    Eo, Ho = O.surface_fields(O.oracle(), mesh, j, m, p, freq, rule=5)
    assert np.abs(E - Eo).max() <= 32 * ULP * phase * np.abs(Eo).max()
    assert np.abs(H - Ho).max() <= 32 * ULP * phase * np.abs(Ho).max()


@pytest.mark.parametrize("name", ["ico20", "geo180", "geo500", "spindle90"])
@pytest.mark.parametrize("ndir", [1, 127, 129, 1000])
@pytest.mark.parametrize("k0", [3.0, "limit", 4.0e7])
def test_far_field_chunks(name, ndir, k0, gpu_ctx):
    """Direction counts around a CTA's; phases of order one, just below the step
    number's limit as the call estimates them, and past it. The bound at large phases as
    for the surface fields (k0 |r'| at most)."""
    import sieb200
    mesh = _mesh(name)
    extent = np.abs(mesh.vertices).max()
    if k0 == "limit":
        k0 = 0.99e7 / (3 * extent)
    rng = np.random.default_rng(ndir)
    j, m = (rng.standard_normal(mesh.num_edges) + 1j * rng.standard_normal(mesh.num_edges) for _ in range(2))
    frames = sieb200.spherical_frames(np.arccos(rng.uniform(-1, 1, ndir)), rng.uniform(0, 2 * math.pi, ndir))
    got = sieb200.far_field(mesh, j, m, k0, 376.73, *frames, ctx=gpu_ctx)
    want = O.far_field(O.oracle(), mesh, j, m, k0, 376.73, *frames)
    bound = 1e-12 + 32 * ULP * k0 * 3 * extent
    for a, b in zip(got, want):
        assert np.abs(a - b).max() <= bound * np.abs(b).max()


@pytest.mark.parametrize("ndir", [0, 3])
def test_far_field_empty_mesh_refused(ndir, gpu_ctx):
    """A mesh without faces is an error, as in the field evaluation (the split
    of its faces into chunks would divide by zero)."""
    import sieb200
    mesh = sieb200.MeshData(np.zeros((3, 3)), np.zeros((0, 3), np.int32), np.zeros((1, 2), np.int32),
                            np.zeros((0, 3), np.int32))
    frames = sieb200.spherical_frames(np.linspace(0.1, 1.0, ndir), np.zeros(ndir))
    with pytest.raises(sieb200.InvalidArgument):
        sieb200.far_field(mesh, np.zeros(1, complex), None, 1.0, 376.73, *frames, ctx=gpu_ctx)
