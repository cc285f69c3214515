"""The blocked schedule of the mixed LU (groups of four block steps, FP16
split packs) at the edges of its groups, and entries far apart in size.

A one-step bound of 1e-5 leaves two digits to the single-precision factors of
these well-conditioned systems (5e-8 by an emulation of the split products)."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(A, b, ctx, **kw):
    import torch
    import sieb200
    n = A.shape[0]
    Z = torch.from_numpy(np.asfortranarray(A).T.copy()).cuda()  # column-major storage
    s = sieb200.DenseLuSolver(n, "mixed_ir", ctx=ctx)
    out = []
    for _ in range(3):  # eager, captured, replayed
        x = torch.from_numpy(b.copy()).cuda()
        torch.cuda.synchronize()
        s.factorize(Z.data_ptr())
        it = s.solve(x.data_ptr(), **kw)
        ctx.synchronize()
        out.append(x.cpu().numpy())
    s.close()
    for x in out[1:]:
        assert np.array_equal(x, out[0])
    return out[0], it


@pytest.mark.parametrize("n", [128, 132, 252, 260, 320, 324, 384, 516, 580, 772])
@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e12])
def test_group_edges_one_step(n, scale, gpu_ctx):
    """One preconditioned step reaches 1e-5 whatever the scale of the system (as
    long as the FP32 square of a pivot is a normal number: the diagonal blocks
    take others as singular)."""
    rng = np.random.default_rng(n)
    A = scale * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 3.0 * math.sqrt(n) * np.eye(n))
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    x, it = _solve(A, b, gpu_ctx, tolerance=1e-5, max_iterations=1)
    assert it == 1 and np.linalg.norm(A @ x - b) <= 1e-5 * np.linalg.norm(b)
    x, _ = _solve(A, b, gpu_ctx, tolerance=1e-12, max_iterations=20)
    assert np.linalg.norm(A @ x - b) <= 1e-12 * np.linalg.norm(b)


def _butterfly(n, offset):
    """The transposed depth-2 butterfly the factorization applies to rows (offset
    0) and columns (offset 4 n): diagonals exp(r / 10) from splitmix64."""
    i = np.arange(offset, offset + 4 * n, dtype=np.uint64)
    with np.errstate(over="ignore"):
        z = np.uint64(0x5EB200) + np.uint64(0x9E3779B97F4A7C15) * (i + np.uint64(1))
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    z ^= z >> np.uint64(31)
    d = np.exp(((z >> np.uint64(11)).astype(np.float64) / 2.0 ** 53 - 0.5) / 10.0) * math.sqrt(0.5)
    h, q = n // 2, n // 4
    a, b, e, f = d[:h], d[h:n], d[n:n + h], d[n + h:n + 2 * h]
    x = np.eye(n).reshape(4, q, n)
    col = lambda v: v[:, None]  # noqa: E731
    y = [(x[0] + x[1]) * col(e[:q]), (x[0] - x[1]) * col(f[:q]), (x[2] + x[3]) * col(e[q:]), (x[2] - x[3]) * col(f[q:])]
    return np.concatenate([(y[0] + y[2]) * col(a[:q]), (y[1] + y[3]) * col(a[q:]), (y[0] - y[2]) * col(b[:q]),
                           (y[1] - y[3]) * col(b[q:])])


@pytest.mark.parametrize("entry", [500.0, 2000.0])
def test_packs_out_of_fp16_range(entry, gpu_ctx, monkeypatch):
    """A transformed matrix whose L21 holds one entry far above its neighbours in
    the row, which leaves FP16's range in an unscaled pack: refined to 1e-10 in as many
    iterations as with TF32 operands (the step-by-step schedule)."""
    n = 192
    rng = np.random.default_rng(5)
    W = np.eye(n) + 0.01 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    L = np.eye(n, dtype=np.complex128)
    L[130, 7] = entry
    A = np.linalg.solve(_butterfly(n, 0), L @ W) @ np.linalg.inv(_butterfly(n, 4 * n)).T
    b = A @ (rng.standard_normal(n) + 1j * rng.standard_normal(n))
    x, it = _solve(A, b, gpu_ctx, tolerance=1e-10, max_iterations=30)
    assert np.linalg.norm(A @ x - b) <= 1e-10 * np.linalg.norm(b)
    monkeypatch.setenv("SIEB200_PAIR_UPDATE", "0")
    _, it_tf32 = _solve(A, b, gpu_ctx, tolerance=1e-10, max_iterations=30)
    assert it <= it_tf32


@pytest.mark.parametrize("diag", ["", "REC", "COMPACT", "PANELS", "SPLIT=0"])
@pytest.mark.parametrize("graded", ["rows", "columns", "both"])
@pytest.mark.parametrize("n", [256, 772, 1024])
def test_graded_system_one_step(n, graded, diag, gpu_ctx, monkeypatch):
    """Rows, columns or both scaled by random powers of two within 2^48: an LU of
    FP32 operands is the same up to those powers, and FP16 packs with a scale per row
    and column alone leave a residual of 2e-3. A scale repeats every n / 4 rows,
    which the butterflies mix, so that it survives them and a block of 64 rows holds
    the whole range. Every diagonal-block kernel, each of which finds the packs' balancing."""
    if diag:
        monkeypatch.setenv("SIEB200_DIAG_" + diag.split("=")[0], diag.split("=")[-1] if "=" in diag else "1")
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 3.0 * math.sqrt(n) * np.eye(n)
    d = 2.0 ** np.round(48.0 * (rng.random((2, n // 4)) - 0.5))
    d1, d2 = np.tile(d, 4)
    d1 = d1 if graded != "columns" else np.ones(n)
    d2 = d2 if graded != "rows" else np.ones(n)
    A *= np.outer(d1, d2)
    b = A @ ((rng.standard_normal(n) + 1j * rng.standard_normal(n)) / d2)
    x, it = _solve(A, b, gpu_ctx, tolerance=1e-5, max_iterations=1)
    r = A @ x - b
    assert it == 1 and np.linalg.norm(r) <= 1e-5 * np.linalg.norm(b)
    assert np.linalg.norm(r / d1) <= 1e-5 * np.linalg.norm(b / d1)
