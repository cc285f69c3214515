"""FP64 LU in groups of four 64-row block steps: sizes around a block, around
a group and with every remainder of blocks in the last group, with the FP64
tensor-core GEMM and with the FMA kernel, against numpy.

Tolerance: the systems have condition numbers below 10, so the forward error
is below 10 times the residual the solve stops at (1e-13); the oracle's own rounding
adds about n eps = 577 * 2.2e-16 = 1.3e-13. Together 1.2e-12; 2e-12 is used.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dmma", ["1", "0"])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 132, 191, 193, 255, 256, 257, 260, 319, 320, 324, 385, 449, 512,
                               516, 577])
def test_fp64_lu_groups(gpu_ctx, monkeypatch, n, dmma):
    import torch
    import sieb200
    monkeypatch.setenv("SIEB200_ZGEMM_DMMA", dmma)
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 4.0 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, 3)) + 1j * rng.standard_normal((n, 3))
    Z = torch.from_numpy(A.T.copy()).cuda()
    X = torch.from_numpy(B.T.copy()).cuda()
    torch.cuda.synchronize()
    s = sieb200.DenseLuSolver(n, "lu_fp64", ctx=gpu_ctx)
    s.factorize(Z.data_ptr())
    s.solve(X.data_ptr(), nrhs=3, tolerance=1e-13, max_iterations=2)
    gpu_ctx.synchronize()
    ref = np.linalg.solve(A, B)
    assert np.linalg.norm(X.cpu().numpy().T - ref) <= 2e-12 * np.linalg.norm(ref)
    s.close()


@pytest.mark.parametrize("n,nrhs", [(n, c) for n in (7, 64, 130, 323) for c in (1, 4, 5, 32, 33)] + [(1300, 33)])
def test_fp64_triangular_columns(gpu_ctx, n, nrhs):
    """Column counts around a CTA's columns of the one-kernel step and around
    the count above which a diagonal kernel and a GEMM take over."""
    import torch
    import sieb200
    rng = np.random.default_rng(1000 * n + nrhs)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 4.0 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    Z = torch.from_numpy(A.T.copy()).cuda()
    X = torch.from_numpy(B.T.copy()).cuda()
    torch.cuda.synchronize()
    s = sieb200.DenseLuSolver(n, "lu_fp64", ctx=gpu_ctx)
    s.factorize(Z.data_ptr())
    s.solve(X.data_ptr(), nrhs=nrhs, tolerance=1e-13, max_iterations=2)
    gpu_ctx.synchronize()
    ref = np.linalg.solve(A, B)
    assert np.linalg.norm(X.cpu().numpy().T - ref) <= 2e-12 * np.linalg.norm(ref)
    s.close()
