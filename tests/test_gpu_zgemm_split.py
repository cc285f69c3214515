"""Multi-right-hand-side mixed solves at sizes where the FP64 product Z X
splits its K over CTAs (few 64 x 64 tiles, K >= 256), with K remainders of every kind,
and just where it does not (K < 256; many columns), against numpy.

The solve stops at a relative residual of 1e-11 that it forms with that
product; the oracle forms the residual again, with a rounding of a few n eps =
1300 * 2.2e-16 = 3e-13 relative to |Z| |x| / |b| < 3. A bound of 2e-11 covers
both; a wrong product gives a residual of order one.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nrhs", [(64, 2), (255, 3), (256, 2), (257, 8), (300, 64), (391, 65), (640, 130),
                                    (1000, 5), (1297, 9)])
def test_split_product_residual(gpu_ctx, n, nrhs):
    import torch
    import sieb200
    rng = np.random.default_rng(n + nrhs)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 4.0 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    Z = torch.from_numpy(A.T.copy()).cuda()
    X = torch.from_numpy(B.T.copy()).cuda()
    torch.cuda.synchronize()
    s = sieb200.DenseLuSolver(n, "mixed_ir", ctx=gpu_ctx)
    s.factorize(Z.data_ptr())
    s.solve(X.data_ptr(), nrhs=nrhs, tolerance=1e-11, max_iterations=30)
    gpu_ctx.synchronize()
    r = B - A @ X.cpu().numpy().T
    assert (np.linalg.norm(r, axis=0) <= 2e-11 * np.linalg.norm(B, axis=0)).all()
    s.close()
