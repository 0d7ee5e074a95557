"""The public single-precision products on the FMA pipes (calaman_gemm_s) against a
float64 product: both kernels at the edges of the rule that chooses between them, of
their tiles and of their depth steps, with aligned and unaligned columns."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(cuda):
    from calaman_g_b200 import capi

    return capi.load()


def colmajor(x, ld):
    buf = np.full((x.shape[1], ld), -7.5, dtype=np.float32)
    buf[:, : x.shape[0]] = x.T
    return buf


@pytest.mark.parametrize("pad", [0, 1])  # columns that start 16-byte aligned where m and k divide by four, or not
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (16, 16, 16), (33, 31, 17), (32, 32, 64), (32, 33, 64), (64, 64, 63),
                                   (64, 64, 65), (65, 129, 64), (129, 65, 31), (333, 130, 97), (900, 1000, 16),
                                   (900, 1000, 20), (1001, 900, 333)])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-0.5, 2.0)])
def test_gemm_s_matches_fp64(lib, m, n, k, pad, alpha, beta):
    """|error| <= (k + 4) eps (|alpha| |A||B| + |beta| |C|) element by element, in any order of the sum; the
    padding rows of C are untouched, and beta = 0 never reads C."""
    import torch

    rng = np.random.default_rng(m + 3 * n + 7 * k)
    a, b, c = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (k, n), (m, n)))
    lda, ldb, ldc = m + pad, k + pad, m + pad
    dA, dB = (torch.from_numpy(colmajor(x, ld)).cuda() for x, ld in ((a, lda), (b, ldb)))
    dC = torch.from_numpy(colmajor(c if beta != 0 else np.full_like(c, np.nan), ldc)).cuda()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    st = lib.calaman_gemm_s(None, m, n, k, alpha, p(dA), lda, p(dB), ldb, beta, p(dC), ldc)
    torch.cuda.synchronize()
    assert st.ok, st
    got = dC.cpu().numpy()
    a, b, c = (x.astype(np.float64) for x in (a, b, c))
    ref, size = alpha * (a @ b) + beta * c, abs(alpha) * (np.abs(a) @ np.abs(b)) + abs(beta) * np.abs(c)
    assert (np.abs(got[:, :m].T - ref) <= (k + 4) * 2.0 ** -24 * size).all()
    assert (got[:, m:] == -7.5).all()
