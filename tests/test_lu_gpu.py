"""GPU LU with partial pivoting and the n-RHS solve (the getrf/getrs pade()
runs on q_m(A)), against the oracle's xGETRF restatement: identical pivot
sequences and factors (FP64 tiers), backward-stable solves (all tiers), and
LAPACK's info code on singular input. Inputs are dense Gaussian matrices, so
every column pivots -- unlike the Pade denominators of well-scaled matrices,
which are close to diagonally dominant."""
import ctypes

import numpy as np
import pytest

from helpers import NP_DTYPE, colmajor_buffer, eps, from_buffer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(cuda):
    from calaman_g_b200 import capi

    return capi.load()


def vp(t):
    return ctypes.c_void_p(t.data_ptr())


def gaussian(n, suf, seed, m=None):
    rng = np.random.default_rng(seed)
    m = m or n
    a = rng.standard_normal((n, m))
    if suf in "cz":
        a = a + 1j * rng.standard_normal((n, m))
    return a.astype(NP_DTYPE[suf])


def run_getrf(lib, a, suf, lda=None):
    import torch

    n = a.shape[0]
    lda = lda or n
    dA = torch.from_numpy(colmajor_buffer(a, lda, suf)).cuda()
    b = ctypes.c_size_t()
    assert lib.calaman_getrf_bufferSize(n, ctypes.byref(b)).ok
    scratch = torch.zeros(b.value, dtype=torch.uint8, device="cuda")
    info = torch.full((1,), -5, dtype=torch.int32, device="cuda")
    st = getattr(lib, f"calaman_getrf_{suf}")(None, n, vp(dA), lda, vp(scratch),
                                             ctypes.cast(info.data_ptr(), ctypes.POINTER(ctypes.c_int)))
    torch.cuda.synchronize()
    assert st.ok, st
    ipiv = scratch[: 4 * n].view(torch.int32).cpu().numpy()
    return dA, scratch, from_buffer(dA.cpu().numpy(), n, lda), ipiv, int(info.item())


@pytest.mark.parametrize("suf", ["d", "z"])
@pytest.mark.parametrize("n", [1, 2, 7, 63, 64, 65, 100, 300, 513, 1024])
def test_getrf_matches_oracle_exactly_in_pivots(lib, oracle, suf, n):
    a = gaussian(n, suf, 500 + n)
    _, _, lu, ipiv, info = run_getrf(lib, a, suf)
    olu, opiv, oinfo = oracle.getrf(a)
    assert info == 0 and oinfo == 0
    assert np.array_equal(ipiv, opiv)
    assert np.abs(lu - olu).max() <= 1e-12 * max(1.0, np.abs(olu).max()) * np.sqrt(n)


@pytest.mark.parametrize("suf", ["s", "c"])
@pytest.mark.parametrize("n", [5, 64, 200, 700, 3001])
def test_getrf_single_backward_error(lib, suf, n):
    a = gaussian(n, suf, 600 + n)
    _, _, lu, ipiv, info = run_getrf(lib, a, suf)
    assert info == 0
    L = np.tril(lu, -1) + np.eye(n)
    U = np.triu(lu)
    pa = a.astype(np.complex128).copy()
    for j, p in enumerate(ipiv):  # replay the row swaps
        pa[[j, p]] = pa[[p, j]]
    res = np.abs(pa - L.astype(np.complex128) @ U.astype(np.complex128)).max()
    assert res <= 64 * eps(suf) * n * np.abs(a).max()
    # partial pivoting on |Re|+|Im| bounds |l_ij| by 1 (real) and sqrt(2) (complex)
    bound = np.sqrt(2.0) if suf in "cz" else 1.0
    assert np.all(np.abs(np.tril(lu, -1)) <= bound * (1 + 1e-6))


@pytest.mark.parametrize("suf", ["s", "d", "c", "z"])
@pytest.mark.parametrize("n,nrhs", [(1, 1), (9, 3), (64, 64), (130, 7), (400, 400), (1500, 77)])
def test_getrs_solves(lib, suf, n, nrhs):
    import torch

    a = gaussian(n, suf, 700 + n)
    b = gaussian(n, suf, 800 + n, nrhs)
    dA, scratch, _, _, info = run_getrf(lib, a, suf)
    assert info == 0
    dB = torch.from_numpy(np.asfortranarray(b).reshape(-1, order="F")).cuda()
    dX = torch.empty_like(dB)
    dinfo = torch.full((1,), -5, dtype=torch.int32, device="cuda")
    st = getattr(lib, f"calaman_getrs_{suf}")(None, n, nrhs, vp(dA), n, vp(scratch), vp(dB), n,
                                             vp(dX), n,
                                             ctypes.cast(dinfo.data_ptr(), ctypes.POINTER(ctypes.c_int)))
    torch.cuda.synchronize()
    assert st.ok and int(dinfo.item()) == 0
    x = dX.cpu().numpy().reshape(nrhs, n).T.astype(np.complex128)
    a64, b64 = a.astype(np.complex128), b.astype(np.complex128)
    res = np.linalg.norm(a64 @ x - b64) / (np.linalg.norm(a64) * np.linalg.norm(x) + np.linalg.norm(b64))
    assert res <= 32 * eps(suf) * np.sqrt(n)


@pytest.mark.parametrize("suf", ["d", "z"])
def test_getrf_singular_info(lib, oracle, suf):
    n = 70
    a = gaussian(n, suf, 900)
    a[:, 5] = 0.0  # column 5 exactly zero -> U(5,5) = 0
    _, _, _, _, info = run_getrf(lib, a, suf)
    _, _, oinfo = oracle.getrf(a)
    assert info == oinfo == 6


def test_getrf_padded_leading_dimension(lib, oracle):
    n, lda = 90, 97
    a = gaussian(n, "d", 901)
    _, _, lu, ipiv, info = run_getrf(lib, a, "d", lda=lda)
    olu, opiv, _ = oracle.getrf(a)
    assert info == 0 and np.array_equal(ipiv, opiv)
    assert np.abs(lu - olu).max() <= 1e-12 * np.abs(olu).max()


@pytest.mark.parametrize("suf,m,target", [("d", 13, 30.0), ("z", 13, 25.0), ("d", 3, 4.0),
                                          ("s", 9, 20.0), ("c", 13, 20.0)])
def test_pade_large_norm_pivoting(oracle, suf, m, target, cuda):
    """pade() does not scale: a large norm makes q_m(A) far from diagonally
    dominant, so the LU inside pivots on most columns."""
    from helpers import Runner, rel_frob, scaled_random

    run = Runner()
    a = scaled_random(120, target, 31 + m, suf in "cz")
    a = a.astype(NP_DTYPE[suf])
    st, r, info = run.pade(a, m, suf)
    ref, _ = oracle.pade(a, m)
    run.close()
    assert st.ok and list(info) == [0, 0]
    assert rel_frob(r, ref) <= (1e-11 if suf in "dz" else 1e-3)


@pytest.mark.parametrize("suf", ["s", "d", "c", "z"])
@pytest.mark.parametrize("n", [600, 1100])
def test_solve_beside_the_factorisation_pivots(cuda, suf, n):
    """pade() solves beside its LU. A has imaginary eigenvalues close to pi and a dense orthogonal (unitary)
    basis, so q_13 is close to a multiple of exp(-A/2), a dense orthogonal matrix with a small diagonal:
    perfectly conditioned, and most of its columns pivot, in panels of eight CTAs and of one, with the
    look-ahead and the right-hand side's swaps and updates. r_13 is exp(A) to rounding at this norm."""
    import torch

    from helpers import Runner, rel_frob

    g = torch.Generator(device="cuda").manual_seed(n)
    wide = torch.complex128 if suf in "cz" else torch.float64
    q, _ = torch.linalg.qr(torch.randn(n, n, generator=g, dtype=wide, device="cuda"))
    w = 3.05 + 0.18 * torch.rand(n // 2, generator=g, dtype=torch.float64, device="cuda")
    if suf in "cz":
        k = torch.diag(torch.cat([1j * w, -1j * w]))
    else:
        k = torch.zeros(n, n, dtype=wide, device="cuda")
        i = torch.arange(0, n, 2, device="cuda")
        k[i, i + 1], k[i + 1, i] = w, -w
    a = (q @ k @ q.mH).to({"s": torch.float32, "c": torch.complex64}.get(suf, wide))
    den, num = torch.linalg.matrix_exp(a.to(wide) / -2), torch.linalg.matrix_exp(a.to(wide) / 2)
    pivots = torch.linalg.lu_factor(den)[1].cpu().numpy()
    assert (pivots != np.arange(1, n + 1)).sum() > n // 2
    run = Runner()
    st, r, info = run.pade(a.cpu().numpy(), 13, suf)
    run.close()
    assert st.ok and list(info) == [0, 0]
    ref = torch.linalg.matrix_exp(a.to(wide)).cpu().numpy()
    # a dense orthogonal matrix has element growth (77 at n = 600, 156 at 1100) that any LU with partial
    # pivoting shows: four times the error of torch's own in this precision (1.9e-5 in float32 at 1100), and
    # a few tens of roundings for the products behind q and p
    other = rel_frob(torch.linalg.solve(den.to(a.dtype), num.to(a.dtype)).cpu().numpy(), ref)
    assert rel_frob(r, ref) <= 4 * other + 64 * eps(suf)


def hadamard(n):
    h = np.ones((1, 1))
    while h.shape[0] < n:
        h = np.block([[h, h], [h, -h]])
    return h


@pytest.mark.parametrize("suf", ["s", "d", "c", "z"])
@pytest.mark.parametrize("n", [64, 512, 1024])  # one CTA, its largest height, a cluster of eight
def test_getrf_ties_take_the_first_row(lib, oracle, suf, n):
    """A Hadamard matrix eliminates without rounding (entries stay powers of two) and ties in every
    column: the pivots are IxAMAX's, and the factors are exact."""
    a = hadamard(n).astype(NP_DTYPE[suf])
    _, _, lu, ipiv, info = run_getrf(lib, a, suf)
    olu, opiv, oinfo = oracle.getrf(a.astype(np.complex128 if suf in "cz" else np.float64))
    assert info == oinfo == 0
    assert np.array_equal(ipiv, opiv)
    assert np.array_equal(lu, olu.astype(lu.dtype))


@pytest.mark.parametrize("suf,n", [("d", 33), ("d", 511), ("z", 31), ("z", 257), ("d", 2049)])
def test_getrf_panel_edges(lib, oracle, suf, n):
    """Ragged last panels and the heights next to a change of the panel's cluster."""
    a = gaussian(n, suf, 910 + n)
    _, _, lu, ipiv, info = run_getrf(lib, a, suf)
    olu, opiv, oinfo = oracle.getrf(a)
    assert info == oinfo == 0 and np.array_equal(ipiv, opiv)
    assert np.abs(lu - olu).max() <= 1e-12 * max(1.0, np.abs(olu).max()) * np.sqrt(n)


@pytest.mark.parametrize("suf,n", [("s", 4096), ("s", 4097), ("z", 2049), ("c", 2300)])
def test_getrf_tallest_panels(lib, suf, n):
    """The tallest one-row-per-thread panels and the first size beyond them, by their residual:
    |PA - LU| <= n eps |L||U| element by element, |L| <= sqrt(2), |U| measured."""
    import torch

    a = gaussian(n, suf, 920 + n)
    _, _, lu, ipiv, info = run_getrf(lib, a, suf)
    assert info == 0
    t = torch.from_numpy(lu.astype(np.complex128 if suf in "cz" else np.float64)).cuda()
    L, U = torch.tril(t, -1), torch.triu(t)
    L.diagonal().fill_(1.0)
    perm = np.arange(n)
    for j, p in enumerate(ipiv):
        perm[[j, p]] = perm[[p, j]]
    pa = torch.from_numpy(a.astype(np.complex128 if suf in "cz" else np.float64)[perm]).cuda()
    assert bool(((pa - L @ U).abs() <= n * eps(suf) * (L.abs() @ U.abs())).all())
    assert float(torch.tril(t, -1).abs().max()) <= (np.sqrt(2.0) if suf in "cz" else 1.0) * (1 + 1e-6)


@pytest.mark.parametrize("n", [96, 700])
def test_getrf_nan_column_keeps_its_row(lib, oracle, n):
    """A column of NaNs has no candidate: its own row is kept, as the oracle does."""
    a = gaussian(n, "d", 930 + n)
    a[:, 40] = np.nan
    _, _, _, ipiv, info = run_getrf(lib, a, "d")
    _, opiv, _ = oracle.getrf(a)
    assert np.array_equal(ipiv[:41], opiv[:41]) and ipiv[40] == 40


@pytest.mark.parametrize("suf,n,lda", [("s", 1300, 1303), ("d", 900, 900), ("c", 700, 701), ("z", 2100, 2100),
                                       ("d", 400, 400)])
@pytest.mark.parametrize("drop,tries", [(0, 1 << 12), (3, 1 << 12), (5, 0)])
def test_panel_waits_run_out_in_range(lib, oracle, suf, n, lda, drop, tries):
    """From panel column `drop` on one CTA of a panel pushes nothing (tries = 0: no wait lasts): every CTA gives
    the panel up with the same outcome. info is n + 1, the pivots are in range, the padding rows, the scratch's
    end and the bytes behind the matrix are untouched, and the next call is right.
    A panel on one CTA (n = 400) has no such wait."""
    import torch

    a = gaussian(n, suf, 940 + n)
    guard = 4096
    buf = np.concatenate([colmajor_buffer(a, lda, suf), np.full(guard, 7, dtype=NP_DTYPE[suf])])
    dA = torch.from_numpy(buf).cuda()
    b = ctypes.c_size_t()
    assert lib.calaman_getrf_bufferSize(n, ctypes.byref(b)).ok
    scratch = torch.full((b.value + guard,), 0x5A, dtype=torch.uint8, device="cuda")
    info = torch.full((2,), -5, dtype=torch.int32, device="cuda")
    ip = ctypes.cast(info.data_ptr(), ctypes.POINTER(ctypes.c_int))
    st = getattr(lib, f"calaman_getrf_wait_check_{suf}")(None, n, vp(dA), lda, vp(scratch), drop, tries, ip)
    torch.cuda.synchronize()
    assert st.ok, st
    got = dA.cpu().numpy()
    ipiv = scratch[: 4 * n].view(torch.int32).cpu().numpy()
    one_cta = n <= 512
    assert info.tolist() == [0 if one_cta else n + 1, -5]
    if not one_cta:
        assert np.array_equal(ipiv, np.arange(n))
    assert bool((scratch[b.value:] == 0x5A).all())
    assert np.array_equal(got[n * lda:], buf[n * lda:])
    assert np.array_equal(got[: n * lda].reshape(n, lda)[:, n:], buf[: n * lda].reshape(n, lda)[:, n:])
    _, _, lu, ipiv, again = run_getrf(lib, a, suf)
    assert again == 0 and np.isfinite(lu).all()
    if suf in "dz" and n < 1000:
        assert np.array_equal(ipiv, oracle.getrf(a)[1])
