"""expm of small matrices (one kernel on one CTA up to n = 64, complex 48)
against the oracle, at the edges of its tile classes and of its range, every
Pade degree, with squarings, padded leading dimensions and in place."""
import ctypes

import numpy as np
import pytest

from helpers import NP_DTYPE, Runner, _dev, colmajor_buffer, from_buffer, rel_frob, scaled_random, vp

pytestmark = pytest.mark.gpu

# FP64 tiers: the library's bar. Single tiers: the one kernel evaluates in FP64 and rounds each
# entry once, so at most 2^-24 (6e-8) of the result's norm, and the oracle's FP64 beside it; FP32
# arithmetic anywhere in it shows (1.8e-7 at norm 1). Sizes beyond the kernel take the general path,
# with eps x the entries' growth in the scaled evaluation (a few tens) x 2^s for the squarings.
BAR = {"d": 1e-12, "z": 1e-12, "s": 6.1e-8, "c": 6.1e-8}
GENERAL = {"d": 1e-12, "z": 1e-12, "s": 2e-5, "c": 2e-5}
NORMS = [0.01, 0.2, 0.9, 2.0, 3.5, 5.3, 40.0]  # m = 3 .. 13, s = 0 and s > 0


def bar(suf, n):
    return BAR[suf] if n <= (48 if suf in "cz" else 64) else GENERAL[suf]


@pytest.fixture(scope="module")
def run(cuda):
    r = Runner()
    yield r
    r.close()


@pytest.mark.parametrize("suf", ["s", "d", "c", "z"])
@pytest.mark.parametrize("n,norm", [(n, t) for n in (17, 48, 64) for t in NORMS]
                         + [(n, NORMS[(i + k) % 7]) for i, n in enumerate((1, 2, 3, 15, 16, 32, 33, 47, 49, 63, 65))
                            for k in (0, 2, 5)])
def test_small_expm_matches_oracle(run, oracle, suf, n, norm):
    a = scaled_random(n, norm, 77 * n + int(10 * norm), suf in "cz")
    if norm > 6:
        # Forming q = V - U loses a factor |V| / |q|, up to exp(|X|) with |X| up to 11 in the single tiers
        # (2e4 eps for the scalar 10), for a positive real spectrum. On skew-Hermitian input |q| stays near
        # |V|, so the bar holds: an imaginary spectrum for the large norm.
        a = a - a.conj().T
        a = a * (norm / max(np.abs(a).sum(axis=0).max(), 1e-300))
    a = a.astype(NP_DTYPE[suf])
    st, plan, e, _, info = run.expm(a, suf)
    ref, oplan, _ = oracle.expm(a, single=suf in "sc")
    assert st.ok and list(info) == [0, 0]
    assert (plan.m, plan.s) == (oplan.m, oplan.s)
    assert rel_frob(e, ref) <= bar(suf, n)


@pytest.mark.parametrize("suf", ["d", "z"])
@pytest.mark.parametrize("n", [2, 10, 34, 48])
def test_small_expm_pivots(run, oracle, suf, n):
    """exp of rotations by almost pi: q_13 is close to exp(-A/2), a quarter turn with a diagonal near zero,
    so every second column pivots."""
    a = np.kron(np.eye(n // 2), np.array([[0.0, 3.1], [-3.1, 0.0]])).astype(NP_DTYPE[suf])
    st, plan, e, _, info = run.expm(a, suf)
    ref, _, _ = oracle.expm(a)
    assert st.ok and list(info) == [0, 0] and plan.m == 13
    assert rel_frob(e, ref) <= BAR[suf]


@pytest.mark.parametrize("suf", ["s", "d", "c", "z"])
@pytest.mark.parametrize("norm", [1.0, 30.0])
def test_small_expm_in_place(run, oracle, suf, norm):
    import torch

    n, ld = 37, 41
    a = scaled_random(n, norm, 5, suf in "cz")
    a = (a - a.conj().T).astype(NP_DTYPE[suf])  # skew, as above
    dA = _dev(colmajor_buffer(a, ld, suf))
    before = dA.cpu().numpy().reshape(n, ld)[:, n:].copy()
    b = ctypes.c_size_t()
    assert getattr(run.lib, f"calaman_expm_bufferSize_{suf}")(run.h, n, ctypes.byref(b)).ok
    w = run.workspace(b.value)
    info = torch.full((2,), -9, dtype=torch.int32, device="cuda")
    plan = run.capi.ExpmPlan()
    st = getattr(run.lib, f"calaman_expm_{suf}")(
        run.h, run.h, ctypes.c_void_p(run.stream), n, vp(dA), ld, vp(dA), ld, vp(w), b.value,
        ctypes.cast(info.data_ptr(), run.capi.c_int_p), ctypes.byref(plan))
    torch.cuda.synchronize()
    assert st.ok and info.tolist() == [0, 0]
    full = dA.cpu().numpy()
    assert np.array_equal(full.reshape(n, ld)[:, n:], before)  # the padding rows are untouched
    ref, _, _ = oracle.expm(a, single=suf in "sc")
    assert rel_frob(from_buffer(full, n, ld), ref) <= bar(suf, n)


@pytest.mark.parametrize("suf", ["s", "d", "c", "z"])
def test_kernel_timing_runs_the_same_kernel(run, suf):
    """With kernel timing on a small matrix takes the same path: the same bits, and no GEMM launch to time."""
    a = scaled_random(37, 2.0, 6, suf in "cz").astype(NP_DTYPE[suf])
    st, _, plain, _, _ = run.expm(a, suf)
    assert st.ok and run.lib.calamanSetKernelTiming(run.h, 1).ok
    try:
        st, _, timed, _, info = run.expm(a, suf)
        kt = run.capi.KernelTiming()
        assert st.ok and list(info) == [0, 0] and run.lib.calamanGetKernelTiming(run.h, ctypes.byref(kt)).ok
    finally:
        run.lib.calamanSetKernelTiming(run.h, 0)
    assert np.array_equal(timed, plain) and kt.gemm_launches == 0
