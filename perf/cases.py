"""The work a program has this library do, as cases that can be timed: what it
has in hand before the call (`prepare`), one pass through the public entry
points (`run`), what a pass cannot do without (`work`), how far apart two correct
results may be (`tolerance`) and the result in 64 bits (`exact`).

Kinds of case:
  expm           exp(A) of one matrix; api "py": calaman_g_b200.expm, which lays
                 the matrix out and allocates on each call; api "abi": the C
                 entry point with a handle, a workspace and an output that the
                 program keeps
  expm_ad        exp(A) through torch autograd, forward and backward
  expm_batched   many matrices of uneven size and norm in one call
  vjp_batched    the adjoint of many pairs of one size in one call
  expm_herm      exp(H) of a Hermitian or symmetric matrix
  polynomial     p(A) by Paterson-Stockmeyer
"""
import ctypes
import math
import random

import torch

import calaman_g_b200 as cg
from calaman_g_b200 import capi

DTYPES = {"f32": torch.float32, "f64": torch.float64, "c64": torch.complex64, "c128": torch.complex128}
SUFFIX = {"f32": "s", "f64": "d", "c64": "c", "c128": "z"}
WIDE = {"f32": torch.float64, "f64": torch.float64, "c64": torch.complex128, "c128": torch.complex128}
BYTES = {"f32": 4, "f64": 8, "c64": 8, "c128": 16}


def listed():
    return [
        # a small generator exponentiated from Python, one at a time: all latency
        dict(name="expm_f64_40", kind="expm", api="py", dtype="f64", n=40, norm=1.0),
        # a control or Markov model of a few hundred states in a C program's loop
        dict(name="expm_f64_256", kind="expm", api="abi", dtype="f64", n=256, norm=4.0),
        # an odd size and a large norm from Python: single precision, squarings
        dict(name="expm_c64_777", kind="expm", api="py", dtype="c64", n=777, norm=20.0),
        # a quantum propagator exp(-iH), H from the Gaussian unitary ensemble
        dict(name="expm_c128_1024", kind="expm", api="abi", dtype="c128", n=1024, norm=50.0),
        # double precision at an odd size, so that no column starts aligned
        dict(name="expm_f64_1501", kind="expm", api="py", dtype="f64", n=1501, norm=3.0),
        # the largest single matrix: float32 on the tensor cores
        dict(name="expm_f32_4096", kind="expm", api="abi", dtype="f32", n=4096, norm=8.0),
        # training through the exponential of a large matrix: forward and backward
        dict(name="expm_ad_f64_2048", kind="expm_ad", dtype="f64", n=2048, norm=6.0),
        # thousands of small matrices of uneven size and norm in one call
        dict(name="batched_f32_8192", kind="expm_batched", dtype="f32", count=8192, lo=16, hi=256, step=16),
        # a few hundred of any size at double precision
        dict(name="batched_f64_500", kind="expm_batched", dtype="f64", count=500, lo=3, hi=200, step=1),
        # the gradient of a layer's worth of matrix exponentials
        dict(name="vjp_f32_512x128", kind="vjp_batched", dtype="f32", count=512, n=128, norm=6.0),
        # exp of a Hermitian matrix by its eigendecomposition
        dict(name="herm_c128_1024", kind="expm_herm", dtype="c128", n=1024, norm=50.0),
        # a matrix polynomial of degree 16 at an even and unaligned size
        dict(name="poly_f32_1000", kind="polynomial", dtype="f32", n=1000, degree=16, norm=2.0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _size(rng, lo, hi):
    return int(round(_log(rng, lo, hi)))


def draw(rng: random.Random):
    kind = rng.choice(["expm"] * 6 + ["expm_ad", "expm_batched", "expm_batched", "vjp_batched", "expm_herm", "polynomial"])
    norm = round(_log(rng, 0.1, 60.0), 4)
    if kind == "expm":
        dtype = rng.choice(list(DTYPES))
        n = _size(rng, 8, {"f32": 4096, "c64": 1500, "f64": 2048, "c128": 1024}[dtype])
        return dict(kind=kind, api=rng.choice(["py", "abi"]), dtype=dtype, n=n, norm=norm)
    if kind == "expm_ad":
        dtype = rng.choice(["f32", "f64", "c128"])
        return dict(kind=kind, dtype=dtype, n=_size(rng, 16, {"f32": 2048, "f64": 1600, "c128": 512}[dtype]), norm=min(norm, 12.0))
    if kind == "expm_batched":
        lo = _size(rng, 2, 64)
        return dict(kind=kind, dtype=rng.choice(["f32", "f64"]), count=_size(rng, 32, 3000), lo=lo,
                    hi=rng.randint(lo, 256), step=1)
    if kind == "vjp_batched":
        return dict(kind=kind, dtype=rng.choice(["f32", "f64"]), count=_size(rng, 16, 400), n=_size(rng, 8, 160),
                    norm=min(norm, 12.0))
    if kind == "expm_herm":
        dtype = rng.choice(["f64", "c128", "f32"])
        return dict(kind=kind, dtype=dtype, n=_size(rng, 16, 1024), norm=norm)
    return dict(kind=kind, dtype=rng.choice(["f32", "f64"]), n=_size(rng, 16, 1500), degree=rng.randint(2, 30),
                norm=min(norm, 4.0))


# ---- inputs -----------------------------------------------------------------
def _generator(seed, what=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + what)


def _randn(g, *shape, dtype):
    return torch.randn(*shape, generator=g, dtype=dtype, device="cuda")


def _to_norm(a, norm):
    """a (..., n, n) rescaled to the 1-norm `norm` (the largest column sum of moduli)."""
    return a * (norm / a.abs().sum(dim=-2, keepdim=True).amax(dim=-1, keepdim=True))


def _matrix(case, seed):
    """Real: N(0,1) entries; complex: -iH with H from the Gaussian unitary ensemble; rescaled to the case's 1-norm."""
    n, wide = case["n"], WIDE[case["dtype"]]
    a = _randn(_generator(seed), n, n, dtype=wide)
    if case["kind"] == "expm_herm":
        a = (a + a.mH) / 2
    elif wide.is_complex:
        a = -0.5j * (a + a.mH)
    return _to_norm(a, case["norm"]).to(DTYPES[case["dtype"]])


def _batch_plan(case):
    """Sizes and 1-norms of the batch, the case's own: uniform sizes, norms log-uniform in [0.1, 100]."""
    rng = random.Random(case["count"] * 7919 + case["lo"] * 263 + case["hi"])
    sizes = [rng.randrange(case["lo"], case["hi"] + 1, case["step"]) for _ in range(case["count"])]
    return sizes, [_log(rng, 0.1, 100.0) for _ in sizes]


def _batch_groups(case):
    """size -> (offset of its matrices in the buffer, their indices in the batch), and the buffer's elements."""
    sizes, _ = _batch_plan(case)
    groups, at = {}, 0
    for n in sorted(set(sizes)):
        groups[n] = (at, [i for i, k in enumerate(sizes) if k == n])
        at += n * n * len(groups[n][1])
    return groups, at


def _batch_matrices(case, seed):
    """The batch in one buffer: the matrices of one size side by side (their order in the batch is another)."""
    _, norms = _batch_plan(case)
    groups, total = _batch_groups(case)
    g, buf = _generator(seed), torch.empty(total, dtype=DTYPES[case["dtype"]], device="cuda")
    for n, (at, idx) in groups.items():
        a = _randn(g, len(idx), n, n, dtype=buf.dtype)
        t = torch.tensor([norms[i] for i in idx], dtype=buf.dtype, device="cuda").reshape(-1, 1, 1)
        # stored column-major: the columns of a matrix are the rows of its block
        buf[at:at + n * n * len(idx)] = _to_norm(a, t).mT.reshape(-1)
    return buf


_stream = None


def _program_stream():
    """The one stream that this program gives its handles."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _ints(t):
    return ctypes.cast(t.data_ptr(), capi.c_int_p)


def _must(what, st):
    if not st.ok:
        raise RuntimeError("%s failed: %r" % (what, st))


def _workspace(size_fn, *args):
    nb = ctypes.c_size_t()
    _must("bufferSize", size_fn(*args, ctypes.byref(nb)))
    return torch.empty(max(nb.value, 256), dtype=torch.uint8, device="cuda")


def prepare(case, seed):
    kind, suf = case["kind"], SUFFIX[case["dtype"]]
    lib, s = cg.lib(), {"case": case}
    if kind in ("expm", "expm_herm") and case.get("api") != "py":
        n = case["n"]
        s["A"] = cg.to_colmajor(_matrix(case, seed))
        s["E"] = torch.zeros_like(s["A"])
        s["info"] = torch.zeros(2, dtype=torch.int32, device="cuda")
        s["h"], s["plan"] = cg.Handle(_program_stream()), capi.ExpmPlan()
        if kind == "expm":
            s["work"] = _workspace(getattr(lib, "calaman_expm_bufferSize_" + suf), s["h"].ptr, n)
        else:
            s["work"] = _workspace(getattr(lib, "calaman_expm_herm_bufferSize_" + suf), s["h"].ptr, capi.FILL_LOWER, n)
    elif kind == "expm":
        s["a"] = _matrix(case, seed)
    elif kind == "expm_ad":
        s["a"] = _matrix(case, seed).requires_grad_(True)
        s["g"] = _randn(_generator(seed, 1), case["n"], case["n"], dtype=DTYPES[case["dtype"]])
    elif kind == "polynomial":
        s["a"] = _matrix(case, seed)
        s["c"] = torch.tensor(_coefficients(case), dtype=DTYPES[case["dtype"]], device="cuda")
    elif kind == "expm_batched":
        sizes, _ = _batch_plan(case)
        groups, total = _batch_groups(case)
        s["A"] = _batch_matrices(case, seed)
        s["E"] = torch.zeros_like(s["A"])
        offs = [0] * len(sizes)
        for n, (at, idx) in groups.items():
            for k, i in enumerate(idx):
                offs[i] = at + k * n * n
        _batch_handle(s, sizes)
        s["pA"], s["pE"] = (_pointers(s[k], offs) for k in "AE")
        s["work"] = _workspace(getattr(lib, "calaman_expm_batched_bufferSize_" + suf), s["h"].ptr, len(sizes), s["n"])
    elif kind == "vjp_batched":
        n, count, dt = case["n"], case["count"], DTYPES[case["dtype"]]
        g = _generator(seed)
        s["A"] = _to_norm(_randn(g, count, n, n, dtype=dt), case["norm"]).mT.contiguous()
        s["G"] = _randn(g, count, n, n, dtype=dt).mT.contiguous()
        s["D"] = torch.zeros_like(s["A"])
        _batch_handle(s, [n] * count)
        s["pA"], s["pG"], s["pD"] = (_pointers(s[k], range(0, count * n * n, n * n)) for k in "AGD")
        s["work"] = _workspace(getattr(lib, "calaman_expm_vjp_batched_bufferSize_" + suf), s["h"].ptr, count, s["n"])
    return s


def _batch_handle(s, sizes):
    s["n"] = (ctypes.c_int * len(sizes))(*sizes)
    s["info"] = torch.zeros(2 * len(sizes), dtype=torch.int32, device="cuda")
    s["h"], s["plans"] = cg.Handle(_program_stream()), (capi.ExpmPlan * len(sizes))()


def _pointers(buf, offs):
    base, size = buf.data_ptr(), buf.element_size()
    return (ctypes.c_void_p * len(offs))(*[base + o * size for o in offs])


# ---- one pass -----------------------------------------------------------------
def run(s):
    case = s["case"]
    kind, lib = case["kind"], cg.lib()
    if kind == "expm" and case["api"] == "py":
        return cg.expm(s["a"])
    if kind == "expm_ad":
        e = cg.expm_ad(s["a"])
        (grad,) = torch.autograd.grad(e, s["a"], s["g"])
        return e.detach(), grad
    if kind == "polynomial":
        return cg.paterson_stockmeyer(s["a"], s["c"])
    suf, h, work = SUFFIX[case["dtype"]], s["h"], s["work"]
    stream, size = ctypes.c_void_p(h.stream), work.numel()
    if kind == "expm":
        n = case["n"]
        _must("expm", getattr(lib, "calaman_expm_" + suf)(
            h.ptr, h.ptr, stream, n, _ptr(s["A"]), n, _ptr(s["E"]), n, _ptr(work), size, _ints(s["info"]),
            ctypes.byref(s["plan"])))
        return s["E"].mT, s["info"]
    if kind == "expm_herm":
        n = case["n"]
        _must("expm_herm", getattr(lib, "calaman_expm_herm_" + suf)(
            h.ptr, h.ptr, stream, capi.FILL_LOWER, n, _ptr(s["A"]), n, _ptr(s["E"]), n, _ptr(work), size,
            _ints(s["info"])))
        return s["E"].mT, s["info"]
    if kind == "expm_batched":
        _must("expm_batched", getattr(lib, "calaman_expm_batched_" + suf)(
            h.ptr, h.ptr, stream, len(s["n"]), s["n"], s["pA"], s["n"], s["pE"], s["n"], _ptr(work), size,
            _ints(s["info"]), s["plans"]))
        return s["E"], s["info"]
    _must("expm_vjp_batched", getattr(lib, "calaman_expm_vjp_batched_" + suf)(
        h.ptr, h.ptr, stream, len(s["n"]), s["n"], s["pA"], s["n"], s["pG"], s["n"], s["pD"], s["n"], None, s["n"],
        _ptr(work), size, _ints(s["info"]), s["plans"]))
    return s["D"], s["info"]


# ---- what a pass cannot do without --------------------------------------------
def _plan(case, norm):
    p = cg.expm_plan(norm, single=case["dtype"] in ("f32", "c64"))
    return p.m, p.s


def _expm_flops(n, m, s):
    """Products, LU and n-right-hand-side solve of scaling and squaring."""
    return ({3: 2, 5: 3, 7: 4, 9: 5, 13: 6}[m] + s) * 2.0 * n ** 3 + (2.0 / 3.0 + 2.0) * n ** 3


def _vjp_flops(n, m, s):
    """The adjoint: three products for each of the forward's, the LU and two solves."""
    gemms = 3 * {3: 1, 5: 2, 7: 3, 9: 4, 13: 3}[m] + (6 if m == 13 else 0) + 4 + 3 * s
    return gemms * 2.0 * n ** 3 + (2.0 / 3.0 + 4.0) * n ** 3


def work(case):
    kind, size = case["kind"], BYTES[case["dtype"]]
    times = 4.0 if case["dtype"] in ("c64", "c128") else 1.0
    if kind == "expm_batched":
        sizes, norms = _batch_plan(case)
        return {"bytes": 2.0 * size * sum(n * n for n in sizes),
                "flops": sum(_expm_flops(n, *_plan(case, t)) for n, t in zip(sizes, norms))}
    n = case["n"]
    nn = float(size) * n * n
    if kind == "vjp_batched":
        return {"bytes": 3 * nn * case["count"], "flops": case["count"] * _vjp_flops(n, *_plan(case, case["norm"]))}
    if kind == "expm":
        return {"bytes": 2 * nn, "flops": times * _expm_flops(n, *_plan(case, case["norm"]))}
    if kind == "expm_ad":
        m, s = _plan(case, case["norm"])
        return {"bytes": 4 * nn, "flops": times * (_expm_flops(n, m, s) + _vjp_flops(n, m, s))}
    if kind == "expm_herm":
        # tridiagonal reduction, back-transformation, product; the divide and conquer's real products
        return {"bytes": 2 * nn, "flops": (times * (4.0 / 3.0 + 4.0) + 8.0 / 3.0) * n ** 3}
    return {"bytes": 2 * nn, "flops": cg.paterson_stockmeyer_plan(case["degree"]).num_gemms * 2.0 * n ** 3}


def tolerance(case):
    # four times the largest error against 64 bits seen over 72 cases of these ranges: 2.3e-6 in single
    # precision (complex64, norm 22), 8.3e-14 in double (complex128, norm 50), the latter rounded up to
    # the library's own bar for it
    if case["dtype"] in ("f32", "c64"):
        return {"rel": 1e-5}
    return {"rel": 1e-12}


# ---- the result in 64 bits ------------------------------------------------------
def _coefficients(case):
    """A Taylor polynomial of exp with signs of its own: c_k = (-1)^(k // 3) / k!"""
    return [(-1.0) ** (k // 3) / math.factorial(k) for k in range(case["degree"] + 1)]


def exact(case, seed):
    kind, wide = case["kind"], WIDE[case["dtype"]]
    if kind == "expm":
        e = torch.linalg.matrix_exp(_matrix(case, seed).to(wide))
        return e if case["api"] == "py" else (e, None)
    if kind == "expm_herm":
        w, u = torch.linalg.eigh(_matrix(case, seed).to(wide))
        return (u * torch.exp(w)) @ u.mH, None
    if kind == "expm_ad":
        a = _matrix(case, seed).to(wide)
        g = _randn(_generator(seed, 1), case["n"], case["n"], dtype=DTYPES[case["dtype"]]).to(wide)
        return torch.linalg.matrix_exp(a), _adjoint(a, g)
    if kind == "polynomial":
        a = _matrix(case, seed).to(wide)
        p = torch.zeros_like(a)
        for c in reversed(_coefficients(case)):
            p = p @ a
            p.diagonal().add_(c)
        return p
    if kind == "expm_batched":
        buf = _batch_matrices(case, seed).to(wide)
        for n, (at, idx) in _batch_groups(case)[0].items():
            part = buf[at:at + n * n * len(idx)].view(len(idx), n, n)
            part.copy_(torch.linalg.matrix_exp(part.mT).mT)
        return buf, None
    n, count, dt = case["n"], case["count"], DTYPES[case["dtype"]]
    g = _generator(seed)
    a = _to_norm(_randn(g, count, n, n, dtype=dt), case["norm"]).to(wide)
    return _adjoint(a, _randn(g, count, n, n, dtype=dt).to(wide)).mT.contiguous(), None


def _adjoint(a, g):
    """The Frechet derivative of exp at A^H in direction G: the upper right block of exp([[A^H, G], [0, A^H]])."""
    n = a.shape[-1]
    b = torch.zeros(*a.shape[:-2], 2 * n, 2 * n, dtype=a.dtype, device=a.device)
    b[..., :n, :n] = a.mH
    b[..., n:, n:] = a.mH
    # the block's norm is kept near A's: the derivative is linear in G
    t = float(a.abs().sum(dim=-2).amax()) / max(float(g.abs().sum(dim=-2).amax()), 1e-300)
    b[..., :n, n:] = t * g
    return torch.linalg.matrix_exp(b)[..., :n, n:] / t
