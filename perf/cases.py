"""Performance cases of the factorizations and their reverse rules.

Each case is one pass through the public entry points as a program calls
them: the out-of-place forms for a single matrix (the caller keeps its
input), caller-held output buffers for the batched forms, and the
differentiable front-end for forward + backward.  Matrices are iid Gaussian,
as random and tensor-network matrices mostly are, except the square polar
problem, whose singular values span four decades.
"""

from __future__ import annotations

import math

import torch

import __graft_entry__

mak = __graft_entry__.load_package()

DTYPES = {"f64": torch.float64, "z": torch.complex128, "f32": torch.float32,
          "c": torch.complex64}
SINGLE = ("qr", "qr_full", "lq", "left_polar", "right_polar")
GRAD = ("grad_qr", "grad_polar")


def _case(name, op, dtype, precision, m, n, count=1, kappa=0.0):
    return {"name": name, "op": op, "dtype": dtype, "precision": precision, "m": m, "n": n,
            "count": count, "kappa": kappa}


def listed():
    return [
        # one small matrix, the call a script makes in a loop: launches and latency count
        _case("qr_f64_96x48", "qr", "f64", "native", 96, 48),
        # an ordinary dense QR in plain Float64 (the default precision), ragged sizes
        _case("qr_f64_1000x501", "qr", "f64", "native", 1000, 501),
        # the largest single problem of the benchmark, in the precision it is quoted on
        _case("qr_f64_16384x8192_mixed", "qr", "f64", "mixed", 16384, 8192),
        # the full orthogonal basis (null spaces, completions), mixed precision
        _case("qr_full_f64_2049x1000_mixed", "qr_full", "f64", "mixed", 2049, 1000),
        # a wide single-precision matrix right-orthogonalised: LQ through the transposed QR
        _case("lq_f32_1537x4093", "lq", "f32", "native", 1537, 4093),
        # polar factor of a tall complex single-precision block, from the right
        _case("right_polar_c_255x612", "right_polar", "c", "native", 255, 612),
        # the ill-conditioned square polar problem (nearest unitary), mixed precision
        _case("left_polar_f64_4096_mixed", "left_polar", "f64", "mixed", 4096, 4096, 1, 1e4),
        # one differentiated tensor of a complex network, through QR and through polar
        _case("grad_qr_z_1024x512_mixed", "grad_qr", "z", "mixed", 1024, 512),
        _case("grad_polar_z_1024x512_mixed", "grad_polar", "z", "mixed", 1024, 512),
        # the symmetry sectors of a block-sparse tensor: many uneven blocks in one call
        _case("batched_qr_300_mixed", "batched_qr", "mix", "mixed", 1024, 1024, 300),
        _case("batched_polar_64_native", "batched_polar", "mix", "native", 768, 768, 64),
        # many small sectors whose work list lives on the device, a launch-bound inner step
        _case("small_qr_400", "small_qr", "f64", "native", 128, 64, 400),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["qr", "qr", "qr_full", "lq", "left_polar", "right_polar", "grad_qr",
                     "grad_polar", "batched_qr", "batched_polar", "small_qr"])
    precision = rng.choice(["native", "mixed"])
    dtype = rng.choice(["f64", "f64", "z", "f32", "c"])
    kappa = 0.0
    count = 1
    if op in ("batched_qr", "batched_polar"):
        dtype = "mix"
        m = n = rng.randint(96, 768)
        count = rng.randint(8, 200 if op == "batched_qr" else 48)
    elif op == "small_qr":
        m, n = rng.randint(8, 150), rng.randint(4, 64)
        count = rng.randint(40, 400)
    else:
        top = {"qr": 6000, "lq": 4100, "qr_full": 2100, "left_polar": 2100, "right_polar": 1500,
               "grad_qr": 1500, "grad_polar": 900}[op]
        m = _log_int(rng, 24, top)
        # in 32 bits the factors of a nearly square Gaussian matrix are themselves ill-conditioned
        n = max(4, int(m * rng.uniform(0.2, 0.75 if dtype in ("f32", "c") else 1.0)))
        if op in ("lq", "right_polar"):
            m, n = n, m
        if op == "left_polar" and rng.random() < 0.5:
            n, kappa = m, 10.0 ** rng.uniform(1.0, 4.0)
            dtype = rng.choice(["f64", "z"])
    return {"op": op, "dtype": dtype, "precision": precision, "m": m, "n": n, "count": count,
            "kappa": kappa}


def _gaussian(gen, m, n, dtype):
    """m x n iid Gaussian (complex: iid real and imaginary parts), column-major."""
    real = torch.float64 if dtype in (torch.float64, torch.complex128) else torch.float32
    if dtype.is_complex:
        x = torch.randn((n, m, 2), generator=gen, device="cuda", dtype=real)
        return torch.view_as_complex(x).t()
    return torch.randn((n, m), generator=gen, device="cuda", dtype=real).t()


def _haar(gen, n, dtype):
    """An n x n orthogonal (unitary) matrix from the QR of a Gaussian one."""
    return torch.linalg.qr(_gaussian(gen, n, n, dtype))[0]


def _graded(gen, n, dtype, kappa):
    """A = U diag(1 .. 1/kappa) V^H, U and V random, the values log-spaced; and (U V^H, V diag V^H)."""
    U, V = _haar(gen, n, dtype), _haar(gen, n, dtype)
    s = torch.logspace(0, -math.log10(kappa), n, device="cuda", dtype=torch.float64)
    return ((U * s) @ V.mH).t().contiguous().t(), (U @ V.mH, (V * s) @ V.mH)


def _shapes(case):
    """Block sizes of a batched case: m_i ~ U{8..m}, n_i ~ U{4..m_i}, the
    first half Float64, the second half ComplexF64 (``small_qr``: U{4..m} x
    U{4..n}, all of the case's type)."""
    g = torch.Generator().manual_seed(1000003 * case["count"] + case["m"])

    def u(lo, hi):
        return int(torch.randint(lo, hi + 1, (1,), generator=g))

    out = []
    for i in range(case["count"]):
        if case["op"] == "small_qr":
            out.append((u(4, max(4, case["m"])), u(4, max(4, case["n"])), case["dtype"]))
        else:
            m = u(8, max(8, case["m"]))
            out.append((m, u(4, m), "f64" if i < case["count"] // 2 else "z"))
    return out


def _flat_outputs(shapes, kind):
    """Output blocks as column-major views of one flat buffer per element
    type, as a block-sparse tensor stores its sectors."""
    flat, at, outs = {}, {}, []
    sizes = []
    for m, n, dt in shapes:
        k = min(m, n)
        sizes.append(((m, k), (k, n)) if kind == "qr" else ((m, n), (n, n)))
    for q in range(2):
        for dt in {s[2] for s in shapes}:
            total = sum(a[q][0] * a[q][1] for a, s in zip(sizes, shapes) if s[2] == dt)
            flat[f"{dt}{q}"] = torch.zeros(total, dtype=DTYPES[dt], device="cuda")
            at[f"{dt}{q}"] = 0
    for a, (m, n, dt) in zip(sizes, shapes):
        pair = []
        for q in range(2):
            key, (r, c) = f"{dt}{q}", a[q]
            pair.append(flat[key][at[key]:at[key] + r * c].view(c, r).t())
            at[key] += r * c
        outs.append(tuple(pair))
    return flat, outs


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    op = case["op"]
    if op in ("batched_qr", "batched_polar", "small_qr"):
        return [_gaussian(gen, m, n, DTYPES[dt]) for m, n, dt in _shapes(case)], None
    m, n, dt = case["m"], case["n"], DTYPES[case["dtype"]]
    A = _graded(gen, n, dt, case["kappa"])[0] if case["kappa"] else _gaussian(gen, m, n, dt)
    if op in GRAD:
        k = min(m, n)
        shapes = ((m, k), (k, n)) if op == "grad_qr" else ((m, n), (n, n))
        return A, tuple(_gaussian(gen, *s, dt) for s in shapes)
    return A, None


def prepare(case, seed):
    A, d = _inputs(case, seed)
    st = {"case": case, "A": A, "d": d}
    op, prec = case["op"], case["precision"]
    st["alg"] = (mak.GB300_PolarNewton(precision=prec) if "polar" in op
                 else mak.GB300_HouseholderQR(precision=prec))
    if op in GRAD:
        st["A"] = A.requires_grad_(True)
    if isinstance(A, list):
        shapes = [(a.shape[0], a.shape[1],
                   next(k for k, v in DTYPES.items() if v == a.dtype)) for a in A]
        st["flat"], st["outs"] = _flat_outputs(shapes, "polar" if "polar" in op else "qr")
    return st


def run(state):
    case, A, alg = state["case"], state["A"], state["alg"]
    op = case["op"]
    if op in SINGLE:
        fn = {"qr": mak.qr_compact, "qr_full": mak.qr_full, "lq": mak.lq_compact,
              "left_polar": mak.left_polar, "right_polar": mak.right_polar}[op]
        return fn(A, alg)
    if op in GRAD:
        fn = mak.autodiff.qr_compact if op == "grad_qr" else mak.autodiff.left_polar
        X, Y = fn(A, alg)
        (dA,) = torch.autograd.grad([X, Y], [A], list(state["d"]))
        return X.detach(), Y.detach(), dA
    fn = {"batched_qr": mak.batched_qr_compact, "batched_polar": mak.batched_left_polar,
          "small_qr": mak.batched_qr_compact_device}[op]
    fn(A, alg, outs=state["outs"])
    return state["flat"]


def _qr_flops(m, n):
    k = min(m, n)
    geqrf = 2.0 * m * n * n - 2.0 * n ** 3 / 3.0 if m >= n else 2.0 * n * m * m - 2.0 * m ** 3 / 3.0
    return geqrf + 2.0 * m * k * k - 2.0 * k ** 3 / 3.0


def _polar_flops(m, n):
    """One QR (m > n), six inverses of the iterate (2 n^3 each), W and P."""
    return (_qr_flops(m, n) + 2.0 * m * n * n if m > n else 0.0) + 14.0 * n ** 3


def work(case):
    """Each input read once and each output written once; the flops of the
    factorization's minimal count (complex counted four times)."""
    op = case["op"]
    shapes = (_shapes(case) if op in ("batched_qr", "batched_polar", "small_qr")
              else [(case["m"], case["n"], case["dtype"])])
    nbytes = flops = 0.0
    for m, n, dt in shapes:
        es = {"f64": 8, "z": 16, "f32": 4, "c": 8}[dt]
        cm = 4.0 if dt in ("z", "c") else 1.0
        k = min(m, n)
        elems = {"qr": m * n + m * k + k * n, "qr_full": 2 * m * n + m * m,
                 "lq": m * n + m * k + k * n, "left_polar": 2 * m * n + n * n,
                 "right_polar": 2 * m * n + m * m, "grad_qr": 2 * (m * n + m * k + k * n),
                 "grad_polar": 4 * m * n + 2 * n * n, "batched_qr": m * n + m * k + k * n,
                 "small_qr": m * n + m * k + k * n, "batched_polar": 2 * m * n + n * n}[op]
        f = {"left_polar": lambda: _polar_flops(m, n), "right_polar": lambda: _polar_flops(n, m),
             "batched_polar": lambda: _polar_flops(m, n),
             "qr_full": lambda: _qr_flops(m, n) + 4.0 * m * (m - k) * k,
             "grad_qr": lambda: _qr_flops(m, n) + 7.0 * m * k * k + k ** 3,
             "grad_polar": lambda: _polar_flops(m, n) + 10.0 * m * n * n + 36.0 * n ** 3,
             }.get(op, lambda: _qr_flops(m, n))()
        nbytes += elems * es
        flops += cm * f
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------ 64-bit values --

def _wide(x):
    return x.to(torch.complex128 if x.is_complex() else torch.float64)


def _qr64(A, mode="reduced"):
    """QR with a real non-negative diagonal of R."""
    Q, R = torch.linalg.qr(_wide(A), mode=mode)
    d = torch.diagonal(R)
    s = torch.where(d.abs() > 0, d / d.abs(), torch.ones_like(d)) if d.is_complex() else \
        torch.where(d < 0, -torch.ones_like(d), torch.ones_like(d))
    k = d.numel()
    Q = Q.clone()
    R = R.clone()
    Q[:, :k] *= s[None, :]
    R[:k] *= s.conj()[:, None]
    return Q, R


def _polar64(A):
    """W, P of A = W P from the singular value decomposition."""
    U, s, Vh = torch.linalg.svd(_wide(A), full_matrices=False)
    return U @ Vh, (Vh.mH * s) @ Vh


def _grad64(op, A, d):
    A = _wide(A.detach())
    d1, d2 = (_wide(x) for x in d)
    if op == "grad_qr":
        Q, R = _qr64(A)
        M = R @ torch.triu(d2).mH - d1.mH @ Q
        M = torch.tril(M, -1)
        D = torch.diagonal(R @ torch.triu(d2).mH - d1.mH @ Q).real
        H = M + M.mH + torch.diag(D).to(A.dtype)
        dA = torch.linalg.solve_triangular(R, (d1 + Q @ H).mH, upper=True).mH
        return Q, R, dA
    W, P = _polar64(A)
    lam, V = torch.linalg.eigh(P)
    dPh = 0.5 * (d2 + d2.mH)
    M = W.mH @ d1 - dPh @ P
    K = V @ ((V.mH @ (M - M.mH) @ V) / (lam[:, None] + lam[None, :])) @ V.mH
    Y = d1 @ (V / lam) @ V.mH
    return W, P, W @ (K + dPh) + Y - W @ (W.mH @ Y)


def _exact(case, seed):
    A, d = _inputs(case, seed)
    op = case["op"]
    if op == "qr":
        return _qr64(A)
    if op == "qr_full":
        Q, R = _qr64(A, "complete")
        # the columns beyond the rank are any basis of the complement
        return (Q if A.shape[0] <= A.shape[1] else None), R
    if op == "lq":
        Q, R = _qr64(A.mH)
        return R.mH, Q.mH
    if op == "left_polar":
        if case["kappa"]:
            gen = torch.Generator(device="cuda").manual_seed(int(seed))
            return _graded(gen, case["n"], DTYPES[case["dtype"]], case["kappa"])[1]
        return _polar64(A)
    if op == "right_polar":
        W, P = _polar64(A.mH)
        return P, W.mH
    if op in GRAD:
        return _grad64(op, A, d)
    flat = {}
    for a in A:
        key = next(k for k, v in DTYPES.items() if v == a.dtype)
        for q, x in enumerate(_polar64(a) if op == "batched_polar" else _qr64(a)):
            flat.setdefault(f"{key}{q}", []).append(x.t().reshape(-1))
    return {k: torch.cat(v) for k, v in flat.items()}


def exact(case, seed):
    def plain(x):
        return x if x is None else x.resolve_conj()

    v = _exact(case, seed)
    return {k: plain(x) for k, x in v.items()} if isinstance(v, dict) else tuple(map(plain, v))
