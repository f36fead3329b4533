"""The work that programs have this library do, as cases that can be timed and checked.

Every case goes through the public entry points of ``rocsolver_b200`` (the C ABI, called with
torch device buffers), on column-major members as the ABI defines them.  The in-place entry
points overwrite their inputs, so a pass of those begins with one device copy of the batch, as
a program that keeps its matrices makes it.

A case is a dict: ``op`` (the call sequence), ``prec`` (s, d, c or z), ``n``, ``batch``,
``nrhs`` and, where the operation has them, ``trans``, ``uplo`` and ``dist`` (the
distribution of the matrices):

* ``lu``       getrf_strided_batched, then getrs_strided_batched
* ``gesv``     gesv_strided_batched
* ``chol``     potrf_strided_batched, then potrs_strided_batched
* ``posv``     posv_batched (pointer arrays)
* ``mixed``    dsgesv_strided_batched (FP32 factorisation, FP64 refinement)
* ``vbatched`` gesv_vbatched: members of different sizes, n the largest, nrhs the largest
* ``adjoint``  getrs_adjoint_strided_batched from factors in hand
* ``inverse``  getri_outofplace_strided_batched from factors in hand
"""
import math

import torch

import rocsolver_b200 as rs

_DT = {"s": torch.float32, "d": torch.float64, "c": torch.complex64, "z": torch.complex128}
_ES = {"s": 4, "d": 8, "c": 8, "z": 16}
_handle = None


def listed():
    return [
        # a few hundred tiny systems in single precision: element-wise solves inside a
        # simulation step, where the launch itself counts
        {"name": "gesv_s_n13", "op": "gesv", "prec": "s", "n": 13, "batch": 300, "nrhs": 2,
         "dist": "dominant"},
        # small dense blocks, one batch that is a single wave on the GPU
        {"name": "lu_d_n32", "op": "lu", "prec": "d", "n": 32, "batch": 1000, "nrhs": 1,
         "trans": "N", "dist": "uniform"},
        # many covariance-sized SPD systems
        {"name": "chol_d_n64", "op": "chol", "prec": "d", "n": 64, "batch": 20000, "nrhs": 4,
         "uplo": "L"},
        # medium SPD systems in single precision, upper triangle, pointer-array batch, an
        # order that is no multiple of a tile
        {"name": "posv_s_n200", "op": "posv", "prec": "s", "n": 200, "batch": 1500, "nrhs": 3,
         "uplo": "U"},
        # the mixed-precision solver on graded matrices, cond 1e1 .. 1e6
        {"name": "mixed_n256", "op": "mixed", "prec": "d", "n": 256, "batch": 2048, "nrhs": 1,
         "dist": "graded"},
        # the same systems through the plain FP64 path
        {"name": "lu_d_n256", "op": "lu", "prec": "d", "n": 256, "batch": 2048, "nrhs": 1,
         "trans": "N", "dist": "graded"},
        # medium general systems in single precision, transposed solve, an odd order
        {"name": "lu_s_n501", "op": "lu", "prec": "s", "n": 501, "batch": 200, "nrhs": 5,
         "trans": "T", "dist": "dominant"},
        # a few large systems: fewer members than the GPU has multiprocessors
        {"name": "lu_d_n2048", "op": "lu", "prec": "d", "n": 2048, "batch": 16, "nrhs": 1,
         "trans": "N", "dist": "uniform"},
        # complex systems (frequency-domain blocks)
        {"name": "gesv_z_n64", "op": "gesv", "prec": "z", "n": 64, "batch": 8192, "nrhs": 1,
         "dist": "uniform"},
        # explicit inverses of small blocks (block preconditioners)
        {"name": "inverse_d_n64", "op": "inverse", "prec": "d", "n": 64, "batch": 16384,
         "nrhs": 0, "dist": "shifted"},
        # members of many different sizes in one call
        {"name": "vbatched_d_512", "op": "vbatched", "prec": "d", "n": 512, "batch": 4096,
         "nrhs": 16, "dist": "vb"},
        # the backward pass of a batched solve
        {"name": "adjoint_d_n128", "op": "adjoint", "prec": "d", "n": 128, "batch": 8192,
         "nrhs": 8, "dist": "shifted"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["small", "small", "chol", "chol", "lu", "lu", "large", "mixed", "complex",
                       "inverse", "vbatched", "adjoint"])
    prec = rng.choice("sd")
    # single precision draws well-conditioned matrices whose pivots are no near ties, so that
    # another correct implementation takes the same ones
    dist = "dominant" if prec == "s" else "uniform"
    if kind == "small":
        n = rng.randint(4, 32)
        c = {"op": rng.choice(["gesv", "lu"]), "prec": prec, "n": n,
             "batch": _log_int(rng, 100, 20000), "nrhs": rng.randint(1, 6), "dist": dist}
        if c["op"] == "lu":
            c["trans"] = rng.choice("NNT")
        return c
    if kind == "chol":
        n = _log_int(rng, 10, 512)
        top = max(4, min(20000, 80_000_000 // (n * n)))
        return {"op": rng.choice(["chol", "posv"]), "prec": prec, "n": n,
                "batch": _log_int(rng, max(2, top // 30), top), "nrhs": rng.randint(1, 8),
                "uplo": rng.choice("LU")}
    if kind in ("lu", "large"):
        n = _log_int(rng, 33, 512) if kind == "lu" else _log_int(rng, 513, 2048)
        # no more elements than 2048 members of n = 256, nor more flops than 16 of n = 2048
        top = min(16000, 134_000_000 // (n * n), int(16 * (2048 / n) ** 3))
        low = max(8, top // 30) if kind == "lu" else 1
        return {"op": "lu", "prec": prec, "n": n, "batch": _log_int(rng, low, max(low, top)),
                "nrhs": rng.randint(1, 8), "trans": rng.choice("NNT"), "dist": dist}
    if kind == "mixed":
        n = _log_int(rng, 40, 500)
        top = min(8000, 134_000_000 // (n * n))
        return {"op": "mixed", "prec": "d", "n": n, "batch": _log_int(rng, max(8, top // 30), top),
                "nrhs": rng.randint(1, 4), "dist": "graded"}
    if kind == "complex":
        prec = rng.choice("cz")
        n = _log_int(rng, 8, 100)
        top = min(16000, 33_000_000 // (n * n))
        return {"op": "gesv", "prec": prec, "n": n, "batch": _log_int(rng, top // 30, top),
                "nrhs": rng.randint(1, 4), "dist": "dominant" if prec == "c" else "uniform"}
    if kind == "inverse":
        n = rng.randint(8, 128)
        top = min(16384, 67_000_000 // (n * n))
        return {"op": "inverse", "prec": prec, "n": n, "batch": _log_int(rng, top // 30, top),
                "nrhs": 0, "dist": "dominant" if prec == "s" else "shifted"}
    if kind == "vbatched":
        return {"op": "vbatched", "prec": prec, "n": rng.randint(40, 512),
                "batch": _log_int(rng, 200, 4096), "nrhs": rng.randint(1, 16), "dist": "vb"}
    n = _log_int(rng, 16, 256)
    top = min(16000, 134_000_000 // (n * n))
    return {"op": "adjoint", "prec": prec, "n": n, "batch": _log_int(rng, top // 30, top),
            "nrhs": rng.randint(1, 16), "dist": "dominant" if prec == "s" else "shifted"}


# ------------------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, shape, dt):
    if dt.is_complex:
        x = torch.rand(*shape, 2, generator=g, device="cuda",
                       dtype=torch.float32 if dt == torch.complex64 else torch.float64)
        return torch.view_as_complex(x.mul_(2).sub_(1))
    return torch.rand(*shape, generator=g, device="cuda", dtype=dt).mul_(2).sub_(1)


def _graded(g, bc, n):
    """U diag(s) V' with orthogonal U and V, s log-spaced from 1 to 1/cond and cond
    log-uniform in [1e1, 1e6] per member.  The orthogonal factors come from a bank of 32,
    row and column signs drawn per member."""
    Q = torch.linalg.qr(torch.randn(64, n, n, generator=g, device="cuda", dtype=torch.float64))[0]
    lk = 1 + 5 * torch.rand(bc, 1, generator=g, device="cuda", dtype=torch.float64)
    t = torch.linspace(0, 1, n, device="cuda", dtype=torch.float64)[None, :]
    iu = torch.randint(0, 32, (bc,), generator=g, device="cuda")
    iv = torch.randint(32, 64, (bc,), generator=g, device="cuda")
    A = torch.empty(bc, n, n, dtype=torch.float64, device="cuda")
    for c0 in range(0, bc, 256):
        k = slice(c0, min(bc, c0 + 256))
        s = torch.pow(10.0, -lk[k] * t)
        torch.bmm(Q[iu[k]] * s[:, None, :], Q[iv[k]], out=A[k])
    sign = torch.randint(0, 2, (2, bc, n), generator=g, device="cuda").to(torch.float64) * 2 - 1
    return A.mul_(sign[0][:, :, None]).mul_(sign[1][:, None, :])


def _matrices(case, g):
    """(batch, n, n): member b is the matrix whose rows are [b, i, :]."""
    n, bc, dt = case["n"], case["batch"], _DT[case["prec"]]
    if case["op"] in ("chol", "posv"):
        G = torch.randn(bc, n, n, generator=g, device="cuda", dtype=dt)
        A = torch.bmm(G, G.transpose(1, 2))
        del G
        A = A.add_(A.transpose(1, 2).clone()).mul_(0.5)
        A.diagonal(dim1=1, dim2=2).add_(n)
        return A
    if case["dist"] == "graded":
        return _graded(g, bc, n)
    A = _uniform(g, (bc, n, n), dt)
    if case["dist"] == "shifted":
        A.diagonal(dim1=1, dim2=2).add_(4)
    elif case["dist"] == "dominant":
        # a large entry in each column, its row drawn at random: interchanges in every column
        rows = torch.rand(bc, n, generator=g, device="cuda").argsort(dim=1)
        big = torch.full((bc, n, 1), 6 + 0.2 * n, device="cuda", dtype=A.real.dtype).to(dt)
        A.scatter_add_(2, rows[:, :, None], big)
    return A


def _vb_sizes(case):
    """The members' sizes: those of the case, whatever the seed of the values."""
    g = _gen(case["n"] * 65536 + case["batch"])
    n = torch.randint(min(8, case["n"]), case["n"] + 1, (case["batch"],), generator=g,
                      device="cuda", dtype=torch.int32)
    r = torch.randint(1, case["nrhs"] + 1, (case["batch"],), generator=g, device="cuda",
                      dtype=torch.int32)
    return n, r


def _offsets(count):
    """Start of each member in a pool of members packed back to back, and the pool's size."""
    end = torch.cumsum(count.to(torch.int64), 0)
    return end - count.to(torch.int64), int(end[-1])


def _vb_pools(case, seed):
    g = _gen(seed)
    dt = _DT[case["prec"]]
    n, r = _vb_sizes(case)
    oa, ta = _offsets(n.to(torch.int64) * n)
    ob, tb = _offsets(n.to(torch.int64) * r)
    op, tp = _offsets(n)
    A, B = _uniform(g, (ta,), dt), _uniform(g, (tb,), dt)
    # 0.1 n on each member's diagonal (single precision: 6 + 0.2 n, see draw())
    which = torch.repeat_interleave(torch.arange(case["batch"], device="cuda"), n.long())
    k = torch.arange(tp, device="cuda") - op[which]
    shift = 0.1 * n.double() if case["prec"] == "d" else 6 + 0.2 * n.double()
    A[oa[which] + k * (n[which] + 1)] += shift[which].to(dt)
    return n, r, (A, oa), (B, ob), (tp, op)


def _buffer(A, B):
    """[A | B] in one allocation, so that a program restores both with one copy; B starts on
    a 512-byte boundary of it."""
    nA = -(-A.numel() // 64) * 64
    src = torch.zeros(nA + B.numel(), dtype=A.dtype, device="cuda")
    src[:A.numel()] = A.reshape(-1)
    src[nA:] = B.reshape(-1)
    work = torch.empty_like(src)
    return src, work, work[:A.numel()].view(A.shape), work[nA:].view(B.shape)


def _call(name, *args):
    rs.check(rs.call("rocsolver_" + name, _handle.value, *args), name)


class State:
    pass


def prepare(case, seed):
    global _handle
    if _handle is None:
        _handle = rs.Handle(torch.cuda.current_stream())
    n, bc, k, p, dt = case["n"], case["batch"], case["nrhs"], case["prec"], _DT[case["prec"]]
    s = State()
    s.case = case
    if case["op"] == "vbatched":
        s.n, s.r, (A, oa), (B, ob), (tp, op) = _vb_pools(case, seed)
        s.src, s.work, s.A, s.B = _buffer(A, B)
        s.ipiv = torch.zeros(tp, dtype=torch.int32, device="cuda")
        s.info = torch.zeros(bc, dtype=torch.int32, device="cuda")
        s.pA = s.A.data_ptr() + oa * _ES[p]
        s.pB = s.B.data_ptr() + ob * _ES[p]
        s.pP = s.ipiv.data_ptr() + op * 4
        return s
    g = _gen(seed)
    A = _matrices(case, g).transpose(1, 2).contiguous()  # column-major members
    s.ipiv = torch.zeros(bc, n, dtype=torch.int32, device="cuda")
    s.info = torch.zeros(bc, dtype=torch.int32, device="cuda")
    if case["op"] in ("adjoint", "inverse"):
        s.A = A
        _call(p + "getrf_strided_batched", n, n, rs.ptr(A), n, n * n, rs.ptr(s.ipiv), n,
              rs.ptr(s.info), bc)
        s.out = torch.empty_like(A)
        if case["op"] == "adjoint":
            s.X = torch.randn(bc, k, n, generator=g, device="cuda", dtype=dt)
            s.G = torch.randn(bc, k, n, generator=g, device="cuda", dtype=dt)
            s.gB = torch.empty_like(s.G)
        return s
    B = _uniform(g, (bc, k, n), dt)
    if case["op"] == "mixed":
        s.A, s.B = A, B
        s.X = torch.empty_like(B)
        s.iter = torch.zeros(bc, dtype=torch.int32, device="cuda")
        return s
    s.src, s.work, s.A, s.B = _buffer(A, B)
    if case["op"] == "posv":
        at = torch.arange(bc, device="cuda", dtype=torch.int64)
        s.pA = s.A.data_ptr() + at * (n * n * _ES[p])
        s.pB = s.B.data_ptr() + at * (n * k * _ES[p])
    return s


def run(s):
    c = s.case
    n, bc, k, p, P = c["n"], c["batch"], c["nrhs"], c["prec"], rs.ptr
    if c["op"] == "adjoint":
        _call(p + "getrs_adjoint_strided_batched", n, k, P(s.A), n, n * n, P(s.ipiv), n, P(s.X),
              n, n * k, P(s.G), n, n * k, P(s.out), n, n * n, P(s.gB), n, n * k, bc)
        return {"gA": s.out, "gB": s.gB}
    if c["op"] == "inverse":
        _call(p + "getri_outofplace_strided_batched", n, P(s.A), n, n * n, P(s.ipiv), n, P(s.out),
              n, n * n, P(s.info), bc)
        return {"inv": s.out, "info": s.info}
    if c["op"] == "mixed":
        _call("dsgesv_strided_batched", n, k, P(s.A), n, n * n, P(s.ipiv), n, P(s.B), n, n * k,
              P(s.X), n, n * k, P(s.iter), P(s.info), bc)
        # the pivots of the FP32 factorisation and the number of corrections follow its
        # rounding, so they are no results to compare
        return {"x": s.X, "info": s.info}
    s.work.copy_(s.src)
    if c["op"] == "vbatched":
        _call(p + "gesv_vbatched", P(s.n), P(s.r), P(s.pA), P(s.n), P(s.pP), P(s.pB), P(s.n),
              P(s.info), n, k, bc)
        return {"lu": s.A, "x": s.B, "ipiv": s.ipiv, "info": s.info}
    if c["op"] == "lu":
        _call(p + "getrf_strided_batched", n, n, P(s.A), n, n * n, P(s.ipiv), n, P(s.info), bc)
        _call(p + "getrs_strided_batched", rs.OP_T if c["trans"] == "T" else rs.OP_N, n, k, P(s.A),
              n, n * n, P(s.ipiv), n, P(s.B), n, n * k, bc)
        return {"lu": s.A, "x": s.B, "ipiv": s.ipiv, "info": s.info}
    if c["op"] == "gesv":
        _call(p + "gesv_strided_batched", n, k, P(s.A), n, n * n, P(s.ipiv), n, P(s.B), n, n * k,
              P(s.info), bc)
        return {"lu": s.A, "x": s.B, "ipiv": s.ipiv, "info": s.info}
    fill = rs.FILL_LOWER if c["uplo"] == "L" else rs.FILL_UPPER
    if c["op"] == "chol":
        _call(p + "potrf_strided_batched", fill, n, P(s.A), n, n * n, P(s.info), bc)
        _call(p + "potrs_strided_batched", fill, n, k, P(s.A), n, n * n, P(s.B), n, n * k, bc)
    else:
        _call(p + "posv_batched", fill, n, k, P(s.pA), n, P(s.pB), n, P(s.info), bc)
    return {"factor": s.A, "x": s.B, "info": s.info}


# ------------------------------------------------------------- what a pass cannot do without
def work(case):
    n, bc, k, p = case["n"], case["batch"], case["nrhs"], case["prec"]
    es, f = _ES[p], 4 if p in "cz" else 1
    op = case["op"]
    if op == "vbatched":
        lo = min(8, n)
        sizes = range(lo, n + 1)
        n2 = sum(i * i for i in sizes) / len(sizes)
        n3 = sum(i ** 3 for i in sizes) / len(sizes)
        n1, kk = (lo + n) / 2, (1 + k) / 2
        return {"bytes": bc * (2 * n2 * es + 2 * n1 * kk * es + 4 * n1 + 4),
                "flops": bc * (2 * n3 / 3 + 2 * n2 * kk)}
    if op in ("lu", "gesv"):
        return {"bytes": bc * (2 * n * n * es + 2 * n * k * es + 4 * n + 4),
                "flops": f * bc * (2 * n ** 3 / 3 + 2 * n * n * k)}
    if op in ("chol", "posv"):
        return {"bytes": bc * (n * (n + 1) * es + 2 * n * k * es + 4),
                "flops": bc * (n ** 3 / 3 + 2 * n * n * k)}
    if op == "mixed":
        return {"bytes": bc * (n * n * es + 2 * n * k * es + 4 * n + 8),
                "flops": bc * (2 * n ** 3 / 3 + 2 * n * n * k)}
    if op == "inverse":
        return {"bytes": bc * (2 * n * n * es + 4 * n + 4), "flops": f * bc * 4 * n ** 3 / 3}
    return {"bytes": bc * (2 * n * n * es + 3 * n * k * es + 4 * n), "flops": bc * 4 * n * n * k}


def tolerance(case):
    # the largest errors against 64 bits (torch's own LU of the same inputs) were 6.4e-7 in
    # single and 7.1e-11 in double precision; the latter is the worst-conditioned member's
    if case["prec"] in "sc":
        return {"rel": 5e-6, "max": 5e-4, "differ": 0.0}
    return {"rel": 5e-10, "max": 1e-6, "differ": 0.0}


# ------------------------------------------------------------------------------ in 64 bits


def exact(case, seed):
    n, bc, k, op = case["n"], case["batch"], case["nrhs"], case["op"]
    wide = torch.complex128 if case["prec"] in "cz" else torch.float64
    if op == "vbatched":
        sizes, rhs, (A, oa), (B, ob), _ = _vb_pools(case, seed)
        lu, x = A.to(wide), B.to(wide)
        sizes, rhs = sizes.long(), rhs.long()
        order = torch.argsort(sizes).tolist()
        for c0 in range(0, bc, 128):  # members of like sizes, padded with the identity
            ids = torch.tensor(order[c0:c0 + 128], device="cuda")
            top, kt = int(sizes[ids].max()), int(rhs[ids].max())
            at = torch.arange(top, device="cuda")
            sz, rr = sizes[ids][:, None, None], rhs[ids][:, None, None]
            col, row = at[None, :, None], at[None, None, :]  # member-major, column, row
            inside = (col < sz) & (row < sz)
            idx = (oa[ids][:, None, None] + col * sz + row)[inside]
            M = torch.eye(top, dtype=wide, device="cuda").repeat(len(ids), 1, 1)
            M[inside] = lu[idx]
            cb = torch.arange(kt, device="cuda")[None, :, None]
            inb = (cb < rr) & (row < sz)
            idb = (ob[ids][:, None, None] + cb * sz + row)[inb]
            R = torch.zeros(len(ids), kt, top, dtype=wide, device="cuda")
            R[inb] = x[idb]
            F, piv = torch.linalg.lu_factor(M.transpose(1, 2))
            x[idb] = torch.linalg.lu_solve(F, piv, R.transpose(1, 2)).transpose(1, 2)[inb]
            lu[idx] = F.transpose(1, 2)[inside]
        return {"lu": lu, "x": x, "ipiv": None, "info": None}
    g = _gen(seed)
    A = _matrices(case, g)
    if op == "inverse":
        return {"inv": torch.linalg.inv(A.to(wide)).transpose(1, 2).contiguous(), "info": None}
    if op == "adjoint":
        dt = _DT[case["prec"]]
        X = torch.randn(bc, k, n, generator=g, device="cuda", dtype=dt).to(wide)
        G = torch.randn(bc, k, n, generator=g, device="cuda", dtype=dt).to(wide)
        gB = torch.linalg.solve(A.to(wide).transpose(1, 2), G.transpose(1, 2))  # (bc, n, k)
        # column-major members: [b, j, i] = gA(i, j) = -sum_k gB(i, k) X(j, k)
        return {"gA": -torch.bmm(X.transpose(1, 2), gB.transpose(1, 2)),
                "gB": gB.transpose(1, 2).contiguous()}
    B = _uniform(g, (bc, k, n), _DT[case["prec"]]).to(wide).transpose(1, 2)
    if op == "mixed":
        return {"x": torch.linalg.solve(A, B).transpose(1, 2).contiguous(), "info": None}
    A = A.to(wide)
    if op in ("lu", "gesv"):
        LU, piv = torch.linalg.lu_factor(A)
        X = torch.linalg.lu_solve(LU, piv, B, adjoint=case.get("trans") == "T")
        return {"lu": LU.transpose(1, 2).contiguous(), "x": X.transpose(1, 2).contiguous(),
                "ipiv": None, "info": None}
    L = torch.linalg.cholesky(A)
    X = torch.cholesky_solve(B, L).transpose(1, 2).contiguous()
    # the other triangle keeps A's entries; [b, j, i] is entry (i, j)
    if case["uplo"] == "L":
        F = L.tril() + A.triu(1)
    else:
        F = L.transpose(1, 2).triu() + A.tril(-1)
    return {"factor": F.transpose(1, 2).contiguous(), "x": X, "info": None}
