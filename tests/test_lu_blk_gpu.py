"""The blocked LU (64-column steps in separate launches: panel, interchanges with U12, trailing
update, L's rows) against the oracle at the sizes where it can go wrong: one column more or
less than a panel, every CTA row count and cluster size of the panel kernel, rectangular
members, padded and odd leading dimensions, tied pivots, infinities and NaN.  With a few
members the built-in choice takes it for FP64 above 512 rows (whose later panels have every
smaller row count) and for FP32 at most sizes; the FP64 cases of up to 512 rows check the same
properties of the CTA kernels that run there."""
import numpy as np
import pytest

import rocsolver_b200 as rs
from tests.gpu_util import GpuHandle, dev, host, ptr
from tests.norms import lu_backward_error
from tests.refcases import from_colmajor, to_colmajor, uniform_general
from tests.test_lu_gpu import check_getrf, gpu_getrf, oracle_getrf

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def handle():
    h = GpuHandle()
    yield h.value
    h.close()


@pytest.fixture(autouse=True)
def no_table():
    """Without tuning entries the built-in choice runs."""
    old = rs.tuning_table()
    assert rs.set_tuning_table("") == rs.SUCCESS
    yield
    assert rs.set_tuning_table(old) == rs.SUCCESS


SIZES = [(33, 33), (64, 64), (65, 65), (64, 130), (130, 64), (127, 127), (129, 129), (256, 256),
         (257, 257), (300, 72), (512, 512), (513, 200), (1024, 1024), (1025, 90), (2048, 130)]


@pytest.mark.parametrize("m,n", SIZES)
@pytest.mark.parametrize("pad", [0, 3])
def test_blocked_getrf(handle, m, n, pad):
    A = uniform_general(m, n, 2, seed=m * 7 + n)
    LU, ipiv, info, _ = gpu_getrf(handle, A, lda=m + pad)
    check_getrf(A, LU, ipiv, info)


@pytest.mark.parametrize("m,n", [(513, 513), (577, 577), (640, 640), (600, 1300), (700, 400)])
@pytest.mark.parametrize("pad", [0, 3])
def test_blocked_dgetrf_above_512_rows(handle, m, n, pad):
    """A last panel of 1, 1, 64 and 24 columns and a wide member, FP64."""
    A = uniform_general(m, n, 2, seed=m * 7 + n)
    LU, ipiv, info, _ = gpu_getrf(handle, A, lda=m + pad)
    check_getrf(A, LU, ipiv, info)


def _dominant32(m, n, bc, seed):
    """uniform[-1, 1] with one large entry per column (the rows drawn at random), so that FP32
    rounding decides no pivot"""
    A = uniform_general(m, n, bc, seed=seed)
    rng = np.random.default_rng(seed)
    for b in range(bc):
        k = min(m, n)
        A[b, rng.permutation(m)[:k], np.arange(k)] += 6 + 0.2 * n
    return A.astype(np.float32)


@pytest.mark.parametrize("m,n", [(20, 100), (32, 33), (33, 33), (64, 64), (33, 100), (64, 130),
                                 (97, 97), (127, 127), (128, 300), (161, 161), (256, 256),
                                 (257, 257), (320, 320), (512, 512), (513, 300), (1025, 600)])
@pytest.mark.parametrize("pad", [0, 3])
def test_blocked_sgetrf_sizes(handle, m, n, pad):
    A = _dominant32(m, n, 2, seed=m * 7 + n)
    LU, ipiv, info, _ = gpu_getrf(handle, A, lda=m + pad)
    check_getrf(A, LU, ipiv, info)


@pytest.mark.parametrize("prec,n", [("d", 1500), ("d", 2048), ("s", 2048), ("t", 2048)])
def test_blocked_getrf_large_square(handle, prec, n):
    """The longest trailing sweep: 24 and 32 panels, clusters of 8 down to single CTAs, L's rows
    with the most interchanges, an odd leading dimension."""
    if prec == "d":
        A = uniform_general(n, n, 1, seed=n)
    else:
        A = _dominant32(n, n, 1, seed=n)
    if prec != "t":
        LU, ipiv, info, _ = gpu_getrf(handle, A, lda=n + 1)
        check_getrf(A, LU, ipiv, info)
        return
    dA = dev(to_colmajor(A, n + 1))
    dP, dI = dev(np.zeros(n, np.int32)), dev(np.full(1, -7, np.int32))
    st = rs.call("rocsolver_sgetrf_tf32_strided_batched", handle, n, n, ptr(dA), n + 1,
                 (n + 1) * n, ptr(dP), n, ptr(dI), 1)
    assert st == rs.SUCCESS
    LU = from_colmajor(host(dA), 1, n, n, n + 1, (n + 1) * n)[0].astype(np.float64)
    _, oipiv, oinfo = oracle_getrf(A)
    np.testing.assert_array_equal(host(dI), oinfo)
    np.testing.assert_array_equal(host(dP), oipiv[0])
    be = lu_backward_error(A[0].astype(np.float64), LU, host(dP))
    assert be / (n * np.finfo(np.float32).eps) < 10


@pytest.mark.parametrize("m,n", [(65, 65), (200, 330), (600, 600)])
def test_blocked_getrf_npvt_and_pointer_batch(handle, m, n):
    A = uniform_general(m, n, 2, seed=m) + 2 * max(m, n) * np.eye(m, n)
    LU, ipiv, info, _ = gpu_getrf(handle, A, pivot=False)
    check_getrf(A, LU, ipiv, info, pivot=False)
    LU, ipiv, info, _ = gpu_getrf(handle, A[:, ::-1].copy(), batched=True)
    check_getrf(A[:, ::-1].copy(), LU, ipiv, info)


@pytest.mark.parametrize("n", [64, 70, 300, 520])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_blocked_getrf_ties_and_zero_columns(handle, n, dtype):
    """Entries -1, 0, 1: columns full of equal candidates (the smallest row position wins, in
    the lane, across lanes, warps and CTAs); a zero column sets info."""
    rng = np.random.default_rng(n)
    A = rng.integers(-1, 2, (3, n, n)).astype(dtype)
    A[1][:, n // 2] = 0.0
    LU, ipiv, info, _ = gpu_getrf(handle, A)
    oLU, oipiv, oinfo = oracle_getrf(A)
    # elimination of small integers is exact only at first: ties are decided alike while the
    # values are, so the first panel's pivots are compared
    k = 8
    np.testing.assert_array_equal(ipiv.reshape(3, n)[:, :k], oipiv[:, :k])
    # and the factors multiply back to the permuted matrix
    for b in range(3):
        F = LU[b].astype(np.float64)
        L = np.tril(F, -1) + np.eye(n)
        R = L @ np.triu(F)
        P = A[b].copy()
        for i, p in enumerate(ipiv.reshape(3, n)[b]):
            P[[i, p - 1]] = P[[p - 1, i]]
        assert np.abs(R - P).max() <= n * np.finfo(dtype).eps * np.abs(L).sum(1).max() \
            * np.abs(F).max()
    assert info[1] == oinfo[1] != 0


@pytest.mark.parametrize("n,dtype", [(64, np.float64), (200, np.float64), (400, np.float64),
                                     (600, np.float64), (64, np.float32), (256, np.float32),
                                     (400, np.float32), (600, np.float32)])
def test_blocked_getrf_nan_and_inf(handle, n, dtype):
    """A NaN below the diagonal never wins the search, a NaN on it is kept; an infinity wins;
    entries that they do not reach stay finite (compared with the oracle up to the column
    where the first of them is eliminated)."""
    A = uniform_general(n, n, 3, seed=n).astype(dtype)
    A[0][n - 1, 0] = np.nan
    A[1][0, 0] = np.nan
    A[2][n // 2, 1] = np.inf
    LU, ipiv, info, _ = gpu_getrf(handle, A)
    oLU, oipiv, oinfo = oracle_getrf(A)
    np.testing.assert_array_equal(ipiv.reshape(3, n)[:, :2], oipiv[:, :2])
    for b in range(3):
        np.testing.assert_array_equal(np.isnan(LU[b][:, :2]), np.isnan(oLU[b][:, :2]))
    # the first row of U is the pivot row as it was
    np.testing.assert_array_equal(LU[0][:1], oLU[0][:1])


@pytest.mark.parametrize("m,n", [(64, 64), (129, 129), (300, 300), (520, 130), (1030, 70)])
def test_blocked_sgetrf(handle, m, n):
    A = (uniform_general(m, n, 2, seed=n) + (6 + 0.2 * n) * np.eye(m, n)).astype(np.float32)
    A = A[:, ::-1].copy()
    LU, ipiv, info, _ = gpu_getrf(handle, A)
    check_getrf(A, LU, ipiv, info)


WAIT_CHILD = r'''
import ctypes, os, sys
import numpy as np
import torch
sys.path.insert(0, ROOT)
import oracle
import rocsolver_b200 as rs
from tests.refcases import to_colmajor, uniform_general
assert rs.LIB_PATH.endswith("_checked.so"), rs.LIB_PATH
h = rs.Handle(torch.cuda.current_stream().cuda_stream)
P = rs.ptr
rec = (ctypes.c_int32 * 4)()
GUARD, SENT, bc = 4096, -12345, 3
for p, n in (("s", 300), ("s", 600), ("s", 1100), ("d", 600), ("d", 1100)):
    dt, lda = np.float32 if p == "s" else np.float64, n + 3
    A = (uniform_general(n, n, bc, seed=n) + 2 * n * np.eye(n)).astype(dt)[:, ::-1].copy()
    flat = to_colmajor(A, lda).reshape(-1)
    guard = np.full(GUARD, SENT, dt)
    pad = np.ones((bc, n, lda), bool)
    pad[:, :, :n] = False
    for limit in ("0", "1", "3", None):
        if limit is None:
            del os.environ["ROCSOLVER_B200_CLUSTER_WAIT"]
        else:
            os.environ["ROCSOLVER_B200_CLUSTER_WAIT"] = limit
        dA = torch.from_numpy(np.concatenate([guard, flat, guard])).cuda()
        dP = torch.full((GUARD + bc * n + GUARD,), SENT, dtype=torch.int32, device="cuda")
        dI = torch.full((GUARD + bc + GUARD,), SENT, dtype=torch.int32, device="cuda")
        B = uniform_general(n, 2, bc, seed=5).astype(dt)
        dB = torch.from_numpy(to_colmajor(B)).cuda()
        B0 = dB.clone()
        rs.check(rs.call(f"rocsolver_{p}gesv_strided_batched", h.value, n, 2, P(dA[GUARD:]), lda,
                         lda * n, P(dP[GUARD:]), n, P(dB), n, 2 * n, P(dI[GUARD:]), bc), "gesv")
        torch.cuda.synchronize()
        rs.call("rocsolver_b200_bounds_check", ctypes.cast(rec, ctypes.c_void_p))
        assert rec[0] == 0, (p, n, limit, list(rec))
        a, ip, info = dA.cpu().numpy(), dP.cpu().numpy(), dI.cpu().numpy()
        for x in (a, ip, info):
            assert (x[:GUARD] == SENT).all() and (x[-GUARD:] == SENT).all(), (p, n, limit)
        a, ip, info = a[GUARD:-GUARD], ip[GUARD:-GUARD].reshape(bc, n), info[GUARD:-GUARD]
        assert np.isnan(a.reshape(bc, n, lda)[pad]).all()  # to_colmajor pads with NaN
        assert (ip >= np.arange(1, n + 1)).all() and (ip <= n).all(), (p, n, limit)
        gave_up = info == np.iinfo(np.int32).min
        print(p, n, limit, "members given up", int(gave_up.sum()), flush=True)
        assert ((info == 0) | gave_up).all(), (p, n, limit, info)
        if limit == "0":
            assert gave_up.all()
        if limit is None:
            assert not gave_up.any()
        oA, oP, oI = to_colmajor(A).copy(), np.zeros(bc * n, np.int32), np.zeros(bc, np.int32)
        oracle.getrf(n, n, oA, n, n * n, oP, n, oI, bc, nthreads=oracle.nthreads_default())
        for b in range(bc):
            if gave_up[b]:
                assert torch.equal(dB.view(bc, -1)[b], B0.view(bc, -1)[b])
            else:
                assert (ip[b] == oP.reshape(bc, n)[b]).all()
                x = dB.view(bc, 2, n)[b].cpu().numpy().astype(np.float64).T
                r = np.abs(A[b].astype(np.float64) @ x - B[b]).max()
                assert r <= n * np.finfo(dt).eps * (np.abs(A[b]).sum(1).max() * np.abs(x).max())
h.close()
print("waits done")
'''


def test_cluster_wait_that_runs_out():
    """A wait between the CTAs of a panel's cluster that runs out ends in info = INT_MIN, pivots
    in range, the right-hand sides of gesv as they were, and nothing written outside the member
    (the checked build: limits of 0, 1 and 3 polls, so that the CTAs give up at different
    columns); the call after it, with the usual limit, is right."""
    import os
    import subprocess
    import sys
    if not os.path.exists(rs.CHECKED_LIB_PATH):
        pytest.skip("bounds-checked library not built (python -m rocsolver_b200.build --checked)")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, ROCSOLVER_B200_LIB=rs.CHECKED_LIB_PATH,
               ROCSOLVER_B200_CLUSTER_WAIT="0")
    r = subprocess.run([sys.executable, "-c", "ROOT = " + repr(root) + "\n" + WAIT_CHILD], env=env,
                       capture_output=True, text=True, timeout=600, cwd=root)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    assert "waits done" in r.stdout


@pytest.mark.parametrize("fn,prec,n,bc", [("getrf", "d", 600, 2), ("getrf", "s", 200, 3),
                                          ("getrf", "s", 65, 3), ("potrf", "d", 200, 3)])
def test_blocked_calls_in_a_captured_graph(fn, prec, n, bc):
    """The launches of a blocked call captured in a CUDA graph: the replay on other values gives
    the direct call's bits."""
    import torch
    dt = torch.float64 if prec == "d" else torch.float32
    g = torch.Generator(device="cuda").manual_seed(n)
    A0 = torch.rand(2, bc, n, n, dtype=dt, device="cuda", generator=g)
    A0 = A0 + A0.transpose(2, 3) + 2 * n * torch.eye(n, dtype=dt, device="cuda")
    src, A = A0[0].clone(), torch.empty_like(A0[0])
    ipiv = torch.zeros(bc, n, dtype=torch.int32, device="cuda")
    info = torch.zeros(bc, dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    h = rs.Handle(stream.cuda_stream)

    def call():
        A.copy_(src)
        if fn == "getrf":
            st = rs.call(f"rocsolver_{prec}getrf_strided_batched", h.value, n, n, ptr(A), n, n * n,
                         ptr(ipiv), n, ptr(info), bc)
        else:
            st = rs.call(f"rocsolver_{prec}potrf_strided_batched", h.value, rs.FILL_UPPER, n,
                         ptr(A), n, n * n, ptr(info), bc)
        rs.check(st, fn)

    try:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            call()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            call()
        src.copy_(A0[1])
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        got = (A.clone(), ipiv.clone(), info.clone())
        with torch.cuda.stream(stream):
            call()
        torch.cuda.synchronize()
        for x, y in zip(got, (A, ipiv, info)):
            assert torch.equal(x, y)
        assert not info.any()
    finally:
        h.close()
