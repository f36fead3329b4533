"""The blocked LU (64-column steps in separate launches: panel, interchanges with U12, trailing
update, L's rows) against the oracle at the sizes where it can go wrong: one column more or
less than a panel, every CTA row count and cluster size of the panel kernel, rectangular
members, padded and odd leading dimensions, tied pivots, infinities and NaN."""
import numpy as np
import pytest

import rocsolver_b200 as rs
from tests.gpu_util import GpuHandle
from tests.refcases import uniform_general
from tests.test_lu_gpu import check_getrf, gpu_getrf, oracle_getrf

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def handle():
    h = GpuHandle()
    yield h.value
    h.close()


@pytest.fixture(autouse=True)
def no_table():
    """Without tuning entries every m > 32 takes the blocked path."""
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


@pytest.mark.parametrize("m,n", [(65, 65), (200, 330), (600, 600)])
def test_blocked_getrf_npvt_and_pointer_batch(handle, m, n):
    A = uniform_general(m, n, 2, seed=m) + 2 * max(m, n) * np.eye(m, n)
    LU, ipiv, info, _ = gpu_getrf(handle, A, pivot=False)
    check_getrf(A, LU, ipiv, info, pivot=False)
    LU, ipiv, info, _ = gpu_getrf(handle, A[:, ::-1].copy(), batched=True)
    check_getrf(A[:, ::-1].copy(), LU, ipiv, info)


@pytest.mark.parametrize("n", [64, 70, 300, 520])
def test_blocked_getrf_ties_and_zero_columns(handle, n):
    """Entries -1, 0, 1: columns full of equal candidates (the smallest row position wins, in
    the lane, across lanes, warps and CTAs); a zero column sets info."""
    rng = np.random.default_rng(n)
    A = rng.integers(-1, 2, (3, n, n)).astype(np.float64)
    A[1][:, n // 2] = 0.0
    LU, ipiv, info, _ = gpu_getrf(handle, A)
    oLU, oipiv, oinfo = oracle_getrf(A)
    # elimination of small integers is exact only at first: ties are decided alike while the
    # values are, so the first panel's pivots are compared
    k = 8
    np.testing.assert_array_equal(ipiv.reshape(3, n)[:, :k], oipiv[:, :k])
    # and the factors multiply back to the permuted matrix
    for b in range(3):
        L = np.tril(LU[b], -1) + np.eye(n)
        R = L @ np.triu(LU[b])
        P = A[b].copy()
        for i, p in enumerate(ipiv.reshape(3, n)[b]):
            P[[i, p - 1]] = P[[p - 1, i]]
        assert np.abs(R - P).max() <= n * np.finfo(float).eps * np.abs(L).sum(1).max() \
            * np.abs(LU[b]).max()
    assert info[1] == oinfo[1] != 0


@pytest.mark.parametrize("n", [64, 200, 400])
def test_blocked_getrf_nan_and_inf(handle, n):
    """A NaN below the diagonal never wins the search, a NaN on it is kept; an infinity wins;
    entries that they do not reach stay finite (compared with the oracle up to the column
    where the first of them is eliminated)."""
    A = uniform_general(n, n, 3, seed=n)
    A[0][n - 1, 0] = np.nan
    A[1][0, 0] = np.nan
    A[2][n // 2, 1] = np.inf
    LU, ipiv, info, _ = gpu_getrf(handle, A)
    oLU, oipiv, oinfo = oracle_getrf(A)
    np.testing.assert_array_equal(ipiv.reshape(3, n)[:, :2], oipiv[:, :2])
    for b in range(3):
        np.testing.assert_array_equal(np.isnan(LU[b][:, :2]), np.isnan(oLU[b][:, :2]))
    np.testing.assert_allclose(LU[0][:1], oLU[0][:1], rtol=1e-13)


@pytest.mark.parametrize("m,n", [(64, 64), (129, 129), (300, 300), (520, 130), (1030, 70)])
def test_blocked_sgetrf(handle, m, n):
    A = (uniform_general(m, n, 2, seed=n) + (6 + 0.2 * n) * np.eye(m, n)).astype(np.float32)
    A = A[:, ::-1].copy()
    LU, ipiv, info, _ = gpu_getrf(handle, A)
    check_getrf(A, LU, ipiv, info)
