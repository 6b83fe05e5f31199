"""Projection and Gram-Schmidt at the edges of their tensor-core tiles: node patterns (three rows of equal
columns) and rows without one in the same matrix, basis widths around the 16- and 48-column limits, odd widths,
row counts that are no multiple of a chunk, unaligned and odd leading dimensions."""
import numpy as np
import pytest
import scipy.sparse as sp

from staccato_b200.project import DeviceCsr, orthonormalize, project

pytestmark = pytest.mark.gpu


def _matrices(nodes, extra, rng, mats):
    """3 nodes DOFs with node patterns (0 to 70 neighbours), then `extra` rows of their own pattern."""
    n = 3 * nodes + extra
    rows, cols = [], []
    for i in range(nodes):
        nb = rng.choice(n, size=max(int(rng.integers(0, min(71, n))), int(i == 0)), replace=False)  # not all empty
        for r in range(3):
            rows += [3 * i + r] * len(nb)
            cols += list(nb)
    for i in range(3 * nodes, n):
        nb = rng.choice(n, size=int(rng.integers(1, min(40, n))), replace=False)
        rows += [i] * len(nb)
        cols += list(nb)
    pat = sp.csr_matrix((np.ones(len(rows)), (rows, cols)), shape=(n, n))
    pat.sort_indices()
    out = []
    for _ in range(mats):
        a = pat.copy()
        a.data = rng.standard_normal(a.nnz)
        out.append(a)
    return out


@pytest.mark.parametrize("mats", [1, 2, 3])
@pytest.mark.parametrize("nodes,extra,k", [(1, 0, 2), (40, 0, 16), (41, 2, 18), (100, 1, 32), (33, 5, 34), (70, 0, 47),
                                           (70, 3, 48), (64, 2, 50), (50, 1, 97), (45, 4, 130)])
def test_projection_tiles(handle, nodes, extra, k, mats):
    import torch

    rng = np.random.default_rng(nodes * 1000 + k + mats)
    A = _matrices(nodes, extra, rng, mats)
    n = A[0].shape[0]
    V = rng.standard_normal((n, k))
    csr = DeviceCsr.from_host(A[0].indptr, A[0].indices)
    R = project(handle, csr, [torch.from_numpy(a.data).cuda() for a in A], torch.from_numpy(np.ascontiguousarray(V.T)).cuda())
    for a, r in zip(A, R):
        ref = V.T @ (a @ V)
        scale = np.abs(V).T @ (abs(a) @ np.abs(V))
        # the longest sum has n terms after 70: a bound of 4 n eps on the sum of moduli
        assert (np.abs(r.cpu().numpy() - ref) <= 4 * n * np.finfo(float).eps * scale).all()


# last windows of every number of 8-column bands after a full 128-column one (three matrices and five bands, k = 161 to
# 168, took more threads than the kernel may have)
@pytest.mark.parametrize("mats,k", [(3, 129), (3, 144), (3, 152), (3, 160), (3, 161), (3, 165), (3, 168), (3, 169), (3, 184),
                                    (3, 200), (3, 216), (3, 232), (3, 248), (3, 256), (3, 293), (2, 165), (1, 165)])
def test_projection_windows(handle, mats, k):
    test_projection_tiles(handle, 37, 2, k, mats)


@pytest.mark.parametrize("n,k,passes", [(5, 5, 2), (33, 7, 2), (64, 32, 2), (127, 33, 2), (1001, 40, 3), (4096, 96, 2),
                                        (2000, 129, 2), (3333, 200, 2)])
def test_orthonormalize_tiles(handle, n, k, passes):
    import torch

    rng = np.random.default_rng(n + k)
    V = rng.standard_normal((n, k)) + 0.3 * rng.standard_normal((n, 1))
    Vd = torch.from_numpy(np.ascontiguousarray(V.T)).cuda()
    orthonormalize(handle, Vd, passes)
    Q = Vd.cpu().numpy().T
    assert np.abs(Q.T @ Q - np.eye(k)).max() <= 1e-13 * max(1.0, k / 32)
    q, r = np.linalg.qr(V)
    q = q * np.sign(np.diag(r))
    assert np.abs(Q - q).max() <= 1e-12 * np.linalg.cond(V)


# a zero column in a panel: it and the panel's later columns come out non-finite, the columns before it are untouched
@pytest.mark.parametrize("n,k,zero", [(500, 32, 20), (500, 32, 31), (777, 30, 1), (300, 17, 16), (1000, 70, 52), (4000, 96, 95),
                                      (640, 64, 33)])
def test_orthonormalize_keeps_the_columns_before_a_dependent_one(handle, n, k, zero):
    import torch

    rng = np.random.default_rng(zero)
    V = rng.standard_normal((n, k)) + 0.3 * rng.standard_normal((n, 1))
    V[:, zero] = 0.0
    Vd = torch.from_numpy(np.ascontiguousarray(V.T)).cuda()
    orthonormalize(handle, Vd, 2)
    Q = Vd.cpu().numpy().T
    assert not np.isfinite(Q[:, zero]).any()
    Q = Q[:, :zero]
    assert np.isfinite(Q).all()
    assert np.abs(Q.T @ Q - np.eye(zero)).max() <= 1e-13 * max(1.0, k / 32)
    q, r = np.linalg.qr(V[:, :zero])
    q = q * np.sign(np.diag(r))
    assert np.abs(Q - q).max() <= 1e-12 * np.linalg.cond(V[:, :zero])


# columns of very small and very large norm: their squares stay in range, the reciprocals of the squares need not
@pytest.mark.parametrize("scale", [1e-157, 1e-155, 1e-150, 1e150])
def test_orthonormalize_range(handle, scale):
    import torch

    rng = np.random.default_rng(7)
    n, k = 900, 40
    V = rng.standard_normal((n, k)) + 0.3 * rng.standard_normal((n, 1))
    Vd = torch.from_numpy(np.ascontiguousarray(scale * V.T)).cuda()
    orthonormalize(handle, Vd, 2)
    Q = Vd.cpu().numpy().T
    assert np.abs(Q.T @ Q - np.eye(k)).max() <= 1e-13 * max(1.0, k / 32)
    q, r = np.linalg.qr(V)
    q = q * np.sign(np.diag(r))
    # the first pass works on squares that have lost digits at 1e-157 (subnormal, n scale^2 = 9e-312: 5e-13 of one)
    tol = 1e-12 if scale > 1e-154 else 1e-12 + 900 * 2.0 ** -1074 / scale ** 2
    assert np.abs(Q - q).max() <= tol * np.linalg.cond(V)
