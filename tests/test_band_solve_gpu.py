"""Band solver: the one-launch block steps for few right-hand sides give the bits of the GEMM route that
serves more of them, so a sweep's columns do not depend on how many are solved at once; and small and
narrow bands (one block, one panel, bandwidth below and above a block) agree with SuperLU."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

from staccato_b200.krylov import fom_sweep
from staccato_b200.project import DeviceCsr

pytestmark = pytest.mark.gpu


def _banded(n, bw, rng):
    diags = [np.full(n, 6.0 + 1.0j)]
    offs = [0]
    for d in sorted({1, bw // 2, bw} - {0}):
        if d < n:
            v = rng.standard_normal(n - d) + 0.1j * rng.standard_normal(n - d)
            diags += [v, v]
            offs += [d, -d]
    return sp.diags(diags, offs, shape=(n, n), format="csr")


@pytest.mark.parametrize("n,bw", [(1, 0), (40, 3), (64, 10), (65, 64), (200, 63), (700, 130), (1500, 400)])
def test_route_by_right_hand_sides_gives_the_same_bits(handle, n, bw):
    import torch

    rng = np.random.default_rng(n + bw)
    K = _banded(n, bw, rng)
    K.sort_indices()
    M = K.copy()
    M.data = 1e-3 * (rng.standard_normal(K.nnz) + 0j)
    M = (0.5 * (M + M.T)).tocsr()
    M.sort_indices()
    assert np.array_equal(M.indices, K.indices)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.complex128)).cuda()
    csr = DeviceCsr.from_host(K.indptr, K.indices)
    F = rng.standard_normal((18, n)) + 1j * rng.standard_normal((18, n))
    freqs = [0.3, 1.1]
    wide = fom_sweep(handle, csr, t(K.data), t(M.data), None, t(F), freqs)
    A = [(K - (2 * np.pi * f) ** 2 * M).tocsc() for f in freqs]
    for r in (1, 3, 8, 9, 16):
        few = fom_sweep(handle, csr, t(K.data), t(M.data), None, t(F[:r]), freqs)
        assert np.array_equal(few.cpu().numpy(), wide[:, :r].cpu().numpy()), r
    for f in range(2):
        x = spla.spsolve(A[f], F.T) if n > 1 else F.T / A[f].toarray()[0, 0]
        assert np.abs(wide[f].cpu().numpy().T - x).max() <= 1e-9 * np.abs(x).max()
