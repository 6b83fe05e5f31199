"""Adjoint backward call at the edges of its 32-row blocks and right-hand-side passes: lambda against
numpy's A^H solve and the gradient against the FP64 CPU adjoint, with and without a lambda array, low-rank
parameters of rank 0 and more, dense ones, and both kinds in one call."""
import numpy as np
import pytest

from oracle import oracle as O
from staccato_b200 import _capi
from staccato_b200.adjoint import Param, backward
from staccato_b200.sweep import DeviceRom, sweep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,r,F", [(1, 1, 3), (5, 3, 4), (31, 1, 5), (32, 2, 3), (33, 5, 2), (64, 1, 300), (200, 4, 3)])
def test_backward_blocks(handle, n, r, F):
    import torch

    rng = np.random.default_rng(100 * n + r)
    c = lambda s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    K, M, D = c((n, n)) + 2.0 * n ** 0.5 * np.eye(n), 0.1 * c((n, n)), 0.1 * c((n, n))
    rhs, omega, gb = c((n, r)), rng.uniform(0.2, 1.5, F), c((F, n, r))
    d = DeviceRom.from_host(K, M, D, rhs, omega, keep_factors=True)
    sweep(handle, [d], flags=_capi.SROM_FLAG_KEEP_FACTORS)
    rank = min(n, 3)
    U, Wm, s, G, G2 = c((n, rank)), c((n, rank)), rng.uniform(0.5, 2, rank), c((n, n)), c((n, n))
    t = lambda a: torch.from_numpy(np.asarray(a)).cuda()
    flat = lambda a: t(np.asfortranarray(a).ravel(order="F").astype(np.complex128))
    params = [Param(U=flat(U), W=flat(Wm), s=t(s), rank=rank, c0=0.3 + 0.1j, c1=0.7, c2=-0.2j),
              Param(G=flat(G), c0=1j, c1=0.5 - 0.5j), Param(U=flat(U), rank=0),
              Param(U=flat(U), rank=rank, c2=1.0), Param(G=flat(G2), c0=0.25)]
    mats = [(U * s) @ Wm.T, G, np.zeros((n, n)), U @ U.T, G2]

    class Terms:
        count = len(params)

        def __call__(self, j, w):
            p = params[j]
            return (p.c0 + p.c1 * (1j * w) + p.c2 * (-w * w)) * mats[j]

    ref = O.adjoint_gradient(K, M, D, 0.0, rhs, omega, gb, Terms())
    g, lam = backward(handle, d, t(gb), params, want_lambda=True)
    g2 = backward(handle, d, t(gb), params)
    assert np.array_equal(g.cpu().numpy(), g2.cpu().numpy())
    assert np.abs(g.cpu().numpy() - ref).max() <= 1e-10 * max(np.abs(ref).max(), 1.0)
    A = np.stack([K - w * w * M + 1j * w * D for w in omega])
    want = np.linalg.solve(A.conj().transpose(0, 2, 1), gb)
    assert np.abs(lam.cpu().numpy() - want).max() <= 1e-10 * np.abs(want).max()
    for only in ([params[1]], [params[0]]):  # one kind alone
        j = params.index(only[0])
        assert abs(backward(handle, d, t(gb), only).item() - ref[j]) <= 1e-10 * max(np.abs(ref).max(), 1.0)
