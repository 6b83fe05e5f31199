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


# both sides of the rule that takes the terms into the solve kernel: one wave of frequencies, n r up to a tile, 512
# terms, 2^17 multiply-adds a frequency; the lambda array must not matter
@pytest.mark.parametrize("n,r,F,terms,dense", [(33, 32, 2, 5, 1), (33, 33, 2, 5, 1), (40, 1, 5, 512, 0), (40, 1, 5, 513, 0),
                                               (128, 1, 3, 0, 8), (128, 1, 3, 1, 8), (128, 1, 600, 3, 1), (20, 2, 592, 3, 2),
                                               (20, 2, 593, 3, 2), (3, 1, 1, 7, 3)])
def test_backward_terms(handle, n, r, F, terms, dense):
    import torch

    rng = np.random.default_rng(100 * n + terms)
    c = lambda s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    K, M = c((n, n)) + 2.0 * n ** 0.5 * np.eye(n), 0.1 * c((n, n))
    rhs, omega, gb = c((n, r)), rng.uniform(0.2, 1.5, F), c((F, n, r))
    d = DeviceRom.from_host(K, M, None, rhs, omega, keep_factors=True)
    sweep(handle, [d], flags=_capi.SROM_FLAG_KEEP_FACTORS)
    t = lambda a: torch.from_numpy(np.asarray(a)).cuda()
    flat = lambda a: t(np.asfortranarray(a).ravel(order="F").astype(np.complex128))
    U, W, s, G = c((n, max(terms, 1))), c((n, max(terms, 1))), rng.uniform(0.5, 2, max(terms, 1)), [c((n, n)) for _ in range(dense)]
    first = min(terms, 2)
    params = [Param(U=flat(U[:, :first]), W=flat(W[:, :first]), s=t(s[:first]), rank=first, c0=0.3 + 0.1j, c1=0.7, c2=-0.2j),
              Param(U=flat(U[:, first:]), rank=terms - first, c2=1.0)] + [Param(G=flat(g), c0=1j, c1=0.5 - 0.5j) for g in G]
    A = np.stack([K - w * w * M for w in omega])
    X = np.linalg.solve(A, np.broadcast_to(rhs, (F, n, r)))
    lam = np.linalg.solve(A.conj().transpose(0, 2, 1), gb)
    mats = [(U[:, :first] * s[:first]) @ W[:, :first].T, U[:, first:terms] @ U[:, first:terms].T] + G
    want, scale = [], []
    for p, m in zip(params, mats):
        coef = p.c0 + p.c1 * (1j * omega) + p.c2 * (-omega * omega)
        S = np.einsum("fir,fir->f", lam.conj(), m @ X)
        want.append(-(coef * S).real.sum())
        scale.append((np.abs(coef) * np.linalg.norm(lam, axis=(1, 2)) * np.linalg.norm(X, axis=(1, 2))).sum() * np.linalg.norm(m))
    g, lam_d = backward(handle, d, t(gb), params, want_lambda=True)
    assert np.array_equal(g.cpu().numpy(), backward(handle, d, t(gb), params).cpu().numpy())
    # the solves: 1e-10 as in the test above; the sums: n^2 terms an entry
    assert np.abs(lam_d.cpu().numpy() - lam).max() <= 1e-10 * np.abs(lam).max()
    assert (np.abs(g.cpu().numpy() - want) <= 1e-10 * np.maximum(np.array(scale), 1e-300)).all()


@pytest.mark.parametrize("n,tiny", [(1, 1e-310), (3, 1e-310), (40, 3e-309), (2, 1e-305), (2, 1e305), (33, 1e306)])
def test_backward_extreme_last_pivot(handle, n, tiny):
    """A last pivot whose reciprocal is out of range (the forward solve divides by it): lambda divides too."""
    import torch

    rng = np.random.default_rng(n)
    k = rng.uniform(1.0, 2.0, n) * np.exp(1j * rng.uniform(0.0, 1.0, n))
    k[-1] = tiny * (1.0 + 0.5j)
    rhs = np.ones((n, 1)) + 0j
    rhs[-1] = 3.0 * tiny
    gb = np.ones((1, n, 1)) * (1.0 - 2.0j)
    gb[0, -1] *= tiny
    d = DeviceRom.from_host(np.diag(k), np.zeros((n, n)) + 0j, None, rhs, np.array([1.0]), keep_factors=True)
    sweep(handle, [d], flags=_capi.SROM_FLAG_KEEP_FACTORS)
    U = torch.from_numpy(np.ones(n) + 0j).cuda()
    g, lam = backward(handle, d, torch.from_numpy(gb).cuda(), [Param(U=U, rank=1)], want_lambda=True)
    # conj(k) as stored, scaled by a power of two into the normal range before the division
    sc = 2.0 ** (-1000.0 * np.sign(np.log10(tiny)))
    want = gb[0, :, 0] / k.conj()
    want[-1] = (gb[0, -1, 0] * sc) / (k[-1].conj() * sc)
    got = lam.cpu().numpy()[0, :, 0]
    assert np.isfinite(got).all() and (np.abs(got - want) <= 8 * np.finfo(float).eps * np.abs(want)).all()
    x = d.solutions()[0, :, 0]
    assert abs(g.item() + (got.conj().sum() * x.sum()).real) <= 1e-13 * np.abs(got).sum() * np.abs(x).sum()
