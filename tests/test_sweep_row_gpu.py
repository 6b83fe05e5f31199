"""FP64 row kernel (orders up to 512): solutions, kept factors, pivots and info bit-identical to the
oracle at the edges of its thread counts (64, 128, 256, 512), 16-column panels and column chunks, with
tied pivots (entries of equal |re| + |im| in one thread block and across its warps), zero columns and
NaN, and for more right-hand sides than one pass of the backward substitution holds."""
import numpy as np
import pytest

from oracle import oracle as O
from staccato_b200 import _capi
from staccato_b200.sweep import DeviceRom, sweep

pytestmark = pytest.mark.gpu


def _matrix(kind, n, rng):
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    if kind == "tied":  # every candidate of a column has the same |re| + |im|
        A = rng.choice([1.0, -1.0, 1j, -1j], (n, n)) * (1.0 + rng.integers(0, 2, (n, n)))
    elif kind == "real":  # zero imaginary parts: zero operands in every pivot division
        A = A.real + 0j
    elif kind == "zero_column":
        A[:, n // 2] = 0.0
    elif kind == "nan":
        A[n // 3, n // 2] = np.nan
    return A


def _same(a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    nan = np.isnan(a) & np.isnan(b)
    assert np.array_equal(np.where(nan, 0, a).view(np.uint64), np.where(nan, 0, b).view(np.uint64))


@pytest.mark.parametrize("kind", ["random", "tied", "real", "zero_column", "nan"])
@pytest.mark.parametrize("n,r", [(1, 1), (2, 3), (15, 2), (16, 1), (17, 9), (33, 2), (64, 1), (65, 40), (97, 3),
                                 (128, 2), (129, 1), (200, 4), (256, 8), (257, 2), (300, 17), (512, 3)])
def test_row_kernel_matches_oracle(handle, kind, n, r):
    rng = np.random.default_rng(1000 * n + r)
    K = _matrix(kind, n, rng)
    D = None if kind in ("tied", "real") else 0.1 * _matrix("random", n, rng)
    M = np.zeros((n, n), dtype=complex) if kind == "tied" else np.eye(n, dtype=complex)
    rhs = rng.standard_normal((n, r)) + 1j * rng.standard_normal((n, r))
    omega = np.array([0.3, 0.7])
    keep = DeviceRom.from_host(K, M, D, rhs, omega, keep_factors=True)
    sweep(handle, [keep], flags=_capi.SROM_FLAG_KEEP_FACTORS)
    free = DeviceRom.from_host(K, M, D, rhs, omega)
    sweep(handle, [free])
    Xo, info = O.sweep(K, M, D, 0.0, rhs, omega)
    _same(keep.solutions(), Xo)
    _same(free.solutions(), Xo)
    assert np.array_equal(keep.info.cpu().numpy(), info) and np.array_equal(free.info.cpu().numpy(), info)
    LU = keep.LU.cpu().numpy().reshape(2, n, n).transpose(0, 2, 1)
    ipiv = keep.ipiv.cpu().numpy().reshape(2, n)
    for f, w in enumerate(omega):
        LUo, ipo, _ = O.zgetrf(O.assemble(K, M, D, 0.0, w))
        assert np.array_equal(ipiv[f], ipo)
        _same(LU[f], LUo)


def test_row_kernel_batch_of_all_thread_counts(handle):
    """One call with every thread count, uneven orders and right-hand sides sharing a launch."""
    rng = np.random.default_rng(5)
    roms, refs = [], []
    for n, r, F in [(3, 2, 4), (60, 1, 7), (64, 5, 3), (100, 3, 5), (128, 1, 3), (131, 6, 4), (250, 2, 3), (400, 1, 2)]:
        K, M = _matrix("random", n, rng), np.eye(n, dtype=complex)
        rhs = rng.standard_normal((n, r)) + 1j * rng.standard_normal((n, r))
        omega = rng.uniform(0.1, 2.0, F)
        roms.append(DeviceRom.from_host(K, M, None, rhs, omega, eta=0.02))
        refs.append(O.sweep(K, M, None, 0.02, rhs, omega)[0])
    sweep(handle, roms)
    for d, x in zip(roms, refs):
        _same(d.solutions(), x)
