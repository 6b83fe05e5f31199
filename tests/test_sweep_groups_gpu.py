"""FP64 sweep above n = 512 (groups of systems advancing panel by panel): bit-identical to the oracle at
the edges of its panels (32 columns), cluster sizes (320 rows a block) and tiles, with tied pivots,
zero columns and NaN, for systems of uneven order in one group and for more systems than one group holds."""
import numpy as np
import pytest

from oracle import oracle as O
from staccato_b200 import _capi
from staccato_b200.sweep import DeviceRom, sweep
from test_sweep_row_gpu import _matrix, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,r,kind", [(513, 2, "random"), (544, 1, "tied"), (545, 3, "zero_column"), (641, 1, "nan"),
                                      (640, 2, "real"), (673, 8, "random"), (961, 1, "tied"), (1281, 1, "random")])
def test_large_orders_match_oracle(handle, n, r, kind):
    rng = np.random.default_rng(n)
    K, M = _matrix(kind, n, rng), np.zeros((n, n), dtype=complex)
    rhs = rng.standard_normal((n, r)) + 1j * rng.standard_normal((n, r))
    omega = np.array([0.6])
    keep = DeviceRom.from_host(K, M, None, rhs, omega, keep_factors=True)
    sweep(handle, [keep], flags=_capi.SROM_FLAG_KEEP_FACTORS)
    free = DeviceRom.from_host(K, M, None, rhs, omega)
    sweep(handle, [free])
    Xo, info = O.sweep(K, M, None, 0.0, rhs, omega)
    LUo, ipo, _ = O.zgetrf(O.assemble(K, M, None, 0.0, 0.6))
    _same(keep.solutions(), Xo)
    _same(free.solutions(), Xo)
    assert np.array_equal(keep.info.cpu().numpy(), info) and np.array_equal(free.info.cpu().numpy(), info)
    assert np.array_equal(keep.ipiv.cpu().numpy(), ipo)
    _same(keep.LU.cpu().numpy().reshape(n, n).T, LUo)


def test_uneven_orders_and_several_groups(handle):
    rng = np.random.default_rng(7)
    roms, refs = [], []
    for n, r, F in [(700, 1, 2), (520, 4, 3), (900, 2, 2)]:
        K, M = _matrix("random", n, rng), np.eye(n, dtype=complex)
        rhs = rng.standard_normal((n, r)) + 1j * rng.standard_normal((n, r))
        omega = rng.uniform(0.1, 2.0, F)
        roms.append(DeviceRom.from_host(K, M, None, rhs, omega, eta=0.02))
        refs.append(O.sweep(K, M, None, 0.02, rhs, omega)[0])
    sweep(handle, roms)
    for d, x in zip(roms, refs):
        _same(d.solutions(), x)
    # 160 systems: more than one multiprocessor's worth of slots; every system the same matrix
    n = 514
    K, M, rhs = _matrix("random", n, rng), np.zeros((n, n), dtype=complex), rng.standard_normal((n, 1)) + 0j
    d = DeviceRom.from_host(K, M, None, rhs, np.full(160, 0.5))
    sweep(handle, [d])
    x = O.sweep(K, M, None, 0.0, rhs, np.array([0.5]))[0]
    _same(d.solutions(), np.repeat(x, 160, axis=0))
