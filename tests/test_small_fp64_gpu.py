"""FP64 sweeps of the smallest orders and of many right-hand sides to a column, which the shared-memory kernel takes where
it is faster than the row kernel: at the edges of that rule (order, right-hand sides, systems to a multiprocessor),
alone and beside larger orders in one call, with kept factors, damping, no mass, through the entry point that does
not allocate and under capture: the results are LAPACK's as restated, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from staccato_b200 import _capi
from staccato_b200.sweep import DeviceRom, Graph, sweep

pytestmark = pytest.mark.gpu


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


def _data(n, r, F, seed=0, damped=True):
    rng = np.random.default_rng(1000 * n + r + seed)
    K = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    M = np.eye(n) + 0j
    D = 0.05 * rng.standard_normal((n, n)) + 0j if damped else None
    rhs = rng.standard_normal((n, r)) + 1j * rng.standard_normal((n, r))
    return K, M, D, 0.02, rhs, np.linspace(0.1, 2.0, F)


def _check(rom, data, sel=None):
    K, M, D, eta, rhs, omega = data
    sel = np.arange(len(omega)) if sel is None or len(omega) <= 6 else np.array(sel)
    X, info = O.sweep(K, M, D, eta, rhs, omega[sel])
    assert np.array_equal(np.ascontiguousarray(rom.solutions()[sel]).view(np.uint64), np.ascontiguousarray(X).view(np.uint64))
    assert np.array_equal(rom.info.cpu().numpy()[sel], info)
    assert (rom.steps.cpu().numpy() == 0).all()


def _dev(data, keep=False):
    K, M, D, eta, rhs, omega = data
    return DeviceRom.from_host(K, M, D, rhs, omega, eta=eta, keep_factors=keep)


ENDS = [0, 1, -2, -1]


@pytest.mark.parametrize("n,r", [(1, 1), (1, 15), (1, 16), (1, 5000), (1, 9500), (2, 1), (3, 7), (3, 8), (4, 1000), (8, 1), (8, 97),
                                 (9, 2), (9, 3), (9, 4), (16, 5), (16, 6), (17, 3), (17, 4), (24, 200), (31, 7), (32, 6), (32, 7),
                                 (32, 300), (33, 40)])
def test_small_orders(handle, n, r):
    data = _data(n, r, 5, damped=n % 2 == 0)
    rom = _dev(data)
    sweep(handle, [rom])
    _check(rom, data)


@pytest.mark.parametrize("n,r,load", [(1, 1, 1.0), (1, 1, 1.01), (8, 1, 1.0), (8, 1, 1.01), (8, 1, 2.0), (8, 1, 2.01), (32, 300, 1.5), (24, 200, 1.5), (3, 8, 2.0), (4, 18, 2.2), (4, 18, 2.3),
                                      (2, 32, 4.0), (2, 32, 4.4), (1, 16, 5.0), (2, 64, 9.0)])
def test_small_orders_by_fill(handle, n, r, load):
    data = _data(n, r, int(load * _sms()))
    rom = _dev(data)
    sweep(handle, [rom])
    _check(rom, data, ENDS)


def test_small_orders_beside_larger_ones(handle):
    for extra in (1, _sms()):  # the second call has more systems than multiprocessors
        datas = [_data(8, 1, 3), _data(24, 200, 2), _data(100, 1, extra), _data(5, 21, 2), _data(300, 2, 2), _data(12, 1, 4)]
        roms = [_dev(d, keep=i == 0) for i, d in enumerate(datas)]
        sweep(handle, roms)
        for rom, d in zip(roms, datas):
            _check(rom, d, ENDS)


def test_small_orders_keep_factors_and_graph(handle):
    import torch

    data = _data(8, 3, 4)
    K, M, D, eta, rhs, omega = data
    rom = _dev(data, keep=True)
    sweep(handle, [rom], flags=_capi.SROM_FLAG_KEEP_FACTORS)
    LU = rom.LU.cpu().numpy().reshape(rom.F, 8, 8).transpose(0, 2, 1)
    ipiv = rom.ipiv.cpu().numpy().reshape(rom.F, 8)
    for f, w in enumerate(omega):
        LUo, ipo, _ = O.zgetrf(O.assemble(K, M, D, eta, w))
        assert np.array_equal(ipiv[f], ipo)
        assert np.array_equal(np.ascontiguousarray(LU[f]).view(np.uint64), np.ascontiguousarray(LUo).view(np.uint64))
    datas = [_data(4, 1000, 3), _data(64, 1, 3)]
    roms = [_dev(d) for d in datas]
    g = Graph(handle, roms)
    for _ in range(2):
        for r in roms:
            r.X.zero_()
        g.launch()
        torch.cuda.synchronize()
        for rom, d in zip(roms, datas):
            _check(rom, d)
    g.close()


@pytest.mark.parametrize("n,r,F", [(1, 1, 8), (1, 16, 148), (8, 16, 8), (8, 16, 700), (16, 6, 4), (32, 8, 4), (64, 1, 4)])
def test_small_orders_without_allocation(handle, n, r, F):
    data = _data(n, r, F)
    rom = _dev(data)
    err = C.create_string_buffer(200)
    d = rom.desc()
    assert _capi.lib().srom_sweep_fp64_noalloc(C.byref(d), None, err, 200) == 0, err.value
    _check(rom, data, ENDS)


def test_small_orders_singular_and_nan(handle):
    n, r = 6, 9
    K, M, D, eta, rhs, omega = _data(n, r, 2, damped=False)
    M = 0.0 * M
    for case in range(3):
        k = K.copy()
        if case == 0:
            k[:, 2] = 0.0  # a zero pivot
        elif case == 1:
            k[0, 0] = np.nan  # a NaN first in its column is the pivot
        else:
            k[3, 1] = np.nan
        data = (k, M, None, 0.0, rhs, omega)
        rom = _dev(data)
        sweep(handle, [rom])
        X, info = O.sweep(k, M, None, 0.0, rhs, omega)
        a, b = rom.solutions(), X
        assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(a[~np.isnan(a)], b[~np.isnan(b)])
        assert np.array_equal(rom.info.cpu().numpy(), info)


@pytest.mark.parametrize("specs", [
    [(64, 1, 3), (65, 2, 1), (128, 1, 2), (129, 1, 1), (257, 1, 1)],   # one launch for all four thread counts
    [(64, 1, 147), (65, 1, 1)], [(64, 1, 300), (100, 3, 290)], [(64, 1, 300), (100, 3, 293)],  # up to a wave of the larger, and past it
    [(200, 1, 147), (300, 2, 1)], [(200, 1, 148), (300, 2, 1)],
    [(40, 2, 1), (500, 1, 1)], [(33, 1, 200), (500, 1, 100)],
])
def test_row_classes_sharing_a_launch(handle, specs):
    datas = [_data(n, r, F, seed=i) for i, (n, r, F) in enumerate(specs)]
    roms = [_dev(d, keep=i == 0) for i, d in enumerate(datas)]
    sweep(handle, roms)
    for rom, d in zip(roms, datas):
        _check(rom, d, ENDS)
    ip = roms[0].ipiv.cpu().numpy().reshape(roms[0].F, -1)
    K, M, D, eta, rhs, omega = datas[0]
    assert np.array_equal(ip[0], O.zgetrf(O.assemble(K, M, D, eta, omega[0]))[1])
