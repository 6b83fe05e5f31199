"""Panel of the mixed kernels (complex FP32, groups of eight columns in registers): refined solutions without the
FP64 fallback at the edges of its groups (8), panels (32) and rows a thread (256, 512), with tied pivots (every
entry of a column of equal |re| + |im|, inside a warp, across warps and across a thread's rows), with zero operands
in every pivot division, and the column of the first zero pivot at every place of a group.

Tolerance 1e-10 against the long-double-refined solution, the form's own gate: the matrices' condition numbers are
below 1e5, so that FP64 refinement ends near 1e-11 and FP32 factors converge."""
import numpy as np
import pytest

from oracle import oracle as O
from staccato_b200 import _capi
from staccato_b200.sweep import DeviceRom, sweep

pytestmark = pytest.mark.gpu

FORMS = [_capi.SROM_MIXED_FP32, _capi.SROM_MIXED_TC]


def _rom(K, omega):
    n = K.shape[0]
    rng = np.random.default_rng(n)
    rhs = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    d = DeviceRom.from_host(K, np.zeros_like(K), None, rhs, omega)
    return d, rhs


def matrix(kind, n):
    rng = np.random.default_rng(10 * n + len(kind))
    if kind == "tied":
        return rng.choice([1.0, -1.0, 1j, -1j], (n, n)) * (1.0 + rng.integers(0, 2, (n, n)))
    A = rng.standard_normal((n, n))
    return A + 0j if kind == "real" else A + 1j * rng.standard_normal((n, n))


@pytest.mark.parametrize("precision", FORMS)
@pytest.mark.parametrize("kind", ["tied", "real", "random"])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 39, 40, 41, 64, 225, 256, 257, 300, 512])
def test_mixed_panel_converges(handle, precision, kind, n):
    K = matrix(kind, n)
    omega = np.array([0.5, 0.7])
    d, rhs = _rom(K, omega)
    sweep(handle, [d], precision=precision, flags=_capi.SROM_FLAG_MIXED_EVERY, max_refine=8)
    xr = O.x_ref(K, np.zeros_like(K), None, 0.0, rhs, omega)
    assert O.rel_err(d.solutions(), xr).max() <= 1e-10
    assert (d.info.cpu().numpy() == 0).all() and (d.steps.cpu().numpy() >= 0).all()


@pytest.mark.parametrize("precision", FORMS)
@pytest.mark.parametrize("n,col", [(40, c) for c in range(0, 40, 3)] + [(41, 40), (300, 263), (512, 511)])
def test_mixed_panel_reports_the_zero_pivot(handle, precision, n, col):
    K = matrix("random", n)
    K[:, col] = 0.0
    omega = np.array([0.5])
    d, _ = _rom(K, omega)
    sweep(handle, [d], precision=precision, flags=_capi.SROM_FLAG_MIXED_EVERY, max_refine=1)
    assert (d.info.cpu().numpy() == col + 1).all()
