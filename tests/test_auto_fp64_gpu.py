"""SROM_MIXED_AUTO in calls of more systems than multiprocessors: orders up to 320 are solved in FP64 outright, so the
solutions are the FP64 form's bit for bit and steps = 0.  At the edges of the rule: the order (320, 321), the number
of systems (a system a multiprocessor, one more; counted over the call's ROMs), every right-hand side count of the
mixed forms' range, with and without D and M, and not with SROM_FLAG_MIXED_EVERY."""
import numpy as np
import pytest

from staccato_b200 import _capi
from staccato_b200.sweep import DeviceRom, solve_batched, sweep

pytestmark = pytest.mark.gpu

AUTO, FB = _capi.SROM_MIXED_AUTO, _capi.SROM_FLAG_FALLBACK_FP64


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


def _rom(n, r, F, damped=False):
    rng = np.random.default_rng(100 * n + r)
    K = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 4.0 * np.sqrt(n) * np.eye(n)
    M = np.eye(n) + 0j
    D = 0.05 * np.eye(n) + 0j if damped else None
    rhs = rng.standard_normal((n, r)) + 1j * rng.standard_normal((n, r))
    omega = np.linspace(0.1, 2.0, F)
    return [DeviceRom.from_host(K, M, D, rhs, omega) for _ in range(2)]


def _same(a, b):
    assert np.array_equal(np.ascontiguousarray(a.solutions()).view(np.uint64),
                          np.ascontiguousarray(b.solutions()).view(np.uint64))
    assert (a.info.cpu().numpy() == b.info.cpu().numpy()).all()


@pytest.mark.parametrize("n,r,damped", [(113, 1, False), (128, 4, True), (129, 2, False), (200, 8, True), (256, 1, True),
                                        (257, 3, False), (320, 1, False), (320, 8, True)])
def test_auto_is_fp64_when_the_call_fills_the_gpu(handle, n, r, damped):
    a, b = _rom(n, r, _sms() + 1, damped)
    sweep(handle, [a], precision=AUTO, flags=FB)
    sweep(handle, [b])
    _same(a, b)
    assert (a.steps.cpu().numpy() == 0).all()


def test_auto_keeps_the_mixed_kernels(handle):
    cases = [(200, _sms(), FB), (321, _sms() + 1, FB), (200, _sms() + 1, FB | _capi.SROM_FLAG_MIXED_EVERY)]
    for n, F, flags in cases:
        a, b = _rom(n, 1, F)
        sweep(handle, [a], precision=AUTO, flags=flags)
        sweep(handle, [b])
        assert (a.steps.cpu().numpy() >= 1).all(), (n, F)
        err = np.linalg.norm(a.solutions() - b.solutions(), axis=1) / np.linalg.norm(b.solutions(), axis=1)
        assert err.max() <= 1e-10


def test_auto_counts_the_systems_of_all_roms(handle):
    pairs = [_rom(150, 1, _sms() // 2 + 1), _rom(300, 2, _sms() // 2 + 1, True), _rom(400, 1, 3), _rom(20, 1, 5)]
    sweep(handle, [p[0] for p in pairs], precision=AUTO, flags=FB)
    sweep(handle, [p[1] for p in pairs])
    for k in (0, 1, 3):
        _same(*pairs[k])
        assert (pairs[k][0].steps.cpu().numpy() == 0).all()
    assert (pairs[2][0].steps.cpu().numpy() >= 1).all()


def test_auto_solve_batched_without_mass(handle):
    import torch

    g = torch.Generator(device="cuda").manual_seed(3)
    n, count = 130, _sms() + 3
    A = torch.randn(count, n, n, dtype=torch.complex128, device="cuda", generator=g) + 20.0 * torch.eye(n, device="cuda")
    B = torch.randn(count, n, 2, dtype=torch.complex128, device="cuda", generator=g)
    X, info = solve_batched(handle, A, B, precision=AUTO)
    Y, _ = solve_batched(handle, A, B)
    assert torch.equal(torch.view_as_real(X), torch.view_as_real(Y)) and int(info.abs().max()) == 0
