"""The tuner's cache and its tables: a file of the earlier format is measured anew, a file of this one is read, and
the thread count of the FP64 kernel has no say in the mixed forms' routing."""
import json

import numpy as np
import pytest

from staccato_b200 import _capi
from staccato_b200.sweep import DeviceRom, sweep, tune

pytestmark = pytest.mark.gpu


def _device():
    import torch

    return torch.cuda.get_device_name(0)


def _rom(n, F):
    rng = np.random.default_rng(n)
    K = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 4.0 * np.sqrt(n) * np.eye(n)
    rhs = rng.standard_normal((n, 1)) + 0j
    return DeviceRom.from_host(K, np.eye(n) + 0j, None, rhs, np.linspace(0.1, 2.0, F))


def test_cache_of_the_earlier_format_is_measured_anew(tmp_path):
    cache = tmp_path / "tune.json"
    cache.write_text('{\n  "device": "%s",\n  "entries": [\n'
                     '    {"precision": "fp64", "n": 64, "r": 1, "kernel": "global", "ms_smem": 2.0, "ms_global": 1.0},\n'
                     '    {"precision": "mixed", "n": 64, "r": 1, "kernel": "mixed_global", "ms_fp64_smem": 2.0, "ms_mixed_global": 1.0}\n'
                     '  ]\n}\n' % _device())
    h = _capi.Handle(0)
    try:
        tune(h, [64], r=1, cache_path=str(cache))
        data = json.loads(cache.read_text())
        assert data["format"] == 2
        e = {(x["precision"], x["n"]): x for x in data["entries"]}
        assert set(e) == {("fp64", 64), ("mixed", 64)}
        assert e["fp64", 64]["threads"] in (64, 128) and e["fp64", 64]["ms"] > 0 and e["fp64", 64]["ms_wide"] > 0
        m = e["mixed", 64]
        assert (m["kernel"] == "mixed_global") == (m["ms_mixed_global"] < m["ms_fp64_smem"])
    finally:
        h.close()


@pytest.mark.parametrize("kernel,outright", [("fp64_smem", True), ("mixed_global", False), (None, True)])
def test_thread_count_leaves_the_mixed_routing_alone(tmp_path, kernel, outright):
    """A file of this format with the larger thread count: FP64 results are the same bits, and the mixed form
    follows its own entry, or its rule where there is none."""
    lines = ['    {"precision": "fp64", "n": 64, "r": 1, "kernel": "smem", "threads": 128, "ms": 2.0, "ms_wide": 1.0}']
    if kernel:
        lines.append('    {"precision": "mixed", "n": 64, "r": 1, "kernel": "%s", "ms_fp64_smem": 1.0, "ms_mixed_global": 2.0}' % kernel)
    cache = tmp_path / "tune.json"
    cache.write_text('{\n  "format": 2,\n  "device": "%s",\n  "entries": [\n%s\n  ]\n}\n' % (_device(), ",\n".join(lines)))
    before = cache.read_text()
    plain, tuned = _capi.Handle(0), _capi.Handle(0)
    try:
        tune(tuned, [], r=1, cache_path=str(cache))
        assert cache.read_text() == before
        a, b = _rom(64, 20), _rom(64, 20)
        sweep(plain, [a])
        sweep(tuned, [b])
        assert np.array_equal(a.solutions().view(np.uint64), b.solutions().view(np.uint64))
        sweep(tuned, [b], precision=_capi.SROM_MIXED_FP32, flags=_capi.SROM_FLAG_FALLBACK_FP64)
        steps = b.steps.cpu().numpy()
        assert (steps == 0).all() if outright else (steps >= 1).all()
    finally:
        plain.close()
        tuned.close()
