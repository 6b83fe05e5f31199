"""Two threads, each with its own handle and stream, running the same kernels at different sizes at the same time: every
call succeeds and gives the bits that it gives alone."""
import threading

import numpy as np
import pytest

from staccato_b200 import _capi
from staccato_b200.adjoint import Param, backward
from staccato_b200.project import DeviceCsr, project
from staccato_b200.sweep import DeviceRom, sweep

pytestmark = pytest.mark.gpu


def _rom(n, r, F, keep=False):
    rng = np.random.default_rng(n)
    K = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 4.0 * np.sqrt(n) * np.eye(n)
    rhs = rng.standard_normal((n, r)) + 0j
    return DeviceRom.from_host(K, np.eye(n) + 0j, None, rhs, np.linspace(0.1, 2.0, F), keep_factors=keep)


def _sweeps(n, r):
    rom = _rom(n, r, 3)

    def call(h):
        sweep(h, [rom])
        return rom.X
    return call


def _backward(n, r):
    import torch

    rom = _rom(n, r, 3, keep=True)
    rng = np.random.default_rng(n)
    gb = torch.from_numpy(rng.standard_normal((3, n, r)) + 0j).cuda()
    U = torch.from_numpy(rng.standard_normal(n) + 0j).cuda()

    def call(h):
        sweep(h, [rom], flags=_capi.SROM_FLAG_KEEP_FACTORS)
        return backward(h, rom, gb, [Param(U=U, rank=1)])
    return call


def _project(k, seed):
    import scipy.sparse as sp
    import torch

    rng = np.random.default_rng(seed)
    a = sp.random(300, 300, density=0.05, random_state=seed, format="csr") + sp.identity(300, format="csr")
    a.sort_indices()
    csr = DeviceCsr.from_host(a.indptr, a.indices)
    vals, V = torch.from_numpy(a.data).cuda(), torch.from_numpy(rng.standard_normal((k, 300))).cuda()
    return lambda h: project(h, csr, [vals], V)[0]


PAIRS = {"row64": lambda: (_sweeps(64, 1), _sweeps(40, 1)), "row256": lambda: (_sweeps(256, 1), _sweeps(130, 1)),
         "smem": lambda: (_sweeps(8, 1), _sweeps(8, 200)), "large": lambda: (_sweeps(530, 4), _sweeps(520, 1)),
         "adjoint": lambda: (_backward(100, 8), _backward(60, 1)), "project": lambda: (_project(120, 1), _project(90, 2))}


@pytest.mark.parametrize("pair", sorted(PAIRS))
def test_two_threads(cuda_device, pair):
    import torch

    calls = PAIRS[pair]()
    handles, streams = [_capi.Handle(0) for _ in calls], [torch.cuda.Stream() for _ in calls]
    want = []
    for h, st, call in zip(handles, streams, calls):
        h.set_stream(st.cuda_stream)
        with torch.cuda.stream(st):
            want.append(call(h).clone())
        st.synchronize()
    errors = []

    def work(q):
        try:
            with torch.cuda.stream(streams[q]):
                for _ in range(300):
                    got = calls[q](handles[q])
                streams[q].synchronize()
                if not torch.equal(torch.view_as_real(got) if got.is_complex() else got,
                                   torch.view_as_real(want[q]) if want[q].is_complex() else want[q]):
                    errors.append("thread %d: other results" % q)
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(q,)) for q in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for h in handles:
        h.close()
    assert not errors, errors
