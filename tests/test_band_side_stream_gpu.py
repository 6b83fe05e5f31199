"""Band solves of one handle called again and again: models of one block and of several, from one stream and then from
another, two handles in turn; every call gives the bits of a fresh handle's first call."""
import numpy as np
import pytest
import scipy.sparse as sp

from staccato_b200 import _capi
from staccato_b200.krylov import fom_sweep
from staccato_b200.project import DeviceCsr

pytestmark = pytest.mark.gpu


def _model(n, bw):
    import torch

    rng = np.random.default_rng(n)
    a = sp.diags([np.full(n, 4.0 * bw + 1.0) if o == 0 else -rng.uniform(0.5, 1.0, n - o) for o in range(bw + 1)], range(bw + 1))
    a = (a + sp.triu(a, 1).T).tocsr()
    a.sort_indices()
    csr = DeviceCsr.from_host(a.indptr, a.indices)
    v = torch.from_numpy(a.data).cuda().to(torch.complex128)
    load = torch.from_numpy(rng.standard_normal((2, n)) + 1j * rng.standard_normal((2, n))).cuda()
    return a, csr, v, (0.01 * v).contiguous(), load


@pytest.mark.parametrize("n,bw", [(2, 1), (64, 3), (65, 3), (700, 90)])
def test_repeated_band_solves(cuda_device, n, bw):
    import torch

    a, csr, K, M, load = _model(n, bw)
    freqs = [0.02, 0.05]
    first = _capi.Handle(0)
    want = fom_sweep(first, csr, K, M, None, load, freqs).clone()
    w = 2 * np.pi * freqs[1]
    ref = np.linalg.solve(a.toarray() * (1 - 0.01 * w * w), load.cpu().numpy().T)
    assert np.abs(want[1].cpu().numpy().T - ref).max() <= 1e-12 * np.abs(ref).max()
    other = _capi.Handle(0)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for h in (first, other, first, other):
        assert torch.equal(torch.view_as_real(fom_sweep(h, csr, K, M, None, load, freqs)), torch.view_as_real(want))
    first.set_stream(stream.cuda_stream)
    with torch.cuda.stream(stream):
        got = fom_sweep(first, csr, K, M, None, load, freqs)
        stream.synchronize()
    assert torch.equal(torch.view_as_real(got), torch.view_as_real(want))
    first.close()
    assert torch.equal(torch.view_as_real(fom_sweep(other, csr, K, M, None, load, freqs)), torch.view_as_real(want))
    other.close()
