"""Descriptors of a batch of one-frequency systems: field by field for few systems, as columns of one array for many;
both give what filling every structure by itself gives, also for addresses in the upper half of the range."""
import pytest

from staccato_b200._capi import RomDesc
from staccato_b200.sweep import _system_descs


@pytest.mark.parametrize("count", [0, 1, 2, 24, 25, 26, 1000])
@pytest.mark.parametrize("n,r,base", [(1, 1, 4096), (24, 5, 0x7F00_0000_1000), (200, 3, (1 << 63) + 256)])
def test_system_descs(count, n, r, base):
    K, rhs, omega, X, info = base, base + (1 << 40), base + 64, base + (2 << 40), base + (3 << 40)
    arr = _system_descs(count, n, r, K, rhs, omega, X, info)
    assert len(arr) == max(count, 1)
    for i in range(count):
        want = RomDesc(n=n, r=r, F=1, ldk=n, K=K + i * n * n * 16, M=None, D=None, eta=0.0, rhs=rhs + i * n * r * 16, ldb=n,
                       omega=omega, X=X + i * n * r * 16, info=info + 4 * i, steps=None, berr=None, LU=None, ipiv=None)
        assert bytes(arr[i]) == bytes(want), i
