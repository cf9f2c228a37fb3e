"""Inverses of the two-level preconditioners' coarse matrices on the device
(coarse.cu): pivot blocks of 32, one launch each, several matrices side by side."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Item(ctypes.Structure):
    _fields_ = [("scratch", ctypes.c_void_p), ("inv", ctypes.c_void_p), ("n", ctypes.c_int)]


def _invert(mats):
    import torch

    from coolfluid3_b200 import _native

    f = _native.lib()._ZN4ufem13coarse_invertEPKNS_13CoarseInverseEiP11CUstream_st
    f.argtypes = [ctypes.POINTER(_Item), ctypes.c_int, ctypes.c_void_p]
    bufs, items = [], (_Item * len(mats))()
    for k, a in enumerate(mats):
        n = len(a)
        pair = [torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2)]
        pair[0 if (n + 31) // 32 % 2 else 1].copy_(torch.from_numpy(a))  # coarse_source
        bufs.append(pair)
        items[k] = _Item(pair[0].data_ptr(), pair[1].data_ptr(), n)
    assert f(items, len(mats), torch.cuda.current_stream().cuda_stream) == 0
    return [pair[1].cpu().numpy() for pair in bufs]


def _spd(n, cond, seed):
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (q * np.logspace(0, np.log10(cond), n)) @ q.T if n > 1 else np.array([[2.5]])
    return 0.5 * (a + a.T)


SIZES = [1, 2, 31, 32, 33, 64, 65, 125, 256, 400, 511, 512]


def test_inverses_alone_and_side_by_side():
    """Against LAPACK, with the error bound of elimination on an SPD matrix,
    8 n eps cond(A) ||A^-1||; and the same bits alone and beside others (40
    matrices: more than one launch takes)."""
    mats = [_spd(n, 1e4, n) for n in SIZES] + [_spd(17 + k, 1e2, k) for k in range(28)]
    both = _invert(mats)
    for a, x in zip(mats, both):
        n = len(a)
        bound = 8 * n * 2.3e-16 * np.linalg.cond(a) * np.linalg.norm(np.linalg.inv(a), 2)
        assert np.abs(x - np.linalg.inv(a)).max() <= bound, n
        assert np.array_equal(_invert([a])[0], x), n


@pytest.mark.parametrize("n,bad", [(5, 3), (70, 0), (70, 40), (100, 99)])
@pytest.mark.parametrize("value", [0.0, -1.0, float("nan"), float("inf")])
def test_a_pivot_that_is_not_positive_gives_zeros(n, bad, value):
    a = _spd(n, 1e2, n)
    a[bad, :] = a[:, bad] = 0.0
    a[bad, bad] = value
    good = _spd(n, 1e2, n + 1)
    x, y = _invert([a, good])
    assert not x.any()
    assert np.abs(y @ good - np.eye(n)).max() <= 8 * n * 2.3e-16 * 1e2 * np.sqrt(n)
