"""Copies of ordinary host memory through the page-locked slots: preprocessing (every input byte in, every output byte out)
bit for bit against the oracle at sizes around the rule and the pieces, from several threads at once, and from and to
page-locked memory, which goes the direct way."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(n, d, seed):
    return np.random.default_rng(seed).uniform(-2, 3, size=(n, d)).astype(np.float32)


# bytes: around the rules of 1 MiB (down) and 32 MiB (up), one to eight workers, ranges that are no multiple of a piece or
# of 4 KiB, more than all slots hold
@pytest.mark.parametrize("n,d", [(262143, 1), (262144, 1), (262145, 1), (1048577, 1), (174763, 9), (100003, 33),
                                 (8388607, 1), (262144, 32), (262145, 32), (30011, 301), (170001, 97)])
def test_copies_are_complete(lib, orc, n, d):
    x = _rows(n, d, n)
    got, mn, mx, mean = lib.stages.preprocess(x)
    exp, emn, emx, emean = orc.preprocess(x)
    assert (mn, mx) == (emn, emx) and np.array_equal(mean, emean) and np.array_equal(got, exp)


def test_copies_from_unaligned_memory(lib, orc):
    n = 300001
    raw = np.zeros(n * 31 * 4 + 64, np.uint8)
    x = raw[12:12 + n * 31 * 4].view(np.float32).reshape(n, 31)
    x[:] = _rows(n, 31, 4)
    got = lib.stages.preprocess(x)[0]
    assert np.array_equal(got, orc.preprocess(x)[0])


def test_copies_from_several_threads(lib, orc):
    xs = [_rows(170001 + 7 * t, 50, t) for t in range(4)]
    want = [orc.preprocess(x)[0] for x in xs]
    bad = []

    def work(t):
        for _ in range(3):
            if not np.array_equal(lib.stages.preprocess(xs[t])[0], want[t]):
                bad.append(t)

    th = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not bad


def test_page_locked_memory(lib, orc):
    import torch

    x = _rows(240000, 40, 8)
    px = torch.empty(x.shape, dtype=torch.float32, pin_memory=True)
    px.copy_(torch.from_numpy(x))
    out = torch.empty_like(px, pin_memory=True)
    mn, mx = C.c_float(0), C.c_float(0)
    lib._check(lib._abi.lib().pacmap_preprocess(px.data_ptr(), 240000, 40, 0, out.data_ptr(), C.byref(mn), C.byref(mx), None))
    assert np.array_equal(out.numpy(), orc.preprocess(x)[0])
