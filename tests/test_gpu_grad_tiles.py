"""The tiled gradient (65,536 rows and more, 2-D and 3-D). With a learning rate of 0 the points stay, so after N iterations
of constant weights Adam's first moment is g (1 - 0.9^N): the gradient is read from it and held to the bound of the other
gradient tests, 1e-5 of a row's sum of |contributions|, against the FP64 oracle."""
import numpy as np
import pytest

from pacmap_b200._abi import ptr

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _lists(n, seed, hubs=()):
    rng = np.random.default_rng(seed)
    out = []
    for k, near in ((20, True), (10, False), (40, False)):
        p = (np.arange(n)[:, None] + rng.integers(1, 300, size=(n, k))) % n if near else rng.integers(0, n, size=(n, k))
        for h, size in hubs:
            p[rng.choice(n, size=int(size * k / 70), replace=False), 0] = h
        out.append(np.stack([np.repeat(np.arange(n), k), p.reshape(-1)], 1).astype(np.uint32))
    return out


def _moment_gradient(lib, y, pairs, begin, iters=14):
    n, dim = y.shape
    yy, m, v = y.copy(), np.zeros_like(y), np.zeros_like(y)
    lib.stages.optimize_steps(yy, m, v, *pairs, 0.0, 100, 100, begin, begin + iters, want_grad=False)
    assert np.array_equal(yy, y)
    return m / (1 - 0.9 ** iters)


# exactly the first size, one more (a last window of one row), a ragged size; both dimensions; mid-near pairs on (weights
# 3, 3, 1) and off (1, 0, 1); a size of 9 to 13 tiles; rows around the limits of 511 and 1,024 entries
@pytest.mark.parametrize("n,dim,begin", [(65536, 2, 150), (65537, 3, 205), (70003, 2, 205), (90001, 3, 150), (250007, 2, 150)])
def test_gradient_matches_oracle(lib, orc, n, dim, begin):
    pairs = _lists(n, n, [(0, 300), (129, 360), (n - 1, 400), (5000, 900), (65000, 1500), (777, 6000)])
    y = np.random.default_rng(dim).normal(0, 4, size=(n, dim)).astype(np.float32)
    y[1000:1050] = y[1000]                     # coincident points
    y[2000:2010] *= np.float32(1e4)            # far ones
    w = (3.0, 3.0, 1.0) if begin < 200 else (1.0, 0.0, 1.0)
    got = _moment_gradient(lib, y, pairs, begin)
    _, exp64, absum = orc.grad(y, *pairs, *w, with64=True)
    assert (np.abs(got - exp64[:-1]) <= TOL * absum + 1e-30).all()
    assert np.array_equal(got, _moment_gradient(lib, y, pairs, begin))


def test_distances_beyond_the_factor_range(lib, orc):
    """Points so far off that the squared denominators leave f32's range: their factors are 0 and nothing is NaN."""
    n = 66001
    pairs = _lists(n, 7)
    y = np.random.default_rng(1).normal(0, 4, size=(n, 2)).astype(np.float32)
    y[::1000] = np.float32(3e10) * np.random.default_rng(2).normal(size=y[::1000].shape).astype(np.float32)
    got = _moment_gradient(lib, y, pairs, 205)
    _, exp64, absum = orc.grad(y, *pairs, 1.0, 0.0, 1.0, with64=True)
    assert np.isfinite(got).all()
    assert (np.abs(got - exp64[:-1]) <= TOL * absum + 1e-26).all()


def test_fit_close_to_one_kernel_per_iteration(lib):
    """The same fit with losses asked for (no tiles): 40 iterations stay within 1e-4 normwise; snapshots too."""
    n = 70001
    x = np.random.default_rng(3).normal(size=(n, 8)).astype(np.float32)
    pnn, pmn, pfp = _lists(n, 11)
    cfg = lib.Configuration(initialization=lib.Initialization.Random(3), seed=5, num_iters=(14, 13, 13), snapshots=[5, 20, 40],
                            pair_configuration=lib.PairConfiguration.AllProvided(pnn, pmn, pfp))
    a, sa = lib.fit_transform(x, cfg)
    b, sb, _ = lib.fit_transform(x, cfg, loss_trace=True)
    assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b)
    assert np.linalg.norm(sa - sb) <= 1e-4 * np.linalg.norm(sb) and np.array_equal(sa[2], a)


def test_output_buffer_off_the_16_byte_grid(lib):
    """fit_transform_device into a buffer at an odd multiple of 8 bytes takes the other kernels: their bits."""
    import torch

    n = 66000
    x = np.random.default_rng(3).normal(size=(n, 8)).astype(np.float32)
    pnn, pmn, pfp = _lists(n, 12)
    cfg = lib.Configuration(initialization=lib.Initialization.Random(3), seed=5, num_iters=(6, 6, 6),
                            pair_configuration=lib.PairConfiguration.AllProvided(pnn, pmn, pfp))
    dx = torch.from_numpy(x).cuda()
    out = torch.zeros(2 * n + 2, device="cuda")
    torch.cuda.synchronize()
    lib.fit_transform_device(dx.data_ptr(), n, 8, out.data_ptr() + 8, cfg)
    b, _, _ = lib.fit_transform(x, cfg, loss_trace=True)
    assert np.array_equal(out[2:].cpu().numpy().reshape(n, 2), b)


@pytest.mark.parametrize("num", [20.0, 40.0, 60.0, -2.0])
def test_division_is_correctly_rounded(lib, num):
    """Every mantissa at x in [4, 8), and every exponent up to 2^126 on a sample, against IEEE division."""
    x = np.arange(0x40800000, 0x41000000, dtype=np.uint32).view(np.float32)
    rng = np.random.default_rng(0)
    for e in range(2, 126, 3):
        x = np.concatenate([x, np.float32(2.0) ** e * rng.uniform(1, 2, 2000).astype(np.float32)])
    out = np.zeros_like(x)
    lib._check(lib._abi.lib().pacmap_debug_divide(num, ptr(x), x.size, 0, ptr(out)))
    assert np.array_equal(out, (np.float32(num) / x).astype(np.float32))
