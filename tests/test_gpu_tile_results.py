"""What a call returns from 65,536 rows on (the tiled gradient, 2-D and 3-D) depends on its data and schedule alone: the
same bits whatever else is asked for, and the losses and the last gradient of the iterations that were run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lists(n, seed, ks=(12, 6, 24), hubs=()):
    rng = np.random.default_rng(seed)
    out = []
    for q, k in enumerate(ks):
        p = (np.arange(n)[:, None] + rng.integers(1, 300, size=(n, k))) % n if q == 0 else rng.integers(0, n, size=(n, k))
        for h, size in hubs:
            p[rng.choice(n, size=size * k // sum(ks), replace=False), 0] = h
        out.append(np.stack([np.repeat(np.arange(n), k), p.reshape(-1)], 1).astype(np.uint32))
    return out


HUBS = [(0, 600), (129, 450), (65000, 1500), (777, 6000)]


@pytest.mark.parametrize("n,dim", [(65537, 2), (66001, 3)])
def test_asking_for_losses_changes_nothing(lib, n, dim):
    x = np.random.default_rng(3).normal(size=(n, 8)).astype(np.float32)
    cfg = lib.Configuration(initialization=lib.Initialization.Random(3), seed=5, num_iters=(14, 13, 13), snapshots=[5, 20, 40],
                            embedding_dimensions=dim,
                            pair_configuration=lib.PairConfiguration.AllProvided(*_lists(n, 11, hubs=HUBS)))
    a, sa = lib.fit_transform(x, cfg)
    b, sb, loss = lib.fit_transform(x, cfg, loss_trace=True)
    assert np.array_equal(a, b) and np.array_equal(sa, sb)
    assert loss.shape == (40,) and (loss > 0).all()


# weights 3, 3, 1 and 1, 0, 1 in the last iteration; exactly the first size and a ragged one
@pytest.mark.parametrize("n,dim,end", [(65536, 2, 164), (66001, 3, 219)])
def test_last_gradient_and_loss(lib, orc, n, dim, end):
    """out_grad leaves the state's bits alone, is the gradient that Adam took (its step on it gives y, m, v bit for bit),
    and lies within the bounds of the other gradient tests: 1e-5 of a row's sum of |contributions|, the loss (a sum of
    positive terms, at most 512 additions after one another and 8 roundings a term: 3e-5) 3e-5 of itself."""
    pairs = _lists(n, n, hubs=HUBS)
    y0 = np.random.default_rng(dim).normal(0, 4, size=(n, dim)).astype(np.float32)
    state = [(y0.copy(), np.zeros_like(y0), np.zeros_like(y0)) for _ in range(2)]
    g = lib.stages.optimize_steps(*state[0], *pairs, 1.0, 100, 100, end - 14, end)
    lib.stages.optimize_steps(*state[1], *pairs, 1.0, 100, 100, end - 14, end, want_grad=False)
    assert all(np.array_equal(p, q) for p, q in zip(*state))
    y, m, v = y0.copy(), np.zeros_like(y0), np.zeros_like(y0)
    lib.stages.optimize_steps(y, m, v, *pairs, 1.0, 100, 100, end - 14, end - 1, want_grad=False)
    _, g64, absum = orc.grad(y, *pairs, *((3.0, 3.0, 1.0) if end < 200 else (1.0, 0.0, 1.0)), with64=True)
    assert (np.abs(g[:-1] - g64[:-1]) <= 1e-5 * absum + 1e-30).all()
    assert abs(g[-1, 0] - g64[-1, 0]) <= 3e-5 * abs(g64[-1, 0])
    orc.adam(y, g, m, v, 1.0, end - 1)
    assert all(np.array_equal(p, q) for p, q in zip((y, m, v), state[0]))


@pytest.mark.parametrize("n,dim", [(66000, 2), (65537, 3), (3000, 2), (20000, 3)])
def test_output_buffer_address_changes_nothing(lib, n, dim):
    """fit_transform_device into a buffer 8 bytes off the 16-byte grid, after an odd and an even number of iterations."""
    import torch

    x = np.random.default_rng(3).normal(size=(n, 8)).astype(np.float32)
    pairs = lib.PairConfiguration.AllProvided(*_lists(n, 12))
    dx = torch.from_numpy(x).cuda()
    for iters in ((6, 6, 6), (6, 6, 7)):
        cfg = lib.Configuration(initialization=lib.Initialization.Random(3), seed=5, num_iters=iters, embedding_dimensions=dim,
                                pair_configuration=pairs)
        out = torch.zeros(dim * n + 2, device="cuda")
        torch.cuda.synchronize()
        lib.fit_transform_device(dx.data_ptr(), n, 8, out.data_ptr() + 8, cfg)
        a, _ = lib.fit_transform(x, cfg)
        assert np.array_equal(out[2:].cpu().numpy().reshape(n, dim), a)


@pytest.mark.parametrize("n,dim", [(65536, 2), (90001, 3)])
def test_a_schedule_cut_into_calls_changes_nothing(lib, n, dim):
    """Twenty iterations across the last change of phase in one call, in two, and one by one; with the gradient asked for in
    some."""
    pairs = _lists(n, n, hubs=HUBS)
    y0 = np.random.default_rng(dim).normal(0, 4, size=(n, dim)).astype(np.float32)
    states = []
    for cuts in ((190, 210), (190, 200, 210), (190, *range(191, 211))):
        y, m, v = y0.copy(), np.zeros_like(y0), np.zeros_like(y0)
        for a, b in zip(cuts, cuts[1:]):
            lib.stages.optimize_steps(y, m, v, *pairs, 1.0, 100, 100, a, b, want_grad=b % 3 == 0)
        states.append((y, m, v))
    for s in states[1:]:
        assert all(np.array_equal(p, q) for p, q in zip(states[0], s))


@pytest.mark.parametrize("dim", [2, 3])
def test_non_finite_coordinates_spread_as_in_the_reference(lib, orc, dim):
    """A NaN in one coordinate of a point makes its pairs' factors NaN, and so all coordinates of its partners' gradients; an
    infinite one makes the factors 0, and only its own coordinate NaN (0 times infinity). The mid-near pairs are left out
    in the last phase, where their weight is 0 (the engine skips them there, in every form)."""
    n = 65600
    pairs = _lists(n, 5, hubs=HUBS)
    y = np.random.default_rng(dim).normal(0, 4, size=(n, dim)).astype(np.float32)
    y[300, 0], y[40000, dim - 1], y[65599] = np.nan, np.nan, np.nan
    y[7, 1], y[50001, 0], y[12345] = np.inf, -np.inf, np.inf
    for itr, w in ((150, (3.0, 3.0, 1.0)), (220, (1.0, 0.0, 1.0))):
        g = lib.stages.optimize_steps(y.copy(), np.zeros_like(y), np.zeros_like(y), *pairs, 1.0, 100, 100, itr, itr + 1)
        with np.errstate(all="ignore"):
            e = orc.grad(y, pairs[0], pairs[1] if w[1] else pairs[1][:0], pairs[2], *w)
        assert np.array_equal(np.isnan(g[:-1]), np.isnan(e[:-1]))
        assert 300 < np.isnan(e[:-1]).any(1).sum() < n // 10


def _moment_gradient(lib, y, pairs):
    """The gradient in the last phase, from Adam's first moment after 14 iterations with a learning rate of 0."""
    m = np.zeros_like(y)
    lib.stages.optimize_steps(y.copy(), m, np.zeros_like(y), *pairs, 0.0, 100, 100, 220, 234, want_grad=False)
    return m / (1 - 0.9 ** 14)


# around 2.1e9, 2.5e9 and 1e30, and at the largest numbers of both signs, in all coordinates and in one
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("at", [2.1e9, 2.5e9, 1e30, -1e30, 3.4e38, -3.4e38])
def test_points_anywhere_have_only_their_own_pairs(lib, orc, dim, at):
    """Far points, whose true factors are 0 or tiny; the places that fill a tile's lists up must not act on them either."""
    n = 65537
    pairs = _lists(n, 8)
    rng = np.random.default_rng(dim)
    y = rng.normal(0, 4, size=(n, dim)).astype(np.float32)
    y[::3000] = np.float32(at)
    y[5::3000] = np.nextafter(np.float32(at), np.float32(0))
    y[9::3000, 0] = np.float32(at)
    g = _moment_gradient(lib, y, pairs)
    with np.errstate(all="ignore"):
        _, e64, absum = orc.grad(y, *pairs, 1.0, 0.0, 1.0, with64=True)
    assert np.isfinite(g).all() and np.isfinite(absum).all()
    assert (np.abs(g - e64[:-1]) <= 1e-5 * absum + 1e-26).all()


def test_points_without_near_and_far_pairs(lib):
    """Points with no pairs at all, or mid-near ones only, among others of their window: no gradient, wherever they lie."""
    n = 65537
    alone = np.array([0, 5, 130, 65536])
    pnn, pmn, pfp = (p[~np.isin(p, alone).any(1)] for p in _lists(n, 8))
    pmn = np.concatenate([pmn, np.array([[5, 9]], np.uint32)])
    y = np.random.default_rng(1).normal(0, 4, size=(n, 2)).astype(np.float32)
    y[alone] = [[np.inf, 1], [3, 4], [np.nan, np.nan], [-1e30, 1e30]]
    g = _moment_gradient(lib, y, (pnn, pmn, pfp))
    assert (g[alone] == 0).all() and np.isfinite(g).all()
