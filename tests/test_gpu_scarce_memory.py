"""Calls that get no memory beyond what they cannot do without: the same results, by the slower way. (The allocations are
refused on the host by a hook of the calling thread.)"""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _scarce(lib):
    hook = lib._abi.lib().pacmap_debug_scarce_memory
    hook(1)
    try:
        yield
    finally:
        hook(0)


def test_copies_without_page_locked_slots(lib, orc):
    """42 MB up and down, past the sizes from which copies are staged."""
    x = np.random.default_rng(0).uniform(-2, 3, size=(105001, 100)).astype(np.float32)
    with _scarce(lib):
        got = lib.stages.preprocess(x)[0]
    assert np.array_equal(got, orc.preprocess(x)[0])
    assert np.array_equal(lib.stages.preprocess(x)[0], got)
