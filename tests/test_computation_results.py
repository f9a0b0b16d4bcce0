"""The Python mirror's accessors over the batch's results (no GPU: a stand-in for the C library)."""
import ctypes

import numpy as np
import pytest

from lc0_b200 import _lib, network


class _FakeLib:
    """The calls of a computation's life, on arrays of its own; counts the calls for results."""

    def __init__(self, moves):
        self.n, self.moves, self.reads = 0, moves, 0

    def b200_comp_add_inputs(self, h, masks, values, n):
        self.n += n
        return 0

    def b200_comp_compute(self, h):
        self.qdm = np.random.default_rng(self.n).random((self.n, 3), np.float32)
        self.probs = np.random.default_rng(self.n + 1).random((self.n, 256), np.float32)
        self.counts = np.arange(self.n, dtype=np.int32) % 257
        return 0

    def b200_comp_batch_size(self, h):
        return self.n

    def b200_comp_results(self, h, qdm, probs, moves):
        self.reads += 1
        qdm._obj.value = self.qdm.ctypes.data
        probs._obj.value = self.probs.ctypes.data if self.moves else None
        moves._obj.value = self.counts.ctypes.data if self.moves else None
        return 0

    def b200_comp_q(self, h, i):
        return -1.0  # what the accessors return for a batch that was not computed

    def b200_comp_legal_policy(self, h, i, probs, n):
        return 1

    def b200_comp_destroy(self, h):
        pass


def _computation(lib):
    c = object.__new__(network.NetworkComputation)
    c._lib, c._net, c._h = lib, None, ctypes.c_void_p(1)
    c._results, c._computed = None, False
    return c


def _add(c, n):
    c.add_inputs(np.zeros((n, 112), np.uint64), np.zeros((n, 112), np.float32))


def test_results_are_fetched_once_and_only_when_asked_for():
    lib = _FakeLib(moves=True)
    c = _computation(lib)
    _add(c, 5)
    c.compute_blocking()
    assert lib.reads == 0  # a caller that reads none of them (raw policies, one sample) does not pay for the batch
    for i in range(5):
        q, d, m = c.get_q_val(i), c.get_d_val(i), c.get_m_val(i)
        assert all(type(v) is float for v in (q, d, m)) and np.array_equal(np.float32([q, d, m]), lib.qdm[i])
        p = c.legal_policy(i)
        assert p.dtype == np.float32 and np.array_equal(p, lib.probs[i, :lib.counts[i]])
        p[:] = 0  # a copy of the caller's own
        assert np.array_equal(c.legal_policy(i), lib.probs[i, :lib.counts[i]])
    assert lib.reads == 1
    for bad in (-1, 5):
        with pytest.raises(IndexError):
            c.get_q_val(bad)
    _add(c, 3)  # more samples: not computed yet
    assert c.get_q_val(0) == -1.0
    c.compute_blocking()
    assert np.float32(c.get_m_val(7)) == lib.qdm[7, 2] and lib.reads == 2
    c.close()


def test_results_without_moves_and_of_an_empty_batch():
    lib = _FakeLib(moves=False)
    c = _computation(lib)
    c.compute_blocking()
    with pytest.raises(IndexError):
        c.get_q_val(0)
    assert lib.reads == 0
    _add(c, 2)
    c.compute_blocking()
    assert np.float32(c.get_d_val(1)) == lib.qdm[1, 1]
    with pytest.raises(_lib.B200Error):
        c.legal_policy(0)
    c.close()
