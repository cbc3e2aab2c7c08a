"""Buffers of the outputs after a refused mesh or cluster count (CPU; the library is a
stand-in): the context keeps what it holds when acvd_set_mesh or acvd_set_labels refuses its
arguments, so the outputs still have those sizes.
"""
import ctypes

import numpy as np
import pytest

from acvd_gb300.engine import AcvdError, Engine


class _Lib:
    """Holds the sizes of the mesh that it took last; the outputs are as long as they can be."""

    def acvd_set_mesh(self, ctx, n, pts, nf, tri, row, col, ne, ev):
        if n <= 0 or nf <= 0 or ne <= 0 or np.ctypeslib.as_array(
                ctypes.cast(row, ctypes.POINTER(ctypes.c_int32)), (n + 1,))[n] != 2 * ne:
            return 1
        self.n, self.nf, self.ne = n, nf, ne
        return 0

    def acvd_set_labels(self, ctx, k, lab):
        if k <= 0 or k >= 1 << 21:
            return 1 if k <= 0 else 3
        self.k = k
        return 0

    def acvd_last_error(self, ctx):
        return b"refused"

    def acvd_get_labels(self, ctx, out):
        self.room = self.n
        return 0

    def acvd_get_boundary_edges(self, ctx, out, n):
        self.room = self.ne
        n._obj.value = 0
        return 0

    def acvd_get_dual_mesh(self, ctx, out, n):
        self.room = 3 * self.nf
        n._obj.value = 0
        return 0

    def acvd_get_clusters(self, ctx, *a):
        self.room = self.k
        return 0

    def acvd_destroy(self, ctx):
        pass


def _mesh(n):
    """A strip of n triangles; the rings are not looked at."""
    tri = np.stack([np.arange(n), np.arange(1, n + 1), np.arange(2, n + 2)], 1).astype(np.int32)
    ev = np.zeros((2 * n + 1, 2), dtype=np.int32)
    row = np.zeros(n + 3, dtype=np.int32)
    row[-1] = ev.size
    return np.zeros((n + 2, 3)), tri, row, np.zeros(ev.size, dtype=np.int32), ev


@pytest.fixture
def engine(monkeypatch):
    import acvd_gb300.engine as eng
    e = Engine.__new__(Engine)
    e._lib, e.ctx, e.n, e.k, e.n_edges = _Lib(), 1, 0, 0, 0
    monkeypatch.setattr(eng, "load", lambda *a, **k: e._lib)
    sizes = []
    empty = np.empty

    def count(shape, dtype=float):
        sizes.append(int(np.prod(shape)))
        return empty(shape, dtype=dtype)

    monkeypatch.setattr(eng.np, "empty", count)
    e.sizes = sizes
    yield e
    e.ctx = None


@pytest.mark.parametrize("what", ["short_rings", "no_faces", "no_edges"])
@pytest.mark.parametrize("output", ["labels", "boundary_edges", "dual_mesh"])
def test_outputs_keep_the_mesh_that_is_held(engine, what, output):
    engine.set_mesh(*_mesh(50))
    pts, tri, row, col, ev = _mesh(4)
    if what == "short_rings":
        row[-1] -= 2
    elif what == "no_faces":
        tri = tri[:0]
    else:
        ev = ev[:0]
    with pytest.raises(AcvdError):
        engine.set_mesh(pts, tri, row, col, ev)
    engine.sizes.clear()
    getattr(engine, output)()
    assert engine.sizes[0] >= engine._lib.room


@pytest.mark.parametrize("k", [0, -3, 1 << 21])
def test_outputs_keep_the_clusters_that_are_held(engine, k):
    engine.set_mesh(*_mesh(50))
    engine.set_labels(7, np.zeros(52, dtype=np.int32))
    with pytest.raises(AcvdError):
        engine.set_labels(k, np.zeros(52, dtype=np.int32))
    engine.sizes.clear()
    engine.clusters()
    assert engine.sizes[0] == engine._lib.room == engine.k
