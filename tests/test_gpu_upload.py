"""Uploads of host arrays around the size from which pageable memory is staged by
host threads (8 MB of ids): the device CSR equals the arrays, from pageable and
from page-locked memory, and ids out of range are refused wherever they stand."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ring(nv, ne, seed):
    rng = np.random.default_rng(seed)
    off = np.sort(rng.integers(0, ne + 1, nv + 1)).astype(np.int64)
    off[0], off[-1] = 0, ne
    return off, rng.integers(0, nv, ne).astype(np.int64), rng.random(ne)


@pytest.mark.parametrize("ne", [1, 1048575, 1048576, 1048577, 1500001])
@pytest.mark.parametrize("pinned", [False, True])
def test_upload_equals_arrays(nido_lib, ctx, ne, pinned):
    off, adj, w = ring(1001, ne, ne)
    if pinned:
        nido_lib.host_register(adj)
        nido_lib.host_register(w)
    try:
        with nido_lib.Graph(ctx, nido_lib.Csr(off, adj, w), 2) as g:
            got = g.download()
    finally:
        if pinned:
            nido_lib.host_unregister(adj)
            nido_lib.host_unregister(w)
    assert np.array_equal(got.off, off) and np.array_equal(got.adj, adj) and np.array_equal(got.w, w)


@pytest.mark.parametrize("ne", [4097, 1048577])
@pytest.mark.parametrize("bad", [-1, 1001, (1 << 32) + 5, -(1 << 40)])
def test_bad_ids_are_refused(nido_lib, ctx, ne, bad):
    off, adj, w = ring(1001, ne, 3)
    for at in (0, ne // 2, ne - 1):
        x = adj.copy()
        x[at] = bad
        with pytest.raises(nido_lib.NidoError):
            nido_lib.Graph(ctx, nido_lib.Csr(off, x, w), 2)
