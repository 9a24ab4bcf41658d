"""Move targets at the edges of the degree tiers, against the CPU oracle.

One vertex of every degree around the tiers' limits, their 32-edge chunks and
table sizes, with all neighbours in distinct communities (full tables) or in
few (many edges a slot).  Weights are unit (many tied gains), integers
(integer tables) or multiples of 1/2 (FP64 tables); every sum is exact, so the
targets equal the oracle's bit for bit under both tie rules."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEGREES = [1, 2, 4, 5, 8, 9, 16, 17, 31, 32, 33, 64, 65, 96, 97, 160, 191, 192, 193, 256, 257, 383, 385, 640, 641, 767,
           768, 769, 1023, 1025, 1281, 1535, 1536, 1537, 1793, 2047, 2048, 2049, 3071, 3072, 3073, 4097, 6143, 6144,
           6145, 7169, 8193, 12287, 12288, 12289, 20000]


@pytest.mark.parametrize("weights", ["unit", "int", "half"])
@pytest.mark.parametrize("tie", [0, 1])
@pytest.mark.parametrize("ncomm", [40000, 37, 1])
def test_targets_at_tier_edges(nido_lib, ctx, orc, weights, tie, ncomm):
    rng = np.random.default_rng(5)
    nv = 40000
    at = rng.permutation(nv)[:len(DEGREES)]
    deg = np.zeros(nv, np.int64)
    deg[at] = DEGREES
    off = np.zeros(nv + 1, np.int64)
    np.cumsum(deg, out=off[1:])
    adj = np.concatenate([rng.permutation(nv)[:d] for d in deg[deg > 0]]).astype(np.int64)
    w = {"unit": np.ones(len(adj)), "int": rng.integers(1, 9, len(adj)).astype(np.float64),
         "half": 0.5 * rng.integers(1, 9, len(adj))}[weights]
    comm = rng.permutation(nv) if ncomm == nv else rng.integers(0, ncomm, nv)
    comm = comm.astype(np.int64)
    with nido_lib.Graph(ctx, nido_lib.Csr(off, adj, w), 1) as g:
        k, m = g.vertex_weights()
        g.set_community_ids(comm)
        g.louvain_update(0, tie)
        _, got, a = g.state()
    assert np.array_equal(a, orc.community_weights(comm, k))
    want, _ = orc.move(off, adj, w, comm, a, k, m, 0, nv, tie=tie)
    bad = np.flatnonzero(got != want)
    assert len(bad) == 0, [(int(deg[v]), int(got[v]), int(want[v])) for v in bad[:10]]
