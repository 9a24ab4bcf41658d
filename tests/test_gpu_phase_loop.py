"""The persistent kernels of small phases (the phase loop, and the coarsening with
the next phase's set-up; the default) against the host driven loop and the
separate stages (host_loop): on weights whose sums are exact every partition,
every phase's Q and every loop count are identical, under both tie rules, for
integer and FP64 tables, with hubs of one and of several segments, communities of
more and of fewer members than a block lists in order, colour-class batches,
loop caps and undone sweeps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def hub_graph(capi, nv, hubs, weights, seed):
    """A sparse ring with hubs of the given degrees."""
    rng = np.random.default_rng(seed)
    u, v = [np.arange(nv - 1)], [np.arange(1, nv)]
    for i, d in enumerate(hubs):
        u.append(np.full(d, 7 * i + 3))
        v.append(rng.permutation(nv)[:d])
    u, v = np.concatenate(u), np.concatenate(v)
    keep = u != v
    u, v = u[keep], v[keep]
    w = {"unit": np.ones(len(u)), "int": rng.integers(1, 9, len(u)).astype(np.float64),
         "half": 0.5 * rng.integers(1, 9, len(u))}[weights]
    src, dst, ww = np.concatenate([u, v]), np.concatenate([v, u]), np.concatenate([w, w])
    order = np.argsort(src, kind="stable")
    off = np.zeros(nv + 1, np.int64)
    np.cumsum(np.bincount(src, minlength=nv), out=off[1:])
    return capi.Csr(off, dst[order].astype(np.int64), ww[order])


def bits(x):
    return np.asarray(x, np.float64).view(np.uint64)


def same(a, b):
    (ca, sa), (cb, sb) = a, b
    assert np.array_equal(ca, cb)
    n = sb.phases
    assert sa.phases == n and sa.total_loops == sb.total_loops
    assert np.array_equal(bits(sa.q_phase[:n]), bits(sb.q_phase[:n]))
    assert list(sa.loops_phase[:n]) == list(sb.loops_phase[:n])
    assert list(sa.nv_phase[:n]) == list(sb.nv_phase[:n]) and list(sa.ne_phase[:n]) == list(sb.ne_phase[:n])
    assert sa.move_bytes == sb.move_bytes and sa.edges_scanned == sb.edges_scanned


@pytest.mark.parametrize("weights", ["unit", "int", "half"])
@pytest.mark.parametrize("nv,hubs", [(2, []), (33, [20]), (700, [650, 300]), (5000, [3072, 3073, 4097]),
                                     (30000, [12288, 12289, 25000])])
@pytest.mark.parametrize("nb,tie", [(1, 0), (2, 1), (5, 0)])
def test_equals_host_loop(nido_lib, ctx, weights, nv, hubs, nb, tie):
    G = hub_graph(nido_lib, nv, hubs, weights, nv)
    with nido_lib.Graph(ctx, G, nb) as g:
        a, b = g.run(tie=tie), g.run(tie=tie, host_loop=True)
    same(a, b)
    assert a[1].kernel_launches < b[1].kernel_launches  # the loop ran as one kernel a phase


@pytest.mark.parametrize("max_iter,tau", [(0, 1e-6), (1, 1e-6), (2, 1e-6), (500, 1e-2), (6, -1.0)])
def test_limits_and_colors(nido_lib, ctx, max_iter, tau):
    G = nido_lib.gen_sbm(9001, cmin=16, cmax=1024, avg_degree=18.0, wmode=nido_lib.W_INT8, seed=3)
    for colors in (False, True):
        with nido_lib.Graph(ctx, G, 2) as g:
            same(g.run(tau=tau, max_iter=max_iter, color_batches=colors),
                 g.run(tau=tau, max_iter=max_iter, color_batches=colors, host_loop=True))


def test_batches_equal_host_loop(nido_lib, ctx):
    gs = [hub_graph(nido_lib, nv, hubs, "int", nv) for nv, hubs in
          [(2, []), (40, [30]), (900, [700]), (6000, [3500]), (20000, [15000, 13000])]]
    gs += [nido_lib.gen_sbm(3000 + 17 * i, cmin=16, cmax=512, avg_degree=12.0, wmode=nido_lib.W_INT8, seed=i)
           for i in range(20)]
    for nb, tie, max_iter in ((1, 0, 500), (2, 1, 500), (3, 0, 2)):
        with nido_lib.Batch(ctx, gs, nb) as B:
            a, b = B.run(tie=tie, max_iter=max_iter), B.run(tie=tie, max_iter=max_iter, host_loop=True)
        for x, y in zip(a[0], b[0]):
            assert np.array_equal(x, y)
        assert np.array_equal(bits(a[1]), bits(b[1]))
        assert np.array_equal(a[2], b[2]) and np.array_equal(a[3], b[3])
