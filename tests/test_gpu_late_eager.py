"""Eager batches of small grids refine and rescore from the device's own results;
every pair's result equals the host-driven refinement's (all values, no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,n,A", [("VecProduct", 1, 30.0), ("VecProduct", 9, 30.0), ("Overlap", 3, 30.0),
                                      ("Laplacian", 2, 30.0), ("VecProduct", 2, 10.0)])
def test_eager_device_refinement_equals_host_driven(dev, mode, n, A):
    from vesper_python_gb300 import align, synth
    items = []
    for i in range(n):
        pair = synth.make_pair(40 + i, 48 + 16 * (i % 3), 40, 14.0 + 4 * (i % 3))
        items.append((dev.to_dev(pair.map1), dev.to_dev(pair.map2), 1.0, 1.0, pair.orig1, pair.orig2))
    p = align.AlignParams(t=0.1, T=0.1, s=3.0, A=A, N=10, mode=mode)
    al = align.Aligner(dev)
    got = al.align_many(items, p)
    again = al.align_many(items, p)
    assert max(r.dim for r in got) <= al.LATE_SIDE
    host = align.Aligner(dev)
    host.LATE_SIDE = 0
    ref = host.align_many(items, p)
    for g in (got, again):
        for a, b in zip(g, ref):
            assert (a.dim, a.std, a.ave, a.top) == (b.dim, b.std, b.ave, b.top)
            assert len(a.models) == len(b.models) == 10
            for x, y in zip(a.models, b.models):
                assert tuple(x.angle) == tuple(y.angle) and tuple(x.vec_trans) == tuple(y.vec_trans)
                assert (x.vec_score, x.overlap, x.cc, x.pcc, x.dot_score) == \
                    (y.vec_score, y.overlap, y.cc, y.pcc, y.dot_score)
                assert np.array_equal(x.translation, y.translation)


@pytest.mark.parametrize("fallback", ["none", "some", "all"])
def test_eager_proposal_refinement_equals_host_driven(dev, fallback):
    """With the rotation proposal: the same results as the host-driven refinement where no pair, some pairs or
    every pair falls back to the exhaustive search; only the pairs that fall back are refined again, and each
    pair has one event."""
    from vesper_python_gb300 import align
    from vesper_python_gb300 import proposal as P
    net = P.load_weights(dev)[0]
    items = []
    for seed in range(30_000_200, 30_000_204):
        m1, m2, o1, o2 = P.blob_pair_torch(seed, side=128, nblob=300, radius=35.0, device=dev.device)
        items.append((m1, m2, 1.0, 1.0, o1, o2))
    p = align.AlignParams(t=0.1, T=0.1, s=3.0, A=10.0, N=10, proposal=net, proposal_fallback_z=None)
    host = align.Aligner(dev)
    host.LATE_SIDE = 0
    if fallback != "none":
        host.align_many(items, p)
        z = sorted(host.proposal_info["z"])
        p.proposal_fallback_z = 0.5 * (z[1] + z[2]) if fallback == "some" else z[-1] + 1.0
    ref = host.align_many(items, p)
    fell = host.proposal_info["fallback"]
    assert sum(fell) == {"none": 0, "some": 2, "all": 4}[fallback]
    al = align.Aligner(dev)
    refined, late = [], al._late_stage
    al._late_stage = lambda sts, *a: (refined.append([st.index for st in sts]), late(sts, *a))
    for _ in range(2):
        del refined[:]
        al.pair_events = []
        got = al.align_many(items, p)
        assert max(r.dim for r in got) <= al.LATE_SIDE and al.proposal_info["fallback"] == fell
        assert refined == [[0, 1, 2, 3]] + ([[i for i in range(4) if fell[i]]] if any(fell) else [])
        assert len(al.pair_events) == 4
        for a, b in zip(got, ref):
            assert (a.dim, a.std, a.ave, a.top) == (b.dim, b.std, b.ave, b.top)
            assert len(a.models) == len(b.models) == 10
            for x, y in zip(a.models, b.models):
                assert (tuple(x.angle), tuple(x.vec_trans), x.vec_score, x.overlap, x.cc, x.pcc, x.dot_score) == \
                    (tuple(y.angle), tuple(y.vec_trans), y.vec_score, y.overlap, y.cc, y.pcc, y.dot_score)
                assert np.array_equal(x.translation, y.translation)


@pytest.mark.parametrize("mode", ["VecProduct", "Overlap", "Laplacian"])
def test_graph_refinement_equals_host_driven(dev, mode):
    """The captured form against the host-driven refinement: at these sides the eager form runs the captured
    form's own stage on the same side streams."""
    from vesper_python_gb300 import align, synth
    items = []
    for i in range(9):
        pair = synth.make_pair(80 + i, 48 + 16 * (i % 3), 40, 14.0 + 4 * (i % 3))
        items.append((dev.to_dev(pair.map1), dev.to_dev(pair.map2), 1.0, 1.0, pair.orig1, pair.orig2))
    p = align.AlignParams(t=0.1, T=0.1, s=3.0, A=30.0, N=10, mode=mode)
    host = align.Aligner(dev)
    host.LATE_SIDE = 0
    ref = host.align_many(items, p)
    al = align.Aligner(dev)
    for _ in range(2):
        al.pair_events = []
        for a, b in zip(al.align_many(items, p, graph=True), ref):
            assert (a.dim, a.std, a.ave, a.top) == (b.dim, b.std, b.ave, b.top)
            assert [(tuple(x.angle), tuple(x.vec_trans), x.vec_score, x.overlap, x.cc, x.pcc, x.dot_score)
                    for x in a.models] == \
                [(tuple(x.angle), tuple(x.vec_trans), x.vec_score, x.overlap, x.cc, x.pcc, x.dot_score) for x in b.models]
        assert len(al.pair_events) == 9
