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
