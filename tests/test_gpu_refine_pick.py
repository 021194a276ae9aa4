"""The refined top-N never holds a slot that the reference's filter drops, also where fewer slots than N
are left: the host-driven refinement, which lists only the kept angles, gives the same models."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kept", [0, 1, 5, 27, 31, 32, 33])
def test_pick_leaves_dropped_slots_out(dev, kept):
    from vesper_python_gb300 import _native
    from vesper_python_gb300 import vesper as vg
    nslot, N, d = 54, 32, 12
    g = torch.Generator().manual_seed(kept)
    where = torch.randperm(nslot, generator=g)[:kept].sort().values
    valid = torch.zeros(nslot, dtype=torch.bool)
    valid[where] = True
    scores = torch.randint(-3, 3, (nslot, 1), generator=g).float()
    scores[~valid] = 50.0
    lin = torch.randint(0, d ** 3, (nslot, 1), generator=g, dtype=torch.int32)
    rows = torch.randint(0, 1000, (nslot,), generator=g)
    t = [x.contiguous().to(dev.device) for x in (scores, lin, valid, rows)]
    out = [torch.full((N,), -7, dtype=k, device=dev.device) for k in (torch.int32, torch.int64, torch.float32, torch.int64)]
    out += [torch.empty((N, 3, 3), device=dev.device), torch.empty((N, 3), dtype=torch.int32, device=dev.device)]
    c_ = lambda x: ctypes.c_void_p(x.data_ptr())  # noqa: E731
    _native.check(dev.lib.vesper_refine_pick(c_(t[0]), c_(t[1]), 1, c_(t[2]), c_(t[3]), nslot, N,
                                             c_(vg.lattice_rot_matrices_device(dev)), d, *[c_(o) for o in out],
                                             dev.stream))
    best = sorted(where.tolist(), key=lambda i: (-float(scores[i, 0]), i))[:N]
    want = best + [-1] * (N - len(best))
    assert out[0].tolist() == want
    sel = [max(i, 0) for i in want]
    assert out[1].tolist() == rows[sel].tolist() and out[3].tolist() == lin[sel, 0].tolist()
    assert out[2].tolist() == scores[sel, 0].tolist()


@pytest.mark.parametrize("A,N", [(360.0, 40), (180.0, 150)])
def test_more_models_than_refined_rotations(dev, A, N):
    from vesper_python_gb300 import align, synth
    pair = synth.make_pair(70, 48, 40, 14.0)
    items = [(dev.to_dev(pair.map1), dev.to_dev(pair.map2), 1.0, 1.0, pair.orig1, pair.orig2)]
    p = align.AlignParams(t=0.1, T=0.1, s=3.0, A=A, N=N)
    al, host = align.Aligner(dev), align.Aligner(dev)
    host.LATE_SIDE = 0
    ref = host.align_many(items, p)[0]
    assert ref.dim <= al.LATE_SIDE and 0 < len(ref.models) < N
    for r in (al.align_many(items, p)[0], al.align_many(items, p, graph=True)[0]):
        assert r.top == ref.top and len(r.models) == len(ref.models)
        for x, y in zip(r.models, ref.models):
            assert (tuple(x.angle), tuple(x.vec_trans), x.vec_score, x.dot_score, x.cc) == \
                (tuple(y.angle), tuple(y.vec_trans), y.vec_score, y.dot_score, y.cc)
