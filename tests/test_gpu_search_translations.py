"""The translations of the register passes.  Where their line DFTs split coprime factors (test_gpu_regsides.PFA)
scores agree with the radix-stage passes to rounding only, so the translation is held against the float64
correlation volume: its score there is the largest to within the float32 error of both (twice SCORE_RTOL).
Where both run the same arithmetic: the sides and modes that test_gpu_regsides.py leaves out, bit for bit."""
import numpy as np
import pytest
import torch

from oracle import vesper_oracle as orc
from test_gpu_regsides import PFA, SCORE_RTOL, SIDES, _fields

pytestmark = pytest.mark.gpu
MIX = (0.5, 0.7, 0.1, 0.3, 0.2)   # alpha, vstd, vave, pstd, pave


@pytest.mark.parametrize("mode,d", [("VecProduct", 13)] +
                         [(m, d) for m in ("VecProduct", "prob", "CC", "PCC", "Laplacian") for d in PFA[m]])
def test_split_sides_find_the_largest_score(dev, mode, d):
    from vesper_python_gb300 import vesper as vg
    rng = np.random.default_rng(d)
    tgt, qry = _fields(rng, d), _fields(rng, d)
    ave, prob = 0.37, mode == "prob"
    td, tv, tp = (dev.to_dev(a) for a in tgt)
    qd, qv, qp = (dev.to_dev(a) for a in qry)
    spec = vg.target_spectra_device(td, tv, mode, ave, probs=tp if prob else None, dev=dev)
    mats = dev.to_dev(vg.rot_matrices(np.concatenate([[[0, 0, 0], [90, 0, 180]], rng.uniform(0, 180, (5, 3))])))
    scores, lin = (t.cpu().numpy() for t in vg.search_device(
        spec, qd, qv, mode, ave, mats, probs=qp if prob else None, mix=MIX if prob else None, opts=(1, 0, 0), dev=dev))
    rd, rv, rp = (t.cpu().numpy() if t is not None else None for t in vg.rot_gather_device(qd, qv, mats, qp, dev=dev))

    def fields(data, vec, probs):
        if prob:
            return [vec[..., 0], vec[..., 1], vec[..., 2], *probs]
        return orc.mode_field(mode, data, vec, ave)

    ts = orc.target_spectra(fields(*tgt))
    for r in range(len(mats)):
        vols = orc.correlate(ts, fields(rd[r], rv[r], rp[r]), fp64=True, workers=8)
        want = [sum(vols[:3]), sum(vols[3:])] if prob else [sum(vols)]
        if prob:
            want.append((1 - MIX[0]) * (want[0] - MIX[2]) / MIX[1] + MIX[0] * (want[1] - MIX[4]) / MIX[3])
        for s, v in enumerate(want):
            tol = 2 * SCORE_RTOL * np.abs(v).max()
            assert abs(scores[r, s] - v.max()) <= tol
            assert v.reshape(-1)[lin[r, s]] >= v.max() - tol, (r, s)


@pytest.mark.parametrize("mode", ["Overlap", "PCC", "Laplacian", "prob"])
def test_remaining_sides_equal_radix_stage_passes(dev, mode):
    from vesper_python_gb300 import vesper as vg
    for d in SIDES:
        if d in PFA[mode] or not (d > 91 or (mode in ("Overlap", "PCC") and d % 3)):
            continue
        rng = np.random.default_rng(d)
        td, tv, tp = (dev.to_dev(a) for a in _fields(rng, d))
        qd, qv, qp = (dev.to_dev(a) for a in _fields(rng, d))
        prob = mode == "prob"
        spec = vg.target_spectra_device(td, tv, mode, 0.37, probs=tp if prob else None, dev=dev)
        mats = dev.to_dev(vg.rot_matrices(np.concatenate([[[0, 0, 0], [0, 90, 270]], rng.uniform(0, 360, (3, 3))])))
        kw = dict(probs=qp if prob else None, mix=MIX if prob else None, dev=dev)
        ref = vg.search_device(spec, qd, qv, mode, 0.37, mats, opts=(0, 0, 0), **kw)
        got = vg.search_device(spec, qd, qv, mode, 0.37, mats, opts=(1, 0, 0), batch=4, **kw)
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1]), d
