"""Search with queries that fill part of their grid, whose empty tiles, steps and planes the register
passes leave out, against the radix-stage passes, which do not: bit for bit where both run the same
arithmetic (test_gpu_regsides.PFA lists the others), else to SCORE_RTOL and the same translations.
A ball, one off the centre, a voxel in a corner, a face; rotations, a scaling, a matrix with a column
of another length, one that is not finite."""
import numpy as np
import pytest
import torch

from test_gpu_regsides import PFA, SCORE_RTOL, _fields

pytestmark = pytest.mark.gpu


def _queries(d):
    x = np.stack(np.meshgrid(*[np.arange(d) - (d - 1) / 2] * 3, indexing="ij"))
    ball = (x ** 2).sum(0) < (0.4 * d) ** 2
    side = ((x - np.array([0.2 * d, -0.1 * d, 0.15 * d])[:, None, None, None]) ** 2).sum(0) < (0.15 * d) ** 2
    corner = np.zeros((d, d, d), bool)
    corner[d - 1, 0, d - 1] = True
    face = np.zeros((d, d, d), bool)
    face[0] = True
    return {"ball": ball, "side": side, "corner": corner, "face": face}


@pytest.mark.parametrize("mode", ["VecProduct", "CC", "prob"])
@pytest.mark.parametrize("d", [27, 28, 36, 45, 50, 55, 64, 75, 80, 99])
def test_partly_filled_queries(dev, mode, d):
    from vesper_python_gb300 import vesper as vg
    rng = np.random.default_rng(d)
    prob = mode == "prob"
    data, vec, probs = _fields(rng, d)
    td, tv, tp = (dev.to_dev(a) for a in (data, vec, probs))
    spec = vg.target_spectra_device(td, tv, mode, 0.37, probs=tp if prob else None, dev=dev)
    mats = vg.rot_matrices(np.concatenate([[[0, 0, 0], [90, 0, 180]], rng.uniform(0, 360, (7, 3))]))
    mats[3] *= np.float32(1.25)
    mats[4, :, 2] *= np.float32(0.05)
    mats[5, :, 0] *= np.float32(40)
    mats[6] *= np.float32(1e30)
    mats[7] = np.nan
    mats = dev.to_dev(mats)
    for name, on in _queries(d).items():
        qd, qv, qp = (dev.to_dev(np.where(m, a, 0).astype(a.dtype)) for m, a in
                      ((on, data), (on[..., None], vec), (on[None], probs)))
        kw = dict(probs=qp if prob else None, mix=(0.5, 0.7, 0.1, 0.3, 0.2) if prob else None, dev=dev)
        ref = vg.search_device(spec, qd, qv, mode, 0.37, mats, opts=(0, 0, 0), **kw)
        got = vg.search_device(spec, qd, qv, mode, 0.37, mats, opts=(1, 0, 0), batch=4, **kw)
        if d not in PFA[mode]:
            assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1]), name
        else:
            assert float((got[0] - ref[0]).abs().max()) <= SCORE_RTOL * float(ref[0].abs().max()), name
