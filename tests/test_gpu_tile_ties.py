"""Equal scores resolve to the first voxel, across the lanes, items and warps of the register passes'
last step, whatever the sign of a zero: a query or a target without a value scores 0 everywhere."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["VecProduct", "CC", "prob"])
@pytest.mark.parametrize("d", [27, 36, 48, 55, 64, 75, 80])
def test_ties_take_the_first_voxel(dev, mode, d):
    from vesper_python_gb300 import vesper as vg
    rng = np.random.default_rng(d)
    full = (dev.to_dev(rng.uniform(0.1, 2.0, (d, d, d))), dev.to_dev(rng.normal(size=(d, d, d, 3)).astype(np.float32)),
            dev.to_dev(rng.uniform(0.1, 1.0, (4, d, d, d)).astype(np.float32)))
    none = tuple(torch.zeros_like(t) for t in full)
    mats = dev.to_dev(vg.rot_matrices(rng.uniform(0, 180, (5, 3))))
    prob = mode == "prob"
    for t, q in ((full, none), (none, full)):
        spec = vg.target_spectra_device(t[0], t[1], mode, 0.0, probs=t[2] if prob else None, dev=dev)
        scores, lin = vg.search_device(spec, q[0], q[1], mode, 0.0, mats, probs=q[2] if prob else None,
                                       mix=(0.5, 0.7, 0.1, 0.3, 0.2) if prob else None, opts=(1, 0, 0), dev=dev)
        assert torch.all(lin == 0)
        assert torch.all(scores[..., :2 if prob else 1] == 0)
