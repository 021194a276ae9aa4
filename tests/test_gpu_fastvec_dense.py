"""fastVEC of maps that are not mostly zero: the x stage with a voxel per thread (grids of 150,000 voxels and more,
above and below 80,000 listed ones) and the z stage's dense rows where its weights are not staged (wide
windows), an odd number of rows and mixed blocks among them.  The bar is that of test_gpu_fastvec_lists.py."""
import numpy as np
import pytest
import torch

from test_gpu_fastvec_lists import _direct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,d,dw,shift,g", [((46, 45, 48), 45, 1.0, 0.5, 5.0), ((48, 50, 47), 54, 0.85, 0.25, 8.0),
                                                ((27, 31, 52), 70, 0.55, -4.0, 24.0), ((40, 33, 21), 81, 0.4, 0.0, 20.0)])
@pytest.mark.parametrize("density", [1.0, 0.9, 0.5, 0.3, 0.1])
def test_dense_maps(dev, shape, d, dw, shift, g, density):
    from vesper_python_gb300 import vesper as vg
    rng = np.random.default_rng(d)
    src = rng.uniform(0.1, 2.0, shape).astype(np.float32)
    src[rng.random(shape) >= density] = 0
    src[3, 4:7] = 0                  # rows without a value
    src[5, :, : shape[2] // 2] = 0   # rows of another density
    data, data32, vec = vg.fastvec_device(torch.from_numpy(src).to(dev.device), 1.0, [0.0] * 3, d, dw, [shift] * 3, g, dev=dev)
    rd, rv = _direct(src, 1.0, [0.0] * 3, d, dw, [shift] * 3, g)
    data, vec = data.cpu().numpy(), vec.cpu().numpy()
    assert np.array_equal(data != 0, rd != 0)
    assert np.all(np.abs(data - rd) <= 1e-12 * np.abs(rd))
    assert np.max(np.abs(vec - rv), initial=0) < 2e-6
    assert np.array_equal(data32.cpu().numpy(), data.astype(np.float32))
