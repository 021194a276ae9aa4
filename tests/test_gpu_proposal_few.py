"""The 8-channel rotation scores and gradients on both sides of the rules that send small calls to the
general kernels: scores against those of nine channels (general kernel, the ninth zero), bit for bit;
gradients against the float64 oracle, float32 sums of m terms within m 2^-24 of the sum of the terms'
magnitudes."""
import numpy as np
import pytest
import torch

from oracle import proposal_oracle as po
from oracle import vesper_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 3, 8, 9, 12, 13, 17, 18])
@pytest.mark.parametrize("nrot", [1, 455, 456, 500, 2431, 2432, 2500])
def test_scores(dev, d, nrot):
    from vesper_python_gb300 import proposal as P
    from vesper_python_gb300 import vesper as vg
    net = P.ProposalNet(dev, seed=1)
    g = torch.Generator().manual_seed(d + nrot)
    t, q = (torch.randn((8, d, d, d), generator=g).to(dev.device) for _ in range(2))
    mats = dev.to_dev(vg.rot_matrices(orc.calc_angle_comb(10.0)[::9][:nrot]))
    ninth = [torch.cat([a, torch.zeros_like(a[:1])]).contiguous() for a in (t, q)]
    assert torch.equal(net.score(t, q, mats), net.score(*ninth, mats))


@pytest.mark.parametrize("d,nrot", [(6, 900), (7, 759), (7, 760), (8, 303), (8, 304), (9, 1)])
def test_gradients(dev, d, nrot):
    from vesper_python_gb300 import proposal as P
    from vesper_python_gb300 import vesper as vg
    net = P.ProposalNet(dev, seed=1)
    rng = np.random.default_rng(d)
    K, n = 8, d ** 3
    ET, EQ = (rng.normal(size=(K, d, d, d)).astype(np.float32) for _ in range(2))
    mats = vg.rot_matrices(orc.calc_angle_comb(10.0)[::27][:nrot])
    maps = [po.src_map(d, F) for F in mats]
    gs = rng.normal(size=nrot).astype(np.float32)
    gT, gQ = (torch.zeros((K, d, d, d), device=dev.device) for _ in range(2))
    net.score_backward(dev.to_dev(ET), dev.to_dev(EQ), dev.to_dev(mats), dev.to_dev(gs), gT, gQ)
    t64, q64, g64 = ET.reshape(K, n).astype(np.float64), EQ.reshape(K, n).astype(np.float64), gs.astype(np.float64)
    oT, oQ = po.score_bwd(t64, q64, maps, g64)
    aT, aQ = po.score_bwd(np.abs(t64), np.abs(q64), maps, np.abs(g64))
    for got, ref, mag in ((gT, oT, aT), (gQ, oQ, aQ)):
        err = np.abs(got.cpu().numpy().reshape(K, n) - ref)
        # a query voxel's sum runs over the rotations and, for each, the target voxels that read it
        assert np.all(err <= mag * (4 * nrot + 256) * 2.0 ** -24 + 1e-30)
