"""The 8-channel rotation scores and their gradients against the float64 oracle:
odd and even sides, the largest side the staged kernels take (18) and the first
that falls back to the general ones (19), zero gradients, matrices that are no
rotations.  Bound: float32 sums of m terms are within m 2^-24 of the sum of the
terms' magnitudes (the features are float32 on both sides)."""
import numpy as np
import pytest
import torch

from oracle import proposal_oracle as po
from oracle import vesper_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [2, 3, 9, 12, 13, 15, 16, 18, 19])
def test_score8_and_gradients_vs_oracle(dev, d):
    from vesper_python_gb300 import proposal as P
    from vesper_python_gb300 import vesper as vg
    net = P.ProposalNet(dev, seed=1)
    rng = np.random.default_rng(d)
    K, n = 8, d ** 3
    ET = rng.normal(size=(K, d, d, d)).astype(np.float32)
    EQ = rng.normal(size=(K, d, d, d)).astype(np.float32)
    mats = vg.rot_matrices(np.concatenate([orc.calc_angle_comb(90.0)[:9], orc.calc_angle_comb(10.0)[3::397]]))
    mats[4] *= np.float32(1.3)                       # a scaling
    mats[7] = rng.normal(size=(3, 3)) * 0.5          # any matrix
    maps = [po.src_map(d, F) for F in mats]
    mats[-1] = np.nan                                # no voxel lands on the grid
    maps[-1] = np.full(n, -1, np.int64)
    R = len(maps)
    gs = rng.normal(size=R).astype(np.float32)
    gs[::5] = 0
    md = dev.to_dev(mats)
    t, q, g = dev.to_dev(ET), dev.to_dev(EQ), dev.to_dev(gs)
    s = net.score(t, q, md).cpu().numpy()
    gT = torch.full((K, d, d, d), 0.5, device=dev.device)      # the gradients accumulate
    gQ = torch.full((K, d, d, d), -0.25, device=dev.device)
    net.score_backward(t, q, md, g, gT, gQ)
    t64, q64 = ET.reshape(K, n).astype(np.float64), EQ.reshape(K, n).astype(np.float64)
    eps = 2.0 ** -24
    bound = po.score_fwd(np.abs(t64), np.abs(q64), maps) * (K * n + 64) * eps
    assert np.all(np.abs(s - po.score_fwd(t64, q64, maps)) <= bound + 1e-30)
    oT, oQ = po.score_bwd(t64, q64, maps, gs.astype(np.float64))
    aT, aQ = po.score_bwd(np.abs(t64), np.abs(q64), maps, np.abs(gs.astype(np.float64)))
    for got, ref, mag, base in ((gT, oT, aT, 0.5), (gQ, oQ, aQ, -0.25)):
        err = np.abs(got.cpu().numpy().reshape(K, n) - (ref + base))
        assert np.all(err <= (mag + abs(base)) * (4 * R + 256) * eps), float((err / (mag + abs(base))).max())


@pytest.mark.parametrize("d,nrot", [(1, 3), (2, 5), (7, 16), (10, 33), (15, 700), (18, 700)])
def test_score8_sums_are_the_general_kernels(dev, d, nrot):
    """A ninth channel of zeros takes the general kernel and adds nothing: the same bits, infinities in features
    that no rotation reaches included."""
    from vesper_python_gb300 import proposal as P
    from vesper_python_gb300 import vesper as vg
    net = P.ProposalNet(dev, seed=1)
    g = torch.Generator().manual_seed(d)
    t, q = (torch.randn((8, d, d, d), generator=g).to(dev.device) for _ in range(2))
    angles = orc.calc_angle_comb(10.0)
    mats = dev.to_dev(vg.rot_matrices(angles[::max(1, len(angles) // nrot)][:nrot]))
    for bad in (False, True):
        if bad:
            t[3, 0, 0, 0] = float("inf")
            q[3, -1, -1, -1] = float("inf")
        ninth = [torch.cat([a, torch.zeros_like(a[:1])]).contiguous() for a in (t, q)]
        a, b = net.score(t, q, mats), net.score(*ninth, mats)
        assert torch.equal(a.view(torch.int32)[~a.isnan()], b.view(torch.int32)[~b.isnan()])
        assert torch.equal(a.isnan(), b.isnan())
