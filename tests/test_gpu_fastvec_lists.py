"""fastVEC's listed stages at the edges of their tiles: source rows that are not a multiple of
four, unaligned sources, grids whose z does not fill a tile, planes and rows without a value
between others, a map with one value, one without any, windows that end outside the source, and
long source rows.  Against the float64 form of the same sums (test_fastvec_float_float.py's bar:
1e-12 relative for densities, 2e-6 for vectors)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _direct(src, sw, so, d, dw, do, g):
    """The separable sums in float64 over dense per-axis weights."""
    half = 2.0 * (g / sw)
    fsiv = 1.0 / (0.5 * (g / sw)) ** 2
    w, pos = [], []
    for a in range(3):
        p = (np.arange(d) * dw + do[a] - so[a]) / sw
        e = np.arange(src.shape[a])
        lo = np.maximum(np.trunc(p - half), 0)
        hi = np.minimum(np.trunc(p + half + 1.0), src.shape[a])
        w.append(np.where((e >= lo[:, None]) & (e < hi[:, None]), np.exp(-1.5 * (e - p[:, None]) ** 2 * fsiv), 0.0))
        pos.append(p)
    m = [a * np.arange(a.shape[1]) for a in w]
    s = src.astype(np.float64)

    def total(a, b, c):
        return np.einsum("ix,jy,kz,xyz->ijk", a, b, c, s, optimize=True)

    dens, mean = total(*w), np.stack([total(m[0], w[1], w[2]), total(w[0], m[1], w[2]), total(w[0], w[1], m[2])], -1)
    at = [np.where((p >= 0) & (p < n), p, -1).astype(int) for p, n in zip(pos, src.shape)]
    ok = (at[0] >= 0)[:, None, None] & (at[1] >= 0)[None, :, None] & (at[2] >= 0)
    i = [np.maximum(a, 0) for a in at]
    ok &= src[np.ix_(*i)] != 0
    some = ok & (dens != 0)
    v = mean / np.where(some, dens, 1)[..., None] - np.stack(np.meshgrid(*pos, indexing="ij"), -1)
    n = np.linalg.norm(v, axis=-1, keepdims=True)
    return np.where(ok, dens, 0), np.where(some[..., None], v / np.where(n == 0, 1, n), 0)


@pytest.mark.parametrize("shape,d,dw,shift,g", [((24, 20, 28), 9, 3.0, 0.0, 6.0), ((21, 19, 23), 33, 1.0, -4.0, 5.0),
                                                ((16, 16, 16), 66, 0.4, -5.0, 4.0), ((30, 31, 33), 13, 2.7, -2.5, 16.0),
                                                ((5, 6, 1500), 12, 2.0, 0.0, 8.0), ((12, 12, 12), 1, 4.0, 4.0, 8.0)])
def test_fastvec_list_edges(dev, shape, d, dw, shift, g):
    from vesper_python_gb300 import vesper as vg
    rng = np.random.default_rng(sum(shape) + d)
    base = rng.uniform(0.1, 2.0, shape).astype(np.float32)
    base[rng.random(shape) < 0.5] = 0
    maps = [base, base.copy(), np.zeros(shape, np.float32), np.zeros(shape, np.float32)]
    maps[1][shape[0] // 3:shape[0] // 2] = 0        # planes and rows without a value
    maps[1][:, shape[1] // 2:shape[1] // 2 + 3] = 0
    maps[2][shape[0] // 2, shape[1] // 2, shape[2] // 2] = 0.75
    for src in maps:
        for off in (0, 1):                          # a source that is not 16-byte aligned
            flat = torch.zeros(src.size + 4, dtype=torch.float32, device=dev.device)
            t = flat[off:off + src.size].reshape(shape)
            t.copy_(torch.from_numpy(src))
            data, data32, vec = vg.fastvec_device(t, 1.0, [0.0, 0.0, 0.0], d, dw, [shift] * 3, g, dev=dev)
            rd, rv = _direct(src, 1.0, [0.0] * 3, d, dw, [shift] * 3, g)
            data, vec = data.cpu().numpy(), vec.cpu().numpy()
            assert np.array_equal(data != 0, rd != 0)
            assert np.all(np.abs(data - rd) <= 1e-12 * np.abs(rd))
            assert np.max(np.abs(vec - rv), initial=0) < 2e-6
            assert np.array_equal(data32.cpu().numpy(), data.astype(np.float32))
