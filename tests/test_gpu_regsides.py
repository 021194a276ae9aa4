"""The register passes of every compiled side against the radix-stage passes.

Where a side and mode repeat the radix stages' arithmetic (all but the ones
listed in PFA, whose line DFTs split coprime factors without twiddles), scores
and translations are equal bit for bit: the two families run the same float32
operations in the same order.  Where they do not, both are float32 FFTs of
length d^3 and agree to SCORE_RTOL of the largest score, as in
test_gpu_parity.py.  Rotation counts and batches leave remainders in every pass."""
import numpy as np
import pytest
import torch

from oracle import vesper_oracle as orc

SCORE_RTOL = 1e-4
PFA = {"VecProduct": (27, 28, 30, 32, 33, 35, 42, 44, 75), "prob": (30, 32, 64), "Overlap": (75,), "CC": (75,),
       "PCC": (75,), "Laplacian": (75,)}


def _sides():
    out = []
    for n in range(25, 101):
        k = n
        for p in (2, 3, 5, 7):
            while k % p == 0:
                k //= p
        if k in (1, 11, 13):
            out.append(n)
    return out


SIDES = _sides()


def test_every_side_from_25_to_100_has_register_passes():
    from vesper_python_gb300 import _native
    import ctypes
    lib = _native.load()
    path, nl = ctypes.c_int(-9), ctypes.c_int(-9)
    opts = (ctypes.c_int * 3)(1, 0, 0)
    for d in SIDES:
        for mode in range(6):
            assert lib.vesper_search_plan(d, mode, 8, 100, opts, ctypes.byref(path), ctypes.byref(nl)) == 0
            assert path.value == 1 and nl.value == 2 + 13 * (5 if mode == 4 else 3), (d, mode)


def _fields(rng, d):
    data = rng.uniform(-0.2, 2.0, size=(d, d, d))
    data[rng.random((d, d, d)) < 0.6] = 0
    vec = rng.normal(size=(d, d, d, 3)).astype(np.float32)   # not zero where the density is: masked by it
    probs = rng.dirichlet([0.5] * 4, size=(d, d, d)).astype(np.float32).transpose(3, 0, 1, 2).copy()
    probs[rng.random(probs.shape) < 0.5] = 0
    return data, vec, probs


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["VecProduct", "Overlap", "CC", "PCC", "Laplacian", "prob"])
def test_register_passes_equal_radix_stage_passes(dev, mode):
    from vesper_python_gb300 import vesper as vg
    for d in SIDES:
        if (mode in ("Overlap", "PCC") and d % 3) or d > 91 and mode not in ("VecProduct", "CC"):
            continue
        rng = np.random.default_rng(d)
        td, tv, tp = (dev.to_dev(a) for a in _fields(rng, d))
        qd, qv, qp = (dev.to_dev(a) for a in _fields(rng, d))
        ave = 0.37
        prob = mode == "prob"
        spec = vg.target_spectra_device(td, tv, mode, ave, probs=tp if prob else None, dev=dev)
        # axis rotations (every voxel on the grid), general ones, and one that is no rotation
        mats = vg.rot_matrices(np.concatenate([orc.calc_angle_comb(90.0)[:7], orc.calc_angle_comb(30.0)[5::131]]))
        mats[-1] = np.nan
        mats = dev.to_dev(mats)
        kw = dict(probs=qp if prob else None, mix=(0.5, 0.7, 0.1, 0.3, 0.2) if prob else None, dev=dev)
        ref = vg.search_device(spec, qd, qv, mode, ave, mats, opts=(0, 0, 0), **kw)
        for batch in (0, 4, 7):
            got = vg.search_device(spec, qd, qv, mode, ave, mats, opts=(1, 0, 0), batch=batch, **kw)
            if d not in PFA[mode]:
                assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1]), (mode, d, batch)
            else:
                assert float((got[0] - ref[0]).abs().max()) <= SCORE_RTOL * float(ref[0].abs().max()), (mode, d)


@pytest.mark.gpu
@pytest.mark.parametrize("mode,d", [("prob", 48), ("VecProduct", 75), ("Laplacian", 50), ("CC", 12)])
def test_default_batch_fits_the_workspace_given(dev, mode, d):
    """batch = 0 takes the library's default where the workspace is as large as it asks for, fewer
    rotations at a time where it is smaller, down to 64 MB of S and U; one smaller still is refused.
    Every batch gives the same bits."""
    import ctypes

    from vesper_python_gb300 import _native
    from vesper_python_gb300 import vesper as vg
    rng = np.random.default_rng(d)
    td, tv, tp = (dev.to_dev(a) for a in _fields(rng, d))
    prob = mode == "prob"
    spec = vg.target_spectra_device(td, tv, mode, 0.0, probs=tp if prob else None, dev=dev)
    mats = dev.to_dev(vg.rot_matrices(orc.calc_angle_comb(30.0)[::11]))
    n, code, ns = int(mats.shape[0]), vg.MODE_CODES[mode], 2 if prob else 1
    per = ((7 + 2) if prob else 4 if mode == "VecProduct" else 2) * d * d * (d // 2 + 1) * 8
    base = min(max(1, (64 << 20) // per), 2048)
    full = _native.size_query("vesper_search_workspace_size", d, code, 0, n)
    least = _native.size_query("vesper_search_workspace_size", d, code, base, n)
    assert least <= full
    ref = vg.search_device(spec, td, tv, mode, 0.0, mats, probs=tp if prob else None, batch=3, dev=dev)

    def call(nbytes):
        ws = torch.empty(nbytes, dtype=torch.uint8, device=dev.device)
        sc = torch.full((n, ns), float("nan"), device=dev.device)
        ln = torch.full((n, ns), -1, dtype=torch.int32, device=dev.device)
        p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        rc = dev.lib.vesper_search(p(spec), p(td), p(tv), p(tp), d, code, 0.0, p(mats), n, None, p(sc), p(ln), 0,
                                   p(ws), nbytes, dev.stream)
        torch.cuda.synchronize()
        return rc, sc, ln

    for nbytes in {full, least, (full + least) // 2}:
        rc, sc, ln = call(nbytes)
        assert rc == 0 and torch.equal(sc, ref[0]) and torch.equal(ln, ref[1]), (nbytes, full, least)
    assert call(least - 4096)[0] == 4
