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
