"""The batch that batch = 0 takes, by the launches that vesper_search_profile counts: the library's default
where the workspace holds it, else the largest that the workspace holds; and search_device where the
device has no room for the default."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _launches(dev, mode, d, n, nbytes):
    """pass_launches of a search of n rotations in ``nbytes`` of scratch."""
    from vesper_python_gb300 import _native
    from vesper_python_gb300 import vesper as vg
    code, prob = vg.MODE_CODES[mode], mode == "prob"
    data, vec = torch.rand((d, d, d), dtype=torch.float64, device=dev.device), torch.rand((d, d, d, 3), device=dev.device)
    probs = torch.rand((4, d, d, d), device=dev.device) if prob else None
    spec = vg.target_spectra_device(data, vec, mode, 0.0, probs=probs, dev=dev)
    mats = dev.to_dev(vg.rot_matrices(vg.calc_angle_comb(30.0)[:n]))
    ws = torch.empty(nbytes, dtype=torch.uint8, device=dev.device)
    sc = torch.empty((n, 2 if prob else 1), device=dev.device)
    ln = torch.empty((n, 2 if prob else 1), dtype=torch.int32, device=dev.device)
    ms, nl = (ctypes.c_float * 4)(), (ctypes.c_int * 4)()
    p = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else None)  # noqa: E731
    _native.check(dev.lib.vesper_search_profile(p(spec), p(data), p(vec), p(probs), d, code, 0.0, p(mats), n, None, p(sc),
                                                p(ln), 0, p(ws), nbytes, dev.stream, ms, nl, None))
    return list(nl)


@pytest.mark.parametrize("mode,d", [("VecProduct", 48), ("prob", 48), ("Laplacian", 36), ("CC", 36), ("CC", 21),
                                    ("VecProduct", 16)])
@pytest.mark.parametrize("room", ["full", "least"])
def test_profile_counts_the_launches_made(dev, mode, d, room):
    from vesper_python_gb300 import _native
    from vesper_python_gb300 import vesper as vg
    n, code, prob = 500, vg.MODE_CODES[mode], mode == "prob"
    per = (9 if prob else 4 if mode == "VecProduct" else 2) * d * d * (d // 2 + 1) * 8
    base = min((64 << 20) // per, 2048)
    nbytes = _native.size_query("vesper_search_workspace_size", d, code, 0 if room == "full" else base, n)
    if vg.search_plan(d, mode, 0, 1, None, dev)[0] == 2:
        want = [1, 0, 0, 1]                                     # the fused kernel
    else:
        total = per + (d ** 3 * 8 if mode == "Laplacian" else 0)
        full = max(base, min(n, 256, (1 << 30) // total))
        steps = -(-n // (full if room == "full" else base))
        want = [steps, steps, steps, 1]
    assert _launches(dev, mode, d, n, nbytes) == want


@pytest.mark.parametrize("mode,d,batch", [("VecProduct", 48, 101), ("prob", 48, 57), ("Laplacian", 36, 255), ("CC", 75, 26)])
def test_default_batch_is_the_largest_that_fits(dev, mode, d, batch):
    from vesper_python_gb300 import _native
    from vesper_python_gb300 import vesper as vg
    n = 4 * batch
    nbytes = _native.size_query("vesper_search_workspace_size", d, vg.MODE_CODES[mode], batch, n)
    assert _launches(dev, mode, d, n, nbytes) == [4, 4, 4, 1]
    assert _launches(dev, mode, d, n, nbytes - 1) == [5, 5, 5, 1]


@pytest.mark.parametrize("mode,d", [("VecProduct", 48), ("prob", 36), ("Laplacian", 36), ("VecProduct", 16)])
def test_search_device_with_little_memory(dev, monkeypatch, mode, d):
    """The default batch's scratch is refused; a smaller batch gives the same bits.  A batch that the caller
    names is not replaced."""
    from vesper_python_gb300 import _native
    from vesper_python_gb300 import vesper as vg
    g = torch.Generator().manual_seed(d)
    data = torch.rand((d, d, d), dtype=torch.float64, generator=g).to(dev.device)
    vec, probs = torch.randn((d, d, d, 3), generator=g).to(dev.device), torch.rand((4, d, d, d), generator=g).to(dev.device)
    kw = {"probs": probs} if mode == "prob" else {}
    spec = vg.target_spectra_device(data, vec, mode, 0.0, dev=dev, **kw)
    mats = dev.to_dev(vg.rot_matrices(vg.calc_angle_comb(30.0)[::5]))
    n, code = int(mats.shape[0]), vg.MODE_CODES[mode]
    ref = vg.search_device(spec, data, vec, mode, 0.0, mats, dev=dev, **kw)
    for batch in (50, 9, 1):
        room = _native.size_query("vesper_search_workspace_size", d, code, batch, n)

        def workspace(key, nbytes):
            if key[0] == "search" and nbytes > room:
                raise torch.cuda.OutOfMemoryError("no room")
            return torch.empty(nbytes, dtype=torch.uint8, device=dev.device)

        monkeypatch.setattr(dev, "workspace", workspace)
        got = vg.search_device(spec, data, vec, mode, 0.0, mats, dev=dev, **kw)
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
        with pytest.raises(torch.cuda.OutOfMemoryError):
            vg.search_device(spec, data, vec, mode, 0.0, mats, batch=batch + 1, dev=dev, **kw)
