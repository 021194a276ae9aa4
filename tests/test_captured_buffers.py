"""What a captured graph reads and writes stays allocated as long as the graph can be replayed: the
weights of the proposal network, the scratch of Device.workspace (without a GPU the allocations are host tensors and the capture is a flag)."""
import contextlib
import types

import numpy as np
import pytest
import torch

from vesper_python_gb300 import align
from vesper_python_gb300 import vesper as vg


def _device(monkeypatch):
    dev = object.__new__(vg.Device)
    dev.device, dev.index, dev._ws = torch.device("cpu"), 0, {}
    dev._captured, dev._kept = set(), []
    state = {"stream": 1, "capturing": False}
    monkeypatch.setattr(vg, "_raw_stream", lambda index: state["stream"])
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state["capturing"])
    return dev, state


def _alive(dev, address, size):
    """Whether a tensor of ``dev`` still holds [address, address + size)."""
    return any(t.data_ptr() <= address and address + size <= t.data_ptr() + t.numel()
               for v in vars(dev).values() if isinstance(v, (dict, list))
               for t in (v.values() if isinstance(v, dict) else v))


def test_scratch_of_a_capture_outlives_a_larger_call(monkeypatch):
    dev, state = _device(monkeypatch)
    key = ("search", 28, 0, 0)
    first = dev.workspace(key, 1000).data_ptr()         # the warm-up before the capture
    state["capturing"] = True
    assert dev.workspace(key, 1000).data_ptr() == first     # what the graph replays with
    state["capturing"] = False
    for nbytes in (900, 1500, 5000, 70000):
        assert dev.workspace(key, nbytes).numel() >= nbytes
        assert _alive(dev, first, 1000), nbytes
    # a second capture's buffer, on a stream of its own too
    state["capturing"] = True
    second = dev.workspace(key, 70000).data_ptr()
    state["stream"] = 2
    third = dev.workspace(key, 300).data_ptr()
    state["capturing"] = False
    dev.workspace(key, 400)
    state["stream"] = 1
    dev.workspace(key, 200000)
    assert _alive(dev, first, 1000) and _alive(dev, second, 70000) and _alive(dev, third, 300)


def test_scratch_without_a_capture_is_given_back_and_kept_scratch_is_bounded(monkeypatch):
    dev, state = _device(monkeypatch)
    key = ("search", 28, 0, 0)
    for nbytes in range(1000, 9000, 1000):
        buf = dev.workspace(key, nbytes)
        assert sum(t.numel() for t in dev._ws.values()) + sum(t.numel() for t in dev._kept) == nbytes
    state["capturing"] = True
    for nbytes in range(10000, 200000, 777):      # every call captured, each needs a little more
        buf = dev.workspace(key, nbytes)
        assert sum(t.numel() for t in dev._kept) <= buf.numel() < 2 * nbytes + 8000


def test_aligners_do_not_share_scratch(monkeypatch):
    """Graphs of two aligners are captured on the same capture stream and may be replayed side by side."""
    dev, state = _device(monkeypatch)
    dev.lib = None
    state["capturing"] = True
    users = [align.Aligner(dev), align.Aligner(dev)]
    spans = []
    for d in [dev] + [al.dev for al in users]:
        buf = d.workspace(("search", 28, 0, 0), 4096)
        assert buf is d.workspace(("search", 28, 0, 0), 4000)
        spans.append((buf.data_ptr(), buf.data_ptr() + buf.numel()))
    spans.sort()
    assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))
    assert all(al.dev.device == dev.device and al.dev.lib is dev.lib for al in users)


def test_captured_stage_keeps_the_networks_weights(monkeypatch):
    """Other weights, of the same network or of one that takes its place, are another signature, and the weights
    that a captured stage reads are not given back."""
    monkeypatch.setattr(torch.cuda, "CUDAGraph", lambda: types.SimpleNamespace(replay=lambda: None))
    monkeypatch.setattr(torch.cuda, "graph", lambda g: contextlib.nullcontext())
    dev, _ = _device(monkeypatch)
    dev.lib = None
    al = align.Aligner(dev)
    monkeypatch.setattr(al, "_global_stage", lambda P, p, mats, nang: (None, None))
    m = torch.zeros(4, 4, 4)
    st = align._Pair(m, m, 1.0, 1.0, np.zeros(3), np.zeros(3))
    st.dim, st.no1, st.no2, st.o1, st.o2 = 8, np.zeros(3), np.zeros(3), np.zeros(3), np.zeros(3)
    for k in al._STAGE_FIELDS:
        if k != "launches":
            setattr(st, k, None)

    def weights():
        return [torch.zeros(300), torch.zeros(500)]

    net = types.SimpleNamespace(Wbf=weights(), b=weights())
    p = align.AlignParams(proposal=net)
    used = set()
    for captures in (1, 2, 3):
        at = {t.data_ptr() for t in net.Wbf + net.b}
        assert not (at & used)           # the ones before are still held
        used |= at
        for _ in range(2):
            al._global_stage_graph([st], p, m, 8)
            assert al.graph_captures == captures
        if captures == 1:
            del net.Wbf, net.b           # load_state_dict
            net.Wbf, net.b = weights(), weights()
        else:
            p.proposal = net = None      # another network
            p.proposal = net = types.SimpleNamespace(Wbf=weights(), b=weights())


@pytest.mark.gpu
def test_replay_after_a_larger_eager_call(dev):
    """A graph with 270 refinement slots per pair, then eager calls with 1,080 on the same side streams, then
    tensors over whatever was given back: the replay gives its results again and the tensors keep their values."""
    from vesper_python_gb300 import synth
    items = []
    for i in range(3):
        pair = synth.make_pair(60 + i, 64, 40, 18.0)
        items.append((dev.to_dev(pair.map1), dev.to_dev(pair.map2), 1.0, 1.0, pair.orig1, pair.orig2))
    al = align.Aligner(dev)
    few = align.AlignParams(t=0.1, T=0.1, s=3.0, A=30.0, N=10)
    many = align.AlignParams(t=0.1, T=0.1, s=3.0, A=30.0, N=40)
    ref = al.align_many(items, few, graph=True)
    for _ in range(2):
        al.align_many(items, many)
        fill = [torch.full((n,), 77, dtype=torch.uint8, device=dev.device) for n in (1 << 12, 1 << 16, 1 << 20, 1 << 24)
                for _ in range(8)]
        again = al.align_many(items, few, graph=True)
        assert al.graph_captures == 2
        for a, b in zip(ref, again):
            assert (a.dim, a.std, a.ave, a.top) == (b.dim, b.std, b.ave, b.top)
            assert [(m.angle, m.vec_score, m.vec_trans, m.dot_score, m.cc) for m in a.models] == \
                [(m.angle, m.vec_score, m.vec_trans, m.dot_score, m.cc) for m in b.models]
        assert all(bool((f == 77).all()) for f in fill)
