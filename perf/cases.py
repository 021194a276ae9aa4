"""The work that is measured, through the package's public entry points.

Kinds of case, and what in real use each stands for:

  fastvec   one density map -> its Gaussian-weighted vector field (``fastvec_device``), the first
            step of every alignment: map sides 64 to 256, voxel spacings 2 to 7, grid sides 12 to 80
  search    the rotational FFT search of one query against one target (``search_device``, autotuned
            as the drop-in and the aligner call it): 12 to 13 is the grid of the default spacing 7, 28
            to 32 of spacing 3, 36 to 50 of large maps at spacing 4, 75 of spacing 2; 1,008 rotations
            are the default 30-degree grid, 1,232 the subset that the rotation proposal hands over;
            modes VecProduct, CC, PCC and Laplacian (Overlap runs the kernels of CC on 0/1 values;
            its scores are whole counts, and rounding alone picks among its tied translations)
  prob      the mixed pass of the probability-map search: 7 channels, 3 scores per rotation
            (``search_device`` with ``mix``, as ``search_map_fft_prob`` calls it)
  propose   the rotation proposal's scores of the whole 10-degree grid for several pairs of one
            pooled side, committed weights (``ProposalNet.rotation_scores_many``)
  train     the proposal's training step of one pair: forward, loss and every gradient
            (``ProposalNet.loss_and_grad``)
  align     whole alignments (``Aligner.align_many``): new maps each time, so launched eagerly; a
            batch of 16 pairs with the rotation proposal (serving), one large pair exhaustively

Inputs are blob maps and the smooth unit-vector fields that fastVEC makes of such maps: a target, and a
query that is the target's rotated, shifted inner half with voxels of its own masked.
"""
import math
import os

import numpy as np
import torch

# each process times launch shapes for the kernels that it runs, instead of taking another's from a file
os.environ.setdefault("VESPER_AUTOTUNE_CACHE", "")

from vesper_python_gb300 import proposal as vp  # noqa: E402
from vesper_python_gb300 import vesper as vg  # noqa: E402
from vesper_python_gb300 import align as va  # noqa: E402

GRID_STEP = 10.0          # the fine angle grid, 24,624 rotations
BANDWIDTH = 16.0          # fastVEC's default bandwidth (A)
THRESHOLD = 0.1
MODES = ("VecProduct", "CC", "PCC", "Laplacian")


def listed():
    return [
        # one 128^3 map at spacing 3, and the largest maps of an uneven batch at spacing 4
        {"name": "fastvec_128_s3", "kind": "fastvec", "side": 128, "d": 28, "s": 3.0},
        {"name": "fastvec_256_s4", "kind": "fastvec", "side": 256, "d": 42, "s": 4.0},
        # the command line's defaults (spacing 7, 30 degrees): the smallest search
        {"name": "search_vec_13", "kind": "search", "mode": "VecProduct", "d": 13, "nrot": 1008, "step": 30.0},
        # the exact search of a proposed subset at spacing 3
        {"name": "search_vec_30", "kind": "search", "mode": "VecProduct", "d": 30, "nrot": 1232, "step": 10.0},
        # a side between the tuned ones
        {"name": "search_vec_48", "kind": "search", "mode": "VecProduct", "d": 48, "nrot": 1008, "step": 30.0},
        # spacing 2 on a 200^3 map, vector and density modes
        {"name": "search_vec_75", "kind": "search", "mode": "VecProduct", "d": 75, "nrot": 1008, "step": 30.0},
        {"name": "search_cc_75", "kind": "search", "mode": "CC", "d": 75, "nrot": 1008, "step": 30.0},
        # probability maps on grids padded to 64^3
        {"name": "search_prob_64", "kind": "prob", "d": 64, "nrot": 1008, "step": 30.0},
        # inference and training of the rotation proposal
        {"name": "propose_8x15", "kind": "propose", "pairs": 8, "d": 15},
        {"name": "train_15", "kind": "train", "d": 15},
        # whole alignments
        {"name": "align_16_proposal", "kind": "align", "pairs": 16, "side": 128, "radius": 40.0, "s": 3.0, "A": 10.0,
         "proposal": True},
        {"name": "align_200_exhaustive", "kind": "align", "pairs": 1, "side": 200, "radius": 70.0, "s": 2.0,
         "A": 10.0, "proposal": False},
    ]


def _fast_sides(lo, hi):
    """Grid sides in [lo, hi] that the sizing rule produces: 2^a 3^b 5^c 7^d (11 or 13 once)."""
    out = []
    for n in range(lo, hi + 1):
        k = n
        for p in (2, 3, 5, 7):
            while k % p == 0:
                k //= p
        if k in (1, 11, 13):
            out.append(n)
    return out


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(_fast_sides(lo, hi), key=lambda n: abs(math.log(n / want)))


def draw(rng):
    kind = rng.choice(("fastvec", "search", "search", "search", "prob", "propose", "train", "align"))
    if kind == "fastvec":
        side = _log(rng, 64, 256)
        s = round(rng.uniform(2.0, 7.0), 2)
        d = max(8, int(2 * (0.33 * side + 4) / s))
        return {"kind": kind, "side": side, "s": s, "d": min(_fast_sides(d, d + 8))}
    if kind == "search":
        mode = rng.choice(("VecProduct", "VecProduct") + MODES)
        return {"kind": kind, "mode": mode, "d": _side(rng, 8, 96), "nrot": _log(rng, 64, 1232), "step": GRID_STEP}
    if kind == "prob":
        return {"kind": kind, "d": _side(rng, 12, 72), "nrot": _log(rng, 64, 1008), "step": GRID_STEP}
    if kind == "propose":
        return {"kind": kind, "pairs": rng.randint(1, 16), "d": rng.randint(8, 20)}
    if kind == "train":
        return {"kind": kind, "d": rng.randint(8, 18)}
    if rng.random() < 0.5:
        return {"kind": kind, "pairs": rng.randint(1, 12), "side": 128, "radius": round(rng.uniform(34.0, 46.0), 1),
                "s": 3.0, "A": GRID_STEP, "proposal": True}
    side = 2 * _log(rng, 32, 80)
    return {"kind": kind, "pairs": rng.randint(1, 4), "side": side, "radius": round(0.32 * side, 1),
            "s": rng.choice((4.0, 5.0, 7.0)), "A": rng.choice((15.0, 30.0)), "proposal": False}


# ---- what a program keeps for all its calls: device, angle grids, aligner, network -------------------

_KEPT = {}


def _kept(key, make):
    if key not in _KEPT:
        _KEPT[key] = make()
    return _KEPT[key]


def _rotations(step):
    """float32 [n][3][3]: the rotation matrices of the angle grid (ZYX Euler angles; x and y over the circle,
    z over half of it, z slowest), rows and columns reversed, as the gather takes them."""
    xy = np.arange(0.0, 360.0, step)
    z = np.arange(0.0, 180.0 + 1e-9, step)
    a = np.radians(np.array(np.meshgrid(xy, xy, z)).T.reshape(-1, 3))
    (ca, cb, cc), (sa, sb, sc) = np.cos(a).T, np.sin(a).T
    m = np.array([[ca * cb, ca * sb * sc - sa * cc, ca * sb * cc + sa * sc],
                  [sa * cb, sa * sb * sc + ca * cc, sa * sb * cc - ca * sc],
                  [-sb, cb * sc, cb * cc]]).transpose(2, 0, 1)
    m[np.abs(m) < 1e-15] = 0.0
    return np.ascontiguousarray(m[:, ::-1, ::-1].astype(np.float32))


def _grid(step):
    return _kept(("grid", step), lambda: torch.from_numpy(_rotations(step)).cuda())


def _some_rotations(case, seed):
    """The whole grid, or ``nrot`` of its rotations in grid order."""
    mats = _grid(case["step"])
    if case["nrot"] >= mats.shape[0]:
        return mats
    g = torch.Generator().manual_seed(seed + 5)
    pick = torch.randperm(mats.shape[0], generator=g)[:case["nrot"]].sort().values
    return mats[pick.cuda()].contiguous()


# ---- inputs ------------------------------------------------------------------------------------------

def _random_rotation(g):
    q, r = np.linalg.qr(torch.randn(3, 3, dtype=torch.float64, generator=g).numpy())
    q = q * np.sign(np.diag(r))
    return torch.from_numpy(q * np.linalg.det(q)).cuda()


def _ball(g, n, radius):
    v = torch.randn(n, 3, dtype=torch.float64, generator=g)
    r = torch.rand(n, 1, dtype=torch.float64, generator=g) ** (1.0 / 3.0)
    return (radius * r * v / v.norm(dim=1, keepdim=True)).cuda()


def _coarse(pos, amp, d, sigma):
    """Density and unit direction field of blobs on a d^3 grid, zero off their narrow mask: what fastVEC
    gives (float64 [d][d][d], float32 [d][d][d][3])."""
    x = torch.arange(d, dtype=torch.float64, device="cuda")
    r = x[None, :, None] - (pos + 0.5 * d)[:, None, :]               # [blob][grid][axis]
    w = torch.exp(-0.5 * (r / sigma) ** 2)
    wx, wy, wz = (w[:, :, a] for a in range(3))
    gx, gy, gz = (-w[:, :, a] * r[:, :, a] for a in range(3))

    def volume(a, b, c):
        return ((a * amp[:, None])[:, :, None] * b[:, None, :]).reshape(len(amp), -1).T.matmul(c).reshape(d, d, d)

    data = volume(wx, wy, wz)
    grad = torch.stack([volume(gx, wy, wz), volume(wx, gy, wz), volume(wx, wy, gz)], -1)
    n = torch.exp(-0.5 * (r / (0.35 * sigma)) ** 2)
    keep = volume(n[:, :, 0], n[:, :, 1], n[:, :, 2]) > 0.1
    vec = grad / (grad.norm(dim=-1, keepdim=True) + 1e-300)
    return torch.where(keep, data, 0.0), torch.where(keep[..., None], vec, 0.0).to(torch.float32).contiguous()


def _pair_fields(seed, d):
    """(target data, vec), (query data, vec)."""
    g = torch.Generator().manual_seed(seed)
    pos = _ball(g, 150, 0.42 * d)
    amp = (0.5 + torch.rand(150, dtype=torch.float64, generator=g)).cuda()
    target = _coarse(pos, amp, d, 0.08 * d)
    m, shift = _random_rotation(g), (0.1 * d * (torch.rand(3, dtype=torch.float64, generator=g) - 0.5)).cuda()
    inner = pos.norm(dim=1) < 0.3 * d
    return target, _coarse(pos[inner] @ m.T + shift, amp[inner], d, 0.08 * d)


def _probabilities(seed, data):
    """float32 [4][d][d][d]: Dirichlet(0.5) in the mask of ``data``, zero off it."""
    g = torch.Generator().manual_seed(seed)
    p = torch.randn((4,) + tuple(data.shape), generator=g).cuda() ** 2
    return torch.where(data != 0, p / p.sum(0, keepdim=True), 0.0).contiguous()


def _blob_map(g, side, radius):
    n = max(8, int(round(400 * (radius / 40.0) ** 3)))
    pos = _ball(g, n, radius) + 0.5 * side
    amp = (0.5 + torch.rand(n, generator=g)).cuda()
    x = torch.arange(side, dtype=torch.float64, device="cuda")
    w = torch.exp(-0.5 * ((x[None, :, None] - pos[:, None, :]) / 1.5) ** 2).float()
    m = ((w[:, :, 0] * amp[:, None])[:, :, None] * w[:, None, :, 1]).reshape(n, -1).T.matmul(w[:, :, 2])
    return m.reshape(side, side, side)


def _noise(seed, shape):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return 0.01 * torch.randn(shape, generator=g, device="cuda")


def _map_pair(seed, side, radius):
    """A map, the rotated and shifted crop of its inner half, and their origins."""
    g = torch.Generator().manual_seed(seed)
    clean = _blob_map(g, side, radius)
    m, shift = _random_rotation(g), (10 * torch.rand(3, dtype=torch.float64, generator=g) - 5).cuda()
    half = side // 2
    ax = torch.arange(half, dtype=torch.float64, device="cuda") - 0.5 * half
    at = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1) @ m.T + 0.5 * side + shift
    i = at.round().long()
    ok = ((i >= 0) & (i < side)).all(-1)
    i = i.clamp(0, side - 1)
    crop = torch.where(ok, clean[i[..., 0], i[..., 1], i[..., 2]], 0.0)
    o2 = np.full(3, 0.5 * (side - half))
    return (clean + _noise(2 * seed, clean.shape)).contiguous(), (crop + _noise(2 * seed + 1, crop.shape)).contiguous(), o2


def _pooled_fields(seed, pairs, d):
    """Network inputs [2 pairs][4][d][d][d]: 2x2x2 means of (vx, vy, vz, mask), target then query of each pair."""
    out = []
    for i in range(pairs):
        for data, vec in _pair_fields(seed + 101 * i, 2 * d):
            f = torch.cat([vec.permute(3, 0, 1, 2), (data != 0).float()[None]])
            out.append(torch.nn.functional.avg_pool3d(f[None], 2)[0])
    return torch.stack(out).contiguous()


def _fastvec_inputs(case, seed):
    side, d, s = case["side"], case["d"], case["s"]
    m = _blob_map(torch.Generator().manual_seed(seed), side, 0.3125 * side) + _noise(seed, (side,) * 3)
    m = torch.where(m < THRESHOLD, 0.0, m).contiguous()
    return m, np.zeros(3), np.full(3, 0.5 * side - 0.5 * d * s)


def _labels(seed, n):
    """The training target of one pair: softmax of twice the standardised scores of every rotation."""
    z = torch.randn(n, generator=torch.Generator().manual_seed(seed + 9))
    z[int(seed) % n] += 8.0
    return torch.softmax(2.0 * (z - z.mean()) / z.std(), 0).cuda().contiguous()


def _ave(data):
    return float(data[data > 0].mean())


def _mix(data):
    """The z-score constants of the first pass: about what its best scores' mean and spread are."""
    n = float((data != 0).sum())
    return (0.5, 0.05 * n, 0.3 * n, 0.02 * n, 0.2 * n)


def prepare(case, seed):
    kind = case["kind"]
    dev = _kept("device", vg.default_device)
    if kind == "fastvec":
        src, o1, o2 = _fastvec_inputs(case, seed)
        return {"case": case, "src": src, "o1": o1, "o2": o2}
    if kind in ("search", "prob"):
        (td, tv), (qd, qv) = _pair_fields(seed, case["d"])
        st = {"case": case, "dev": dev, "qd": qd, "qv": qv, "mats": _some_rotations(case, seed), "ave": _ave(td)}
        if kind == "prob":
            st["qp"], st["mix"] = _probabilities(seed + 2, qd), _mix(qd)
            st["spec"] = vg.target_spectra_device(td, tv, "prob", 0.0, probs=_probabilities(seed + 1, td), dev=dev)
        else:
            st["spec"] = vg.target_spectra_device(td, tv, case["mode"], st["ave"], dev=dev)
        return st
    if kind == "propose":
        return {"case": case, "net": _kept("net", lambda: vp.load_weights(dev)[0]), "mats": _grid(GRID_STEP),
                "fields": _pooled_fields(seed, case["pairs"], case["d"])}
    if kind == "train":
        f = _pooled_fields(seed, 1, case["d"])
        mats = _grid(GRID_STEP)
        return {"case": case, "net": vp.load_weights(dev)[0], "mats": mats, "fT": f[0], "fQ": f[1],
                "q": _labels(seed, int(mats.shape[0]))}
    items = []
    for i in range(case["pairs"]):
        m1, m2, o2 = _map_pair(seed * 64 + i, case["side"], case["radius"])
        items.append((m1, m2, 1.0, 1.0, np.zeros(3), o2))
    p = va.AlignParams(t=THRESHOLD, T=THRESHOLD, g=BANDWIDTH, s=case["s"], A=case["A"], N=10, mode="VecProduct",
                       proposal=_kept("net", lambda: vp.load_weights(dev)[0]) if case["proposal"] else None)
    return {"case": case, "aligner": _kept("aligner", lambda: va.Aligner(dev)), "items": items, "params": p}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "fastvec":
        data, data32, vec = vg.fastvec_device(state["src"], 1.0, state["o1"], case["d"], case["s"], state["o2"],
                                              BANDWIDTH)
        return {"data": data, "data32": data32, "vec": vec}
    if kind == "search":
        scores, lin = vg.search_device(state["spec"], state["qd"], state["qv"], case["mode"], state["ave"],
                                       state["mats"], dev=state["dev"], tuned=True)
        return {"scores": scores, "lin": lin}
    if kind == "prob":
        scores, lin = vg.search_device(state["spec"], state["qd"], state["qv"], "prob", 0.0, state["mats"],
                                       probs=state["qp"], mix=state["mix"], dev=state["dev"])
        return {"scores": scores, "lin": lin}
    if kind == "propose":
        return {"scores": state["net"].rotation_scores_many(state["fields"], state["mats"])}
    if kind == "train":
        net = state["net"]
        net.zero_grad()
        loss = net.loss_and_grad(state["fT"], state["fQ"], state["mats"], state["q"], 0.5)
        return {"loss": loss, "gW": list(net.gW), "gb": list(net.gb)}
    results = [_alignment(r) for r in state["aligner"].align_many(state["items"], state["params"])]
    return {k: np.stack([r[k] for r in results]) for k in results[0]}


def _alignment(r):
    """One alignment's result as arrays; the search's scores are single precision, the models' are double."""
    return {"dim": np.array([r.dim]), "grid": np.array([r.std, r.ave], np.float32),
            "top_angles": np.array([t[0] for t in r.top], np.float32),
            "top_scores": np.array([t[1] for t in r.top], np.float32),
            "top_trans": np.array([[int(v) for v in t[2]] for t in r.top], np.int32),
            "angles": np.array([m.angle for m in r.models], np.float32),
            "scores": np.array([m.vec_score for m in r.models], np.float32),
            "trans": np.array([[int(v) for v in m.vec_trans] for m in r.models], np.int32),
            "models": np.array([[m.overlap, m.cc, m.pcc, m.dot_score] for m in r.models], np.float64)}


def work(case):
    """Bytes: every input read once, every output written once.  Flops: the transforms (2.5 N log2 N of a real
    3-D one), the products and sums that the path cannot do without."""
    kind = case["kind"]
    if kind == "fastvec":
        side, d, wb = case["side"], case["d"], min(case["side"], 4 * BANDWIDTH + 3)
        return {"bytes": 4.0 * side ** 3 + 24.0 * d ** 3,
                "flops": 4.0 * side * side * d * wb + 6.0 * side * d * d * wb + 8.0 * d ** 3 * wb}
    if kind in ("search", "prob"):
        c, g = (7, 2) if kind == "prob" else (3 if case["mode"] == "VecProduct" else 1, 1)
        return _search_work(case["d"], case["nrot"], c, g)
    rot = 24624
    if kind in ("propose", "train"):
        n = case["d"] ** 3
        maps = 2 * case.get("pairs", 1)
        encode = maps * 2.0 * 27 * (4 * 32 + 32 * 32 + 32 * 32 + 32 * 8) * n
        score = maps / 2 * 2.0 * rot * n * 8
        wbytes = 4.0 * 27 * (4 * 32 + 32 * 32 + 32 * 32 + 32 * 8)
        if kind == "train":   # two products of the same size backwards, and the gradients written
            return {"bytes": 16.0 * maps * n + 2 * wbytes + 40.0 * rot, "flops": 3 * (encode + score)}
        return {"bytes": 16.0 * maps * n + wbytes / 2 + 4.0 * rot * maps / 2, "flops": encode + score}
    d = int(2 * (case["radius"] + 4) / case["s"])
    full = int((360 / case["A"]) ** 2 * (180 / case["A"] + 1))
    nrot = (math.ceil(0.05 * full) if case["proposal"] else full) + 150
    s = _search_work(d, nrot, 3, 1)
    f1 = work({"kind": "fastvec", "side": case["side"], "d": d})
    f2 = work({"kind": "fastvec", "side": case["side"] // 2, "d": d})
    more = work({"kind": "propose", "pairs": 1, "d": (d + 1) // 2}) if case["proposal"] else {"flops": 0.0}
    return {"bytes": case["pairs"] * 4.5 * case["side"] ** 3,
            "flops": case["pairs"] * (s["flops"] + f1["flops"] + f2["flops"] + more["flops"])}


def _search_work(d, nrot, c, g):
    n, nh = float(d) ** 3, float(d) * d * (d // 2 + 1)
    return {"bytes": n * (20.0 if c == 3 else 36.0 if c == 7 else 8.0) + 8.0 * c * nh + nrot * (36.0 + 8.0 * (3 if g == 2 else 1)),
            "flops": nrot * ((c + g) * 2.5 * n * math.log2(n) + 8.0 * c * nh + n)}


# ---- the same in 64 bits, in plain torch ---------------------------------------------------------------

def _candidates(d):
    """Source rows that land on each destination index of one axis (the last row wins): two of them at the
    middle of an odd side, none at its end; -1 for none."""
    t = torch.arange(d, device="cuda")
    none = torch.full_like(t, -1)
    if d % 2 == 0:
        return t, none
    m = (d - 1) // 2
    return torch.where(t < m, t, torch.where(t < d - 1, t + 1, none)), torch.where(t == m, t, none)


def _sources(mats, d, ok):
    """int64 [rotations][d^3]: the voxel that the rotated grid takes at each place, -1 for none.  The position is
    a float32 fused multiply-add chain; ``ok`` [d^3] says which voxels count."""
    n, c = mats.shape[0], _candidates(d)
    src = torch.full((n, d, d, d), -1, dtype=torch.int64, device="cuda")
    f = mats.double()[:, :, :, None, None, None]
    for az in (0, 1):
        for ax in (0, 1):
            for ay in (0, 1):
                if d % 2 == 0 and (az or ax or ay):
                    continue
                ix, iy, iz = c[ax][:, None, None], c[ay][None, :, None], c[az][None, None, :]
                there = ((ix >= 0) & (iy >= 0) & (iz >= 0))[None].expand(n, d, d, d)
                h = [(i.double() - 0.5 * d)[None] for i in (ix, iy, iz)]
                at, inside = 0, there
                for a in range(3):
                    o = (h[0] * f[:, a, 0]).float()
                    o = (h[1] * f[:, a, 1] + o.double()).float()
                    o = (h[2] * f[:, a, 2] + o.double()).float() + 0.5 * d
                    inside = inside & (o >= 0) & (o < d)
                    at = at * d + o.clamp(0, d - 1).long()
                inside = inside & ok[at]
                src = torch.where((src < 0) & inside, at, src)
    return src.reshape(n, -1)


def _take(values, src):
    """values [..., d^3] at src [rotations][d^3], zero where there is none: [rotations][..., d^3]."""
    padded = torch.cat([values, torch.zeros_like(values[..., :1])], -1)
    return padded[..., src].movedim(-2, 0)


def _laplacian(v):
    """Six-neighbour Laplacian of [..., d, d, d] where v > 0, zero beyond the edges."""
    acc = -6.0 * v
    for a in (-3, -2, -1):
        z = torch.zeros_like(v.narrow(a, 0, 1))
        acc = acc + torch.cat([v.narrow(a, 1, v.shape[a] - 1), z], a) + torch.cat([z, v.narrow(a, 0, v.shape[a] - 1)], a)
    return torch.where(v > 0, acc, 0.0)


def _exact_search(case, seed):
    d, prob = case["d"], case["kind"] == "prob"
    (td, tv), (qd, qv) = _pair_fields(seed, d)
    mats, ave = _some_rotations(case, seed), _ave(td)
    mode = "prob" if prob else case["mode"]
    n3 = d ** 3

    def density(v):
        if mode == "CC":
            return torch.where(v > 0, v, 0.0)
        if mode == "PCC":
            return torch.where(v > 0, v - ave, 0.0)
        return _laplacian(v)

    if mode in ("VecProduct", "prob"):
        x1 = tv.permute(3, 0, 1, 2).double()
        if prob:
            x1 = torch.cat([x1, _probabilities(seed + 1, td).double()])
            qp = _probabilities(seed + 2, qd).double().reshape(4, n3)
    else:
        x1 = density(td)[None]
    t = torch.fft.rfftn(x1, dim=(1, 2, 3)).conj()
    flat, some = qd.reshape(-1), (qd != 0).reshape(-1)
    out = []
    per = max(1, min(32, int(2e8 / (n3 * 8 * (x1.shape[0] + 6)))))
    for r0 in range(0, mats.shape[0], per):
        f = mats[r0:r0 + per]
        src = _sources(f, d, some)
        if mode in ("VecProduct", "prob"):
            v = _take(qv.reshape(n3, 3).T.double(), src)                                   # [r][3][n]
            x2 = torch.einsum("rkn,rkj->rjn", v, f.double())
            if prob:
                x2 = torch.cat([x2] + [_take(qp[k:k + 1], _sources(f, d, qp[k] != 0)) for k in range(4)], 1)
        else:
            rot = _take(flat[None], src)
            x2 = _laplacian(rot.reshape(-1, d, d, d)).reshape(rot.shape) if mode == "Laplacian" else \
                torch.where((src >= 0)[:, None], density(rot), 0.0)
        prod = torch.fft.rfftn(x2.reshape(f.shape[0], -1, d, d, d), dim=(2, 3, 4)) * t

        def volume(p):
            return (torch.fft.irfftn(p.sum(1), s=(d, d, d), dim=(1, 2, 3)) * n3).reshape(f.shape[0], -1)

        if prob:
            alpha, vstd, vave, pstd, pave = _mix(qd)
            a, b = volume(prod[:, :3]), volume(prod[:, 3:])
            m = (1 - alpha) * (a - vave) / vstd + alpha * (b - pave) / pstd
            out.append(torch.stack([a.amax(1), b.amax(1), m.amax(1)], 1))
        else:
            out.append(volume(prod).amax(1, keepdim=True))
    return {"scores": torch.cat(out), "lin": None}


def _exact_fastvec(case, seed):
    side, d, s = case["side"], case["d"], case["s"]
    src, _, o2 = _fastvec_inputs(case, seed)
    half = 2.0 * BANDWIDTH
    pos = [torch.arange(d, dtype=torch.float64, device="cuda") * s + o for o in o2]
    grid = torch.arange(side, device="cuda")
    w = []
    for p in pos:
        lo = (p - half).long().clamp(min=0)
        hi = (p + half + 1.0).long().clamp(max=side)
        band = (grid[None] >= lo[:, None]) & (grid[None] < hi[:, None])
        w.append(torch.where(band, torch.exp(-1.5 * (grid[None] - p[:, None]) ** 2 / (0.5 * BANDWIDTH) ** 2), 0.0))
    moment = [a * grid[None] for a in w]

    def total(a, b, c):
        t = torch.matmul(src.double(), c.T)
        t = torch.einsum("xyk,jy->xjk", t, b)
        return torch.einsum("xjk,ix->ijk", t, a)

    dens = total(*w)
    at = [torch.where((p >= 0) & (p < side), p.long(), -1) for p in pos]
    inside = (at[0] >= 0)[:, None, None] & (at[1] >= 0)[None, :, None] & (at[2] >= 0)[None, None, :]
    i = [a.clamp(min=0) for a in at]
    keep = inside & (src[i[0]][:, i[1]][:, :, i[2]] != 0)
    some = keep & (dens != 0)
    mean = torch.stack([total(moment[0], w[1], w[2]), total(w[0], moment[1], w[2]), total(w[0], w[1], moment[2])], -1)
    v = mean / torch.where(some, dens, 1.0)[..., None] - torch.stack(torch.meshgrid(*pos, indexing="ij"), -1)
    norm = v.norm(dim=-1, keepdim=True)
    v = torch.where(some[..., None], v / torch.where(norm == 0, 1.0, norm), 0.0)
    dens = torch.where(keep, dens, 0.0)
    return {"data": dens, "data32": dens, "vec": v}


def _weights():
    z = np.load(vp.WEIGHTS)
    n = len(vp.CHANNELS) - 1
    return [torch.from_numpy(z["W%d" % i]).cuda().bfloat16().double() for i in range(n)], \
        [torch.from_numpy(z["b%d" % i]).cuda().double() for i in range(n)]


def _encode(fields, ws, bs):
    x = fields.double()
    for i, (w, b) in enumerate(zip(ws, bs)):
        x = torch.nn.functional.conv3d(x, w.reshape(w.shape[0], w.shape[1], 3, 3, 3), b, padding=1)
        x = torch.relu(x) if i + 1 < len(ws) else x
    return x


def _source_chunks(d, per):
    mats, every = _grid(GRID_STEP), torch.ones(d ** 3, dtype=torch.bool, device="cuda")
    for r0 in range(0, mats.shape[0], per):
        src = _sources(mats[r0:r0 + per], d, every)
        yield r0, torch.where(src < 0, d ** 3, src)


def _padded(feat):
    flat = feat.reshape(feat.shape[0], -1)
    return torch.cat([flat, torch.zeros_like(flat[:, :1])], 1)


def _exact_propose(case, seed):
    with torch.no_grad():
        feat = _encode(_pooled_fields(seed, case["pairs"], case["d"]), *_weights())
        out = [[] for _ in range(case["pairs"])]
        for _, src in _source_chunks(case["d"], 256):
            for i in range(case["pairs"]):
                t, q = feat[2 * i].reshape(feat.shape[1], -1), _padded(feat[2 * i + 1])
                out[i].append(sum((q[k][src] * t[k]).sum(1) for k in range(t.shape[0])))
    return {"scores": torch.stack([torch.cat(o) for o in out])}


def _exact_train(case, seed):
    ws, bs = _weights()
    for p in ws + bs:
        p.requires_grad_(True)
    feat = _encode(_pooled_fields(seed, 1, case["d"]), ws, bs)
    t, q = feat[0].detach().reshape(feat.shape[1], -1), _padded(feat[1].detach())
    s = torch.cat([sum((q[k][src] * t[k]).sum(1) for k in range(t.shape[0])) for _, src in _source_chunks(case["d"], 256)])
    s.requires_grad_(True)
    u = (s - s.mean()) / (s.std(unbiased=False) + 1e-6)
    loss = -(_labels(seed, s.numel()).double() * torch.log_softmax(u / 0.5, 0)).sum()
    gs, = torch.autograd.grad(loss, s)
    gt, gq = torch.zeros_like(t), torch.zeros_like(q)
    for r0, src in _source_chunks(case["d"], 256):
        g = gs[r0:r0 + src.shape[0], None]
        for k in range(t.shape[0]):
            gt[k] += (g * q[k][src]).sum(0)
            gq[k].index_add_(0, src.reshape(-1), (g * t[k]).reshape(-1))
    g = torch.stack([gt, gq[:, :-1]]).reshape(feat.shape)
    grads = torch.autograd.grad(feat, ws + bs, g)
    n = len(ws)
    return {"loss": loss.detach().reshape(1), "gW": list(grads[:n]), "gb": list(grads[n:])}


def exact(case, seed):
    if case["kind"] == "fastvec":
        return _exact_fastvec(case, seed)
    if case["kind"] in ("search", "prob"):
        return _exact_search(case, seed)
    if case["kind"] == "propose":
        return _exact_propose(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return None
