"""The work a user of this framework has it do, as measurable cases: single
image pairs, batched zones, regions that stream in, the descriptor producer,
RANSAC scoring and tracks, each through its public entry point (include/slm.h
or the skylens_match package).

Inputs are seeded synthetic data with the distributions of the benchmark
configurations: SIFT-like unit descriptors (|N(0,1)|, normalised, clipped at
0.2, normalised), views that share 30-60 % of their landmarks as noisy copies
(sigma 0.05), textured scenes for the detector, two-view geometry with noisy
and wrong matches for RANSAC.
"""
import ctypes
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "skylens-stream-rs_gb300"))

import skylens_match as sm  # noqa: E402
from skylens_match import features, synth, tracks  # noqa: E402
from skylens_match._lib import PRECISIONS, SlmKeypoint, SlmPair, SlmTrackStats, check  # noqa: E402

P = ctypes.POINTER
U64 = P(ctypes.c_uint64)


def listed():
    return [
        # the smallest ordinary call: two sparse views (300 is the least a zone's view has), host arrays, the
        # default precision: latency and launches
        {"name": "pair_317x300_fp32", "kind": "pair", "na": 317, "nb": 300, "true": 0.6, "prec": "fp32", "mutual": True},
        # one large pair from host arrays through the BF16 shortlist (the large single pair configuration)
        {"name": "pair_8192_bf16", "kind": "pair", "na": 8192, "nb": 8192, "true": 0.5, "prec": "bf16", "mutual": True},
        # the high-resolution FP8 pair, descriptors resident, its plan kept and launched again
        {"name": "pair_32768_fp8", "kind": "plan_pair", "na": 32768, "nb": 32768, "true": 0.4, "prec": "fp8",
         "mutual": True},
        # a newly arrived view against its partners in the store: one one-shot batch (a serving tick)
        {"name": "arrival_30_bf16", "kind": "arrival", "partners": 30, "lo": 500, "hi": 4000, "prec": "bf16",
         "mutual": True},
        # a region's views arrive in pinned host memory, are uploaded, matched by the pipeline's schedule and
        # filtered at 20 matches
        {"name": "region_96_bf16", "kind": "region", "positions": 32, "prec": "bf16", "mutual": True},
        # the headline: the 240-view zone's candidate pairs in one planned batch, lists read back
        {"name": "zone_240_bf16", "kind": "zone", "positions": 80, "prec": "bf16", "mutual": True},
        # a quarter of that zone on the plain FP32 kernel
        {"name": "zone_60_fp32", "kind": "zone", "positions": 20, "prec": "fp32", "mutual": True},
        # a batch of photos at the pipeline's frame size: pinned RGB8 in, descriptors left on the device
        {"name": "detect_24x960x540_rgb", "kind": "detect", "n": 24, "w": 960, "h": 540, "rgb": True},
        # one small gray photo of odd size (below 800 pixels, so the 2x upsampled detection runs too), host to host
        {"name": "detect_1x717x531_gray", "kind": "detect", "n": 1, "w": 717, "h": 531, "rgb": False},
        # descriptors of given keypoints of one photo
        {"name": "describe_1500", "kind": "describe", "w": 960, "h": 540, "n": 1500},
        # RANSAC scoring of a zone's kept pairs: 100 pairs of 200-550 matches, 2000 hypotheses each
        {"name": "ransac_100x2000", "kind": "ransac", "pairs": 100, "hyps": 2000, "lo": 200, "hi": 550, "masks": 100},
        # tracks of the 240-view zone's match lists
        {"name": "tracks_zone_240", "kind": "tracks", "positions": 80},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["pair", "pair", "plan_pair", "arrival", "region", "zone", "zone", "detect", "detect", "describe",
                       "ransac", "tracks"])
    mutual = rng.random() < 0.8
    if kind == "pair":
        return {"kind": kind, "na": _log(rng, 100, 8192), "nb": _log(rng, 100, 8192), "true": round(rng.uniform(0.2, 0.7), 3),
                "prec": rng.choice(["fp32", "bf16", "fp8", "auto"]), "mutual": mutual}
    if kind == "plan_pair":
        return {"kind": kind, "na": _log(rng, 1024, 32768), "nb": _log(rng, 1024, 32768),
                "true": round(rng.uniform(0.2, 0.6), 3), "prec": rng.choice(["bf16", "fp8"]), "mutual": mutual}
    if kind == "arrival":
        return {"kind": kind, "partners": rng.randint(1, 40), "lo": 500, "hi": 4000, "prec": rng.choice(["bf16", "bf16", "auto"]),
                "mutual": mutual}
    if kind == "region":
        return {"kind": kind, "positions": _log(rng, 3, 48), "prec": "bf16", "mutual": mutual}
    if kind == "zone":
        prec = rng.choice(["bf16", "bf16", "fp32", "fp8"])
        return {"kind": kind, "positions": _log(rng, 3, 20 if prec == "fp32" else 80 if prec == "bf16" else 40), "prec": prec,
                "mutual": mutual}
    if kind == "detect":
        w, h = _log(rng, 160, 1920), _log(rng, 120, 1080)
        most = max(1, min(24, 24 * 960 * 540 // (w * h * (5 if max(w, h) < 800 else 1))))
        return {"kind": kind, "n": _log(rng, 1, most), "w": w, "h": h, "rgb": rng.random() < 0.6}
    if kind == "describe":
        return {"kind": kind, "w": _log(rng, 320, 1920), "h": _log(rng, 240, 1080), "n": _log(rng, 1, 4000)}
    if kind == "ransac":
        pairs = _log(rng, 1, 200)
        return {"kind": kind, "pairs": pairs, "hyps": _log(rng, 200, min(20000, 200000 // pairs)), "lo": 20, "hi": _log(rng, 40, 600),
                "masks": rng.randint(0, pairs)}
    return {"kind": "tracks", "positions": _log(rng, 3, 80)}


# ------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)


def _normalise(x):
    x = x / x.norm(dim=1, keepdim=True).clamp_min(1e-30)
    x = x.clamp_max(0.2)
    return x / x.norm(dim=1, keepdim=True).clamp_min(1e-30)


def _sift(g, n):
    return _normalise(torch.randn(n, 128, device="cuda", generator=g).abs())


def _noisy(g, x, sigma):
    return _normalise(x + torch.randn(x.shape, device="cuda", generator=g) * sigma)


def _pair(case, seed):
    """a, b on the GPU: a share of b's rows are noisy copies of rows of a (sigma 0.05; 0.02-0.08 for FP8)."""
    g = _gen(seed)
    na, nb = case["na"], case["nb"]
    a = _sift(g, na)
    k = int(case["true"] * min(na, nb))
    src = torch.randperm(na, device="cuda", generator=g)[:k]
    sigma = 0.05
    if case["prec"] == "fp8":
        sigma = 0.02 + 0.06 * torch.rand(k, 1, device="cuda", generator=g)
    b = torch.cat([_noisy(g, a[src], sigma), _sift(g, nb - k)])
    return a, b[torch.randperm(nb, device="cuda", generator=g)].contiguous()


def _views(seed, positions, counts=None, lifetime=40, alive=1500, shared=0.595):
    """Views of a 3-camera rig along `positions`: descriptors (GPU), counts (the case's, whatever the seed), each row's
    landmark (-1: its own)."""
    rng = np.random.default_rng(int(seed) + 1)
    if counts is None:
        counts = np.random.default_rng(positions).integers(300, 2001, 3 * positions)
    n_land = int(np.ceil((positions + lifetime) * alive / lifetime))
    birth = np.sort(rng.uniform(-lifetime, positions, n_land))
    strength = rng.random(n_land)
    land = []
    for v, n in enumerate(counts):
        p = v // 3
        live = np.nonzero((birth <= p) & (birth + lifetime > p))[0]
        k = min(len(live), int(round(shared * n)))
        pick = live[np.argsort(-strength[live], kind="stable")[:k]]
        land.append(rng.permutation(np.concatenate([pick, np.full(n - k, -1)])))
    g = _gen(seed)
    base = _sift(g, n_land)
    lm = torch.from_numpy(np.concatenate(land)).cuda()
    own = _sift(g, len(lm))
    desc = torch.where((lm >= 0)[:, None], _noisy(g, base[lm.clamp_min(0)], 0.05 / 2 ** 0.5), own)
    return desc.contiguous(), np.asarray(counts), land


def _offsets(counts):
    return np.concatenate([[0], np.cumsum(counts)[:-1]]).astype(np.uint64)


def _store(desc, counts):
    """A store holding the views (device rows, one upload call)."""
    st = sm.default_matcher().store(int(np.sum(counts)), len(counts))
    torch.cuda.synchronize()
    st.add_views_ptr(desc.data_ptr(), _offsets(counts), counts)
    torch.cuda.synchronize()
    return st


def _plan_state(st, pairs, case):
    plan = st.plan(pairs, 0.8, case["mutual"], case["prec"])
    out = torch.zeros(max(plan.total_rows, 1), 2, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    return {"kind": "plan", "store": st, "plan": plan, "out": out, "off": np.zeros(plan.np + 1, np.uint64)}


def _lists(counts, pairs):
    """Room for the match lists of `pairs`, and their offsets."""
    return {"out": np.zeros((int(counts[pairs[:, 0]].sum()) + 1, 2), np.uint32), "off": np.zeros(len(pairs) + 1, np.uint64)}


def _two_view(rng, pairs, counts):
    """Matches of `pairs` calibrated image pairs, flat (M, 4), and each pair's essential matrix: 60 % inliers with
    half a pixel of noise at focal 800, the rest wrong."""
    def essential():
        ax = rng.normal(size=(pairs, 3))
        ax /= np.linalg.norm(ax, axis=1, keepdims=True)
        t = rng.normal(size=(pairs, 3))
        t /= np.linalg.norm(t, axis=1, keepdims=True)
        z = np.zeros(pairs)
        k = np.stack([z, -ax[:, 2], ax[:, 1], ax[:, 2], z, -ax[:, 0], -ax[:, 1], ax[:, 0], z], 1).reshape(-1, 3, 3)
        ang = rng.uniform(0.05, 0.35, pairs)[:, None, None]
        r = np.eye(3) + np.sin(ang) * k + (1 - np.cos(ang)) * (k @ k)
        tx = np.stack([z, -t[:, 2], t[:, 1], t[:, 2], z, -t[:, 0], -t[:, 1], t[:, 0], z], 1).reshape(-1, 3, 3)
        return r, t, tx @ r
    r, t, e = essential()
    who = np.repeat(np.arange(pairs), counts)
    m = len(who)
    x = np.stack([rng.uniform(-3, 3, m), rng.uniform(-3, 3, m), rng.uniform(4, 10, m)], 1)
    x2 = np.einsum("mij,mj->mi", r[who], x) + 0.5 * t[who]
    n1, n2 = x[:, :2] / x[:, 2:], x2[:, :2] / x2[:, 2:]
    n1, n2 = (v + rng.normal(0, 0.5 / 800, v.shape) for v in (n1, n2))
    bad = rng.random(m) < 0.4
    n2[bad] = rng.uniform(-0.6, 0.6, (int(bad.sum()), 2))
    return np.concatenate([n1, n2], 1), e, essential


def _image_views(seed, n, w, h):
    return synth.scene_views(n, w, h, seed=int(seed) + 11)


def prepare(case, seed):
    kind, m = case["kind"], sm.default_matcher()
    if kind == "pair":
        a, b = (v.cpu().numpy() for v in _pair(case, seed))
        return {"kind": kind, "case": case, "a": a, "b": b, "out": np.zeros((case["na"], 2), np.uint32), "m": m}
    if kind == "plan_pair":
        a, b = _pair(case, seed)
        return _plan_state(_store(torch.cat([a, b]), [len(a), len(b)]), [(0, 1)], case)
    if kind == "zone":
        desc, counts, _ = _views(seed, case["positions"])
        return _plan_state(_store(desc, counts), synth.candidate_pairs_np(synth.rig_views(case["positions"])), case)
    if kind == "arrival":
        k = case["partners"]
        rng = np.random.default_rng(k)
        n = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), 3 * (k // 3 + 1))).astype(np.int64)
        desc, counts, _ = _views(seed, len(n) // 3, n)
        pairs = np.array([(v, k) for v in range(k)], np.uint32)
        return {"kind": kind, "case": case, "m": m, "store": _store(desc, counts), "pairs": pairs, **_lists(counts, pairs)}
    if kind == "region":
        desc, counts, _ = _views(seed, case["positions"])
        host = torch.empty(desc.shape, dtype=torch.float32, pin_memory=True)
        host.copy_(desc)
        views = synth.rig_views(case["positions"])
        pairs = np.array(sm.scheduled_pairs(views), np.uint32).reshape(-1, 2)
        return {"kind": kind, "case": case, "m": m, "host": host, "counts": counts, "first": _offsets(counts),
                "store": m.store(int(counts.sum()), len(counts)), "views": np.array(views, np.uint64),
                "kept": np.zeros((len(pairs) + 1, 2), np.uint32), **_lists(counts, pairs)}
    if kind == "detect":
        n, w, h = case["n"], case["w"], case["h"]
        rgb = _image_views(seed, n, w, h)
        cfg = features.detector_config()
        cap = n * min(cfg.max_features, 256 + w * h // 80)
        st = {"kind": kind, "case": case, "m": m, "cfg": cfg, "cap": cap, "off": np.zeros(n + 1, np.uint64),
              "kps": np.zeros((cap, 5), np.float32)}
        if case["rgb"]:
            st["img"] = torch.empty(rgb.shape, dtype=torch.uint8, pin_memory=True)
            st["img"].copy_(torch.from_numpy(rgb))
            st["desc"] = torch.zeros(cap, 128, device="cuda")
        else:
            st["img"] = torch.from_numpy(np.ascontiguousarray(rgb.astype(np.float32).mean(axis=3, dtype=np.float32) / np.float32(255)))
            st["desc"] = torch.zeros(cap, 128)
        return st
    if kind == "describe":
        return {"kind": kind, "m": m, **_describe_input(case, seed)}
    if kind == "ransac":
        rng = np.random.default_rng(int(seed))
        np_, nh = case["pairs"], case["hyps"]
        counts = np.random.default_rng(np_).integers(case["lo"], case["hi"] + 1, np_)
        pts, e, essential = _two_view(rng, np_, counts)
        # a pool of 5-point hypotheses: some near the true matrix (noise of 1e-6 to 1e-1), the rest from wrong samples
        hp = np.repeat(np.arange(np_, dtype=np.uint32), nh)
        E = e[hp] + rng.normal(size=(len(hp), 3, 3)) * 10.0 ** rng.uniform(-6, -1, (len(hp), 1, 1))
        wrong = rng.random(len(hp)) < 0.66
        if np_ > 1:
            E[wrong] = essential()[2][rng.integers(0, np_, int(wrong.sum()))] + 0.3 * rng.normal(size=(int(wrong.sum()), 3, 3))
        masks = [int(k * nh + rng.integers(0, nh)) for k in range(case["masks"])]
        return {"kind": kind, "m": m, "pts": pts, "off": np.concatenate([[0], np.cumsum(counts)]).astype(np.uint64),
                "th": rng.uniform(1.0, 2.0, np_) / 800, "E": E, "hp": hp, "masks": masks}
    # tracks: the zone's matches by shared landmark, two in a hundred of them wrong
    rng = np.random.default_rng(int(seed) + 2)
    _, counts, land = _views(seed, case["positions"])
    order = [np.argsort(v, kind="stable") for v in land]
    sorted_ = [v[o] for v, o in zip(land, order)]
    pairs = []
    for u, v in synth.candidate_pairs_np(synth.rig_views(case["positions"])):
        s = sorted_[u]
        k = int(np.searchsorted(s, 0))
        at = np.searchsorted(sorted_[v], s[k:])
        ok = at < len(sorted_[v])
        ok[ok] = sorted_[v][at[ok]] == s[k:][ok]
        i, j = order[u][k:][ok], order[v][at[ok]]
        j = np.where(rng.random(len(j)) < 0.02, rng.integers(0, counts[v], len(j)), j)
        pairs.append((int(u), int(v), np.stack([i, j], 1)))
    arr, flat = tracks.pack(pairs)
    return {"kind": "tracks", "m": m, "nf": counts.astype(np.uint32), "arr": arr, "np": len(pairs), "flat": flat,
            "toff": np.zeros(int(counts.sum()) + 1, np.uint64), "obs": np.zeros((int(counts.sum()), 2), np.uint32)}


def _describe_input(case, seed):
    w, h, n = case["w"], case["h"], case["n"]
    img = synth.scene_canvas(w, h, seed=int(seed) + 29)
    rng = np.random.default_rng(int(seed))
    kp = np.stack([rng.uniform(0, w - 1, n), rng.uniform(0, h - 1, n), np.exp(rng.uniform(np.log(1.6), np.log(13.0), n)),
                   np.zeros(n), rng.uniform(0, 2 * np.pi, n)], 1).astype(np.float32)
    return {"img": img, "kp": kp}


# -------------------------------------------------------------------- passes

def _ptr(a, t):
    return a.ctypes.data_as(P(t))


def run(s):
    """Lists come back in the caller's buffers, whole: what lies past the lists' end stays as prepare() made it."""
    kind = s["kind"]
    if kind == "plan":
        s["plan"].launch()
        s["plan"].results_into(s["out"], s["off"])
        return s["out"].view(np.int32), s["off"].view(np.int64)
    if kind == "describe":
        return features.describe(s["m"], s["img"], s["kp"])
    if kind == "ransac":
        counts, masks = s["m"].sampson_score(s["pts"], s["off"], s["th"], s["E"], s["hp"], s["masks"])
        return counts.view(np.int32), np.concatenate(list(masks.values())) if masks else np.zeros(1, bool)
    m = s["m"]
    c, lib, n = s.get("case"), m._L, ctypes.c_uint64()
    if kind == "pair":
        n = ctypes.c_uint32()
        check(lib.slm_ratio_match(m.handle, _ptr(s["a"], ctypes.c_float), c["na"], _ptr(s["b"], ctypes.c_float), c["nb"],
                                  ctypes.c_float(0.8), int(c["mutual"]), PRECISIONS[c["prec"]], _ptr(s["out"], SlmPair),
                                  c["na"], ctypes.byref(n), None), "slm_ratio_match")
        return s["out"].view(np.int32), n.value
    if kind == "arrival":
        check(lib.slm_match_batch(m.handle, s["store"].handle, _ptr(s["pairs"], SlmPair), len(s["pairs"]),
                                  ctypes.c_float(0.8), int(c["mutual"]), PRECISIONS[c["prec"]], _ptr(s["out"], SlmPair),
                                  len(s["out"]), _ptr(s["off"], ctypes.c_uint64), None), "slm_match_batch")
        return s["out"].view(np.int32), s["off"].view(np.int64)
    if kind == "region":
        st = s["store"]
        st.clear()
        st.add_views_ptr(s["host"].data_ptr(), s["first"], s["counts"])
        check(lib.slm_match_pairs(m.handle, st.handle, _ptr(s["views"], ctypes.c_uint64), len(s["views"]), None,
                                  ctypes.c_float(0.8), int(c["mutual"]), PRECISIONS[c["prec"]], 20, _ptr(s["kept"], SlmPair),
                                  len(s["kept"]) - 1, ctypes.byref(n), _ptr(s["out"], SlmPair), len(s["out"]),
                                  _ptr(s["off"], ctypes.c_uint64), None), "slm_match_pairs")
        return s["kept"].view(np.int32), s["out"].view(np.int32), s["off"].view(np.int64), n.value
    if kind == "detect":
        fn = lib.slm_detect_and_describe_rgb8 if c["rgb"] else lib.slm_detect_and_describe
        check(fn(m.handle, ctypes.c_void_p(s["img"].data_ptr()), c["n"], c["w"], c["h"], ctypes.byref(s["cfg"]),
                 s["kps"].ctypes.data_as(ctypes.c_void_p), ctypes.c_void_p(s["desc"].data_ptr()), s["cap"],
                 _ptr(s["off"], ctypes.c_uint64)), "slm_detect_and_describe")
        return s["kps"], s["desc"], s["off"].view(np.int64)
    nt, stats = ctypes.c_uint64(), SlmTrackStats()
    check(lib.slm_build_tracks_drop(m.handle, _ptr(s["nf"], ctypes.c_uint32), len(s["nf"]), s["arr"], s["np"],
                                    _ptr(s["flat"], SlmPair), 3, 100_000, _ptr(s["toff"], ctypes.c_uint64),
                                    len(s["toff"]) - 1, _ptr(s["obs"], SlmPair), len(s["obs"]), ctypes.byref(nt),
                                    ctypes.byref(n), ctypes.byref(stats)), "slm_build_tracks_drop")
    return s["toff"].view(np.int64), s["obs"].view(np.int32), np.array(list(stats.as_dict().values()), np.int64)


# ---------------------------------------------------------------------- work

def work(case):
    """Bytes: each input read once and each output written once. Operations: one 128-long dot product a distance
    (2 x 128) for the tensor-core precisions, subtract, multiply and add (3 x 128) for plain FP32; the detector's
    blurs and window samples; a residual's 34 multiplies and adds, division and root."""
    kind = case["kind"]
    per = 384 if case.get("prec") == "fp32" else 256
    if kind in ("pair", "plan_pair"):
        na, nb = case["na"], case["nb"]
        return {"bytes": 512 * (na + nb) + 8 * int(case["true"] * min(na, nb)), "flops": per * na * nb}
    if kind == "arrival":
        mean = float((case["hi"] - case["lo"]) / np.log(case["hi"] / case["lo"]))
        return {"bytes": 512 * mean * (case["partners"] + 1), "flops": per * case["partners"] * mean * mean}
    if kind in ("zone", "region"):
        views, pairs = 3 * case["positions"], len(synth.candidate_pairs_np(synth.rig_views(case["positions"])))
        if kind == "region":
            pairs = len(sm.scheduled_pairs(synth.rig_views(case["positions"])))
        return {"bytes": 512 * 1150 * views + 8 * 0.4 * 1150 * pairs, "flops": per * pairs * 1150 * 1150}
    if kind == "detect":
        px = case["n"] * case["w"] * case["h"] * (5 if max(case["w"], case["h"]) < 800 else 1)
        feats = 0.0023 * px
        # 4/3 of a level's pixels over the octaves; six layers blurred with about 25 taps in two directions
        return {"bytes": case["n"] * case["w"] * case["h"] * (3 if case["rgb"] else 4) + feats * (512 + 20),
                "flops": px * 4 / 3 * (6 * 2 * 25 + 3 * 20 + 3 * 26) + feats * 2000 * 40}
    if kind == "describe":
        return {"bytes": 4 * case["w"] * case["h"] + case["n"] * (512 + 20), "flops": case["w"] * case["h"] * 20 + case["n"] * 3000 * 40}
    if kind == "ransac":
        m, h = case["pairs"] * (case["lo"] + case["hi"]) / 2, case["pairs"] * case["hyps"]
        return {"bytes": 32 * m + 76 * h, "flops": 36 * h * (case["lo"] + case["hi"]) / 2}
    pairs = len(synth.candidate_pairs_np(synth.rig_views(case["positions"])))
    return {"bytes": 8 * 460 * pairs + 8 * 1150 * 3 * case["positions"], "flops": 10 * 460 * pairs}


# --------------------------------------------------------------------- exact

def exact(case, seed):
    """describe() in 64 bits. Every other output is whole numbers, or, for the detector, a list whose length and order
    hang on comparisons of 32-bit values (which extrema pass, which orientation peaks): 64 bits give another list."""
    if case["kind"] != "describe":
        return None
    s = _describe_input(case, seed)
    im = s["img"].astype(np.float64)
    h, w = im.shape
    mag, ang = np.zeros((h, w)), np.zeros((h, w))
    gx, gy = im[1:-1, 2:] - im[1:-1, :-2], im[2:, 1:-1] - im[:-2, 1:-1]
    mag[1:-1, 1:-1], ang[1:-1, 1:-1] = np.hypot(gx, gy), np.arctan2(gy, gx)
    out = np.zeros((len(s["kp"]), 128))
    for q, (x, y, sig, _, a) in enumerate(s["kp"].astype(np.float64)):
        cell = 3.0 * sig
        r = int(np.floor(cell * np.sqrt(2.0) * 2.5 + 0.5))
        xi, yi = int(np.floor(x + 0.5)), int(np.floor(y + 0.5))
        py, px = np.mgrid[max(1, yi - r):min(h - 1, yi + r + 1), max(1, xi - r):min(w - 1, xi + r + 1)]
        py, px = py.ravel(), px.ravel()
        fx, fy = px - x, py - y
        u, v = (np.cos(a) * fx + np.sin(a) * fy) / cell, (-np.sin(a) * fx + np.cos(a) * fy) / cell
        bu, bv = u + 1.5, v + 1.5
        k = (bu > -1) & (bv > -1) & (bu < 4) & (bv < 4)
        u, v, bu, bv, py, px = u[k], v[k], bu[k], bv[k], py[k], px[k]
        m = mag[py, px] * np.exp(-(u * u + v * v) / 8.0)
        bo = np.mod(ang[py, px] - a, 2 * np.pi) / (2 * np.pi) * 8
        hist = np.zeros((6, 6, 9))  # a margin of one cell around the 4 x 4
        u0, v0, o0 = np.floor(bu).astype(int), np.floor(bv).astype(int), np.floor(bo).astype(int)
        for dv in (0, 1):
            for du in (0, 1):
                for do in (0, 1):
                    wgt = m * np.abs(1 - dv - (bv - v0)) * np.abs(1 - du - (bu - u0)) * np.abs(1 - do - (bo - o0))
                    np.add.at(hist, (v0 + dv + 1, u0 + du + 1, (o0 + do) % 8), wgt)
        d = hist[1:5, 1:5, :8].ravel()
        for clip in (0.2, np.inf):
            n = np.sqrt((d * d).sum())
            d = np.minimum(d / n if n > 0 else d, clip)
        out[q] = d
    return out
