"""Performance cases of the feature hot path: what a program that uses this library has it do.

Each case is one call, or one short sequence of calls, through the public entry points
(`psift.py` and the C ABI it mirrors), over synthetic inputs with the statistics of the
package's own workloads (`synth.py`): Gaussian-blob images, SIFT-like descriptors, putative
matches with known geometry.  Host entries get host arrays; the `_dev` / batch entries get
device buffers and queue their work on the context's stream, as a pipeline that keeps its data on
the GPU calls them.

Kinds:
  detect          one host image into the caller's feature arrays (the per-image call)
  detect_batch    device-resident batch, equal sizes or ragged, features left on the device
  pair            one image pair on the host: Lowe matching, then the homography estimate
  match_batch     device-resident batch of matching problems
  ransac_batch    device-resident batch of similarity / homography estimations
  fundamental     device-resident batch of fundamental-matrix estimations
  panorama        stitch_panorama of overlapping RGBA tiles (registration and compositing)
  catalog_search  search_features on a device-resident catalog
  catalog_topk    binarise queries, top-k Hamming shortlist, exact L2 re-rank
  sampler         train the learned sampler, then score every match with it
"""
import ctypes as C
import math
import os
import random
import struct
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pure-sift_b200"))
import psift  # noqa: E402
import synth  # noqa: E402

DESC_BYTES = 128 * 4
FEATURE_BYTES = 5 * 4 + DESC_BYTES
MATCH_BYTES = 40


def listed():
    return [
        # The smallest everyday call: one camera frame from host memory, library defaults.  Latency and
        # launches count, not bandwidth.
        {"name": "detect_vga_u8", "kind": "detect", "height": 480, "width": 640, "f32": False, "octaves": 3,
         "scales": 3, "upsample": True, "rootsift": False},
        # The reference's own call pattern: one full-HD f32 luma image per detect_and_compute call.
        {"name": "detect_1080p_f32", "kind": "detect", "height": 1080, "width": 1920, "f32": True, "octaves": 4,
         "scales": 3, "upsample": True, "rootsift": False},
        # Bulk extraction of equal frames kept on the device (the benchmark's headline batch).
        {"name": "detect_batch8_1080p", "kind": "detect_batch", "n": 8, "height": 1080, "width": 1920,
         "ragged": False, "octaves": 4, "scales": 3, "upsample": True, "rootsift": False, "max_features": 4096},
        # A photo collection: images of different, odd sizes in one batch, RootSIFT, no feature cap.
        {"name": "detect_ragged12", "kind": "detect_batch", "n": 12, "height": 2101, "width": 2731,
         "ragged": True, "octaves": 4, "scales": 3, "upsample": True, "rootsift": True, "max_features": 0},
        # Two images already described on the host: exact f32 mutual matching and the homography.
        {"name": "pair_host_fp32", "kind": "pair", "nq": 1837, "nt": 1503, "ratio": 0.75, "mutual": True,
         "fp32": True},
        # Many-pair matching at the feature cap with the default arithmetic (tensor cores, certified).
        {"name": "match_batch32_4096", "kind": "match_batch", "n": 32, "nq": 4096, "nt": 4096, "ragged": False,
         "ratio": 0.8, "mutual": False, "fp32": False},
        # Geometric verification of a batch of pairs: homography RANSAC with the library's sampling.
        {"name": "homography_batch128", "kind": "ransac_batch", "n": 128, "lo": 2000, "hi": 8000,
         "outliers_lo": 0.1, "outliers_hi": 0.7, "homography": True, "guided": False},
        # Two-view geometry of a batch of pairs.
        {"name": "fundamental_batch48", "kind": "fundamental", "n": 48, "lo": 2000, "hi": 8000,
         "outliers_lo": 0.1, "outliers_hi": 0.6},
        # A whole application call: register and blend four overlapping tiles.
        {"name": "panorama_4x960x540", "kind": "panorama", "n": 4, "height": 540, "width": 960, "overlap": 0.3,
         "multiband": True},
        # Image retrieval: one 4096-feature query against a resident catalog of 2000 images.
        {"name": "catalog_search_2000", "kind": "catalog_search", "entries": 2000, "per_entry": 200, "nq": 4096},
        # Large-scale shortlist: every query against two million binary codes, top 64, exact re-rank.
        {"name": "catalog_topk_2M", "kind": "catalog_topk", "ncat": 2_000_000, "nq": 4096, "k": 64},
        # Learned sampler: 100 training steps (forward and backward), then inference over all matches.
        {"name": "sampler_train_infer", "kind": "sampler", "n": 300_000, "steps": 100, "batch": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["detect", "detect", "detect_batch", "detect_batch", "pair", "match_batch", "ransac_batch",
                       "fundamental", "panorama", "catalog_search", "catalog_topk", "sampler"])
    flag = lambda: rng.random() < 0.5  # noqa: E731
    if kind == "detect":
        w = _log_int(rng, 320, 1920)
        return {"kind": kind, "height": max(200, int(w * rng.uniform(0.5, 1.1))), "width": w, "f32": flag(),
                "octaves": rng.choice([3, 4, 5]), "scales": rng.choice([3, 3, 3, 2, 4]), "upsample": rng.random() < 0.8,
                "rootsift": flag()}
    if kind == "detect_batch":
        ragged = flag()
        w = _log_int(rng, 400, 2700 if ragged else 1920)
        return {"kind": kind, "n": rng.randint(2, 12 if ragged else 8), "height": max(300, int(w * rng.uniform(0.5, 0.75))),
                "width": w, "ragged": ragged, "octaves": rng.choice([3, 4]), "scales": 3,
                "upsample": rng.random() < 0.8, "rootsift": flag(), "max_features": rng.choice([0, 2000, 4096])}
    if kind == "pair":
        return {"kind": kind, "nq": _log_int(rng, 200, 4096), "nt": _log_int(rng, 200, 4096),
                "ratio": rng.choice([0.75, 0.8]), "mutual": flag(), "fp32": flag()}
    if kind == "match_batch":
        fp32 = flag()
        return {"kind": kind, "n": _log_int(rng, 2, 8 if fp32 else 32), "nq": _log_int(rng, 300, 4096),
                "nt": _log_int(rng, 300, 4096), "ragged": flag(), "ratio": rng.choice([0.75, 0.8]), "mutual": flag(),
                "fp32": fp32}
    if kind == "ransac_batch":
        lo = _log_int(rng, 100, 4000)
        return {"kind": kind, "n": _log_int(rng, 8, 128), "lo": lo, "hi": 2 * lo, "outliers_lo": 0.1,
                "outliers_hi": rng.uniform(0.3, 0.7), "homography": rng.random() < 0.7, "guided": flag()}
    if kind == "fundamental":
        lo = _log_int(rng, 200, 4000)
        return {"kind": kind, "n": _log_int(rng, 4, 48), "lo": lo, "hi": 2 * lo, "outliers_lo": 0.1,
                "outliers_hi": rng.uniform(0.3, 0.6)}
    if kind == "panorama":
        w = _log_int(rng, 480, 960)
        return {"kind": kind, "n": rng.randint(2, 4), "height": int(w * rng.uniform(0.5, 0.7)), "width": w,
                "overlap": rng.uniform(0.3, 0.45), "multiband": flag()}
    if kind == "catalog_search":
        return {"kind": kind, "entries": _log_int(rng, 200, 2000), "per_entry": rng.randint(100, 200),
                "nq": _log_int(rng, 400, 4096)}
    if kind == "catalog_topk":
        return {"kind": kind, "ncat": _log_int(rng, 50_000, 2_000_000), "nq": _log_int(rng, 128, 4096),
                "k": rng.choice([16, 32, 64])}
    return {"kind": kind, "n": _log_int(rng, 20_000, 300_000), "steps": rng.randint(20, 100),
            "batch": rng.choice([1024, 2048, 4096])}


# ---------------------------------------------------------------- inputs

def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((seed * 1_000_003 + salt * 7919 + 17) & 0x7FFFFFFF)
    return g


def _scene(h, w, g, density=2000.0, noise=3.0):
    """u8 blob image on the GPU with synth.blob_image's statistics (128 background, sigma U(1.5, 20),
    amplitude +-U(40, 120), N(0, 3) noise); the sum of separable Gaussians is one matrix product."""
    n = max(8, int(density * h * w / (1920 * 1080)))
    u = torch.rand((5, n), generator=g, device="cuda")
    sig = 1.5 + 18.5 * u[2]
    amp = (40.0 + 80.0 * u[3]) * torch.where(u[4] < 0.5, 1.0, -1.0)
    ys = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    xs = torch.arange(w, device="cuda", dtype=torch.float32)[:, None]
    gy = torch.exp(-0.5 * ((ys - u[1] * h) / sig) ** 2)
    gx = torch.exp(-0.5 * ((xs - u[0] * w) / sig) ** 2) * amp
    img = 128.0 + gy @ gx.T
    if noise > 0:
        img = img + noise * torch.randn((h, w), generator=g, device="cuda")
    return img.round().clamp_(0, 255).to(torch.uint8)


def _descriptors(n, g):
    """synth.sift_like_descriptors on the GPU."""
    d = torch.randn((n, 128), generator=g, device="cuda").abs_()
    d /= d.norm(dim=1, keepdim=True)
    d.clamp_(max=0.2)
    d /= d.norm(dim=1, keepdim=True)
    return d


def _pair_descriptors(nq, nt, g):
    """Query and target descriptors; the first third of the queries are perturbed targets."""
    t = _descriptors(nt, g)
    q = _descriptors(nq, g)
    k = min(nq, nt) // 3
    q[:k] = t[:k] + 0.02 * _descriptors(k, g)
    return q, t, k


def _pair_points(nq, nt, k, g):
    """Coordinates: the k true pairs follow a similarity with 0.5 px noise, the rest are uniform."""
    size = torch.tensor([1920.0, 1080.0], device="cuda")
    qxy = torch.rand((nq, 2), generator=g, device="cuda") * size
    txy = torch.rand((nt, 2), generator=g, device="cuda") * size
    c, s = 1.1 * math.cos(0.2), 1.1 * math.sin(0.2)
    rot = torch.tensor([[c, s], [-s, c]], device="cuda")
    txy[:k] = qxy[:k] @ rot + torch.tensor([40.0, -25.0], device="cuda")
    txy[:k] += 0.5 * torch.randn((k, 2), generator=g, device="cuda")
    return qxy.contiguous(), txy.contiguous()


def _match_sizes(case):
    n, nq, nt = case["n"], case["nq"], case["nt"]
    if not case["ragged"]:
        return [(nq, nt)] * n
    r = random.Random(n * 31 + nq * 7 + nt)
    return [(max(2, int(nq * r.uniform(0.3, 1.0))), max(2, int(nt * r.uniform(0.3, 1.0)))) for _ in range(n)]


def _image_shapes(case):
    n, h, w = case["n"], case["height"], case["width"]
    if not case["ragged"]:
        return [(h, w)] * n
    r = random.Random(n * 131 + h * 7 + w)  # sides from a quarter of the largest up, either aspect
    return [(max(160, int(h * r.uniform(0.25, 1.0))), max(200, int(w * r.uniform(0.25, 1.0)))) for _ in range(n)]


def _set_sizes(case):
    r = random.Random(case["n"] * 17 + case["lo"])
    return [(r.randint(case["lo"], case["hi"]), r.uniform(case["outliers_lo"], case["outliers_hi"]))
            for _ in range(case["n"])]


def _config(case):
    c = psift.SiftConfig().with_octaves(case["octaves"]).with_scales(case["scales"])
    c = c.upsample_first_octave(case["upsample"]).descriptor_kind(int(case["rootsift"]))
    return c.max_features(case.get("max_features", psift.MAX_FEATURES_PER_IMAGE))


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def _prepare_detect(case, seed):
    img = _scene(case["height"], case["width"], _gen(seed)).cpu().numpy()
    if case["f32"]:
        img = (img.astype(np.float32) * np.float32(1.0 / 255.0)).astype(np.float32)
    cap = psift.MAX_FEATURES_PER_IMAGE
    out = {k: np.zeros(cap, np.float32) for k in ("x", "y", "scale", "response", "orientation")}
    out["descriptors"] = np.zeros((cap, 128), np.float32)
    return {"kind": "detect", "cfg": _config(case).to_c(), "img": img, "f32": case["f32"],
            "ctx": psift.default_context(), "out": out,
            "features": psift.CFeatures(cap, 0, *(a.ctypes.data for a in out.values()))}


def _run_detect(s):
    ctx, img, f = s["ctx"], s["img"], s["features"]
    h, w = img.shape
    fn = ctx.lib.psift_detect_and_compute if s["f32"] else ctx.lib.psift_detect_and_compute_u8
    ctx.check(fn(ctx.handle, img.ctypes.data, h, w, w, C.byref(s["cfg"]), C.byref(f)))
    return {"count": f.count, **s["out"]}


def _prepare_detect_batch(case, seed):
    shapes = _image_shapes(case)
    n = len(shapes)
    imgs = [_scene(h, w, _gen(seed, i)) for i, (h, w) in enumerate(shapes)]
    cap = case["max_features"] or 16384
    cols = {k: torch.zeros((n, cap), device="cuda") for k in ("x", "y", "scale", "response", "orientation")}
    desc = torch.zeros((n, cap, 128), device="cuda")
    counts = torch.zeros(n, dtype=torch.int32, device="cuda")
    cimgs = (psift.CImageU8 * n)(*[psift.CImageU8(t.data_ptr(), t.shape[0], t.shape[1], t.shape[1]) for t in imgs])
    couts = (psift.CFeatures * n)(*[psift.CFeatures(cap, 0, *(cols[k][i].data_ptr() for k in cols),
                                                    desc[i].data_ptr()) for i in range(n)])
    return {"kind": "detect_batch", "ctx": psift.default_context(), "n": n, "imgs": imgs, "cimgs": cimgs,
            "couts": couts, "cfg": _config(case).to_c(), "counts": counts,
            "out": {**cols, "descriptors": desc, "counts": counts}}


def _run_detect_batch(s):
    ctx = s["ctx"]
    ctx.check(ctx.lib.psift_detect_and_compute_batch_dev(ctx.handle, s["cimgs"], s["n"], C.byref(s["cfg"]),
                                                         s["couts"], s["counts"].data_ptr()))
    return s["out"]


def _prepare_pair(case, seed):
    g = _gen(seed)
    nq, nt = case["nq"], case["nt"]
    q, t, k = _pair_descriptors(nq, nt, g)
    qxy, txy = _pair_points(nq, nt, k, g)
    wrong = torch.rand(k, generator=g, device="cuda") < 0.25  # repeated structure: right descriptor, wrong place
    txy[:k][wrong] = txy[:k].flip(0)[wrong]
    opt = psift.MatchOptions(case["ratio"], case["mutual"],
                             psift.PRECISION_FP32 if case["fp32"] else psift.PRECISION_BF16_RERANK)
    return {"kind": "pair", "ctx": psift.default_context(), "match": opt.to_c(),
            "ransac": psift.RansacOptions().to_c(), "q": q.cpu().numpy(), "t": t.cpu().numpy(),
            "qxy": qxy.cpu().numpy(), "txy": txy.cpu().numpy(), "matches": np.zeros(nq, psift.MATCH_DTYPE),
            "inliers": np.zeros(nq, np.uint8), "h": np.zeros(9, np.float32)}


def _run_pair(s):
    ctx, lib, m = s["ctx"], s["ctx"].lib, s["matches"]
    n, has, inliers = C.c_uint32(), C.c_int32(), C.c_uint32()
    ctx.check(lib.psift_match_descriptors(ctx.handle, s["q"].ctypes.data, len(s["q"]), s["t"].ctypes.data,
                                          len(s["t"]), s["qxy"].ctypes.data, s["txy"].ctypes.data,
                                          C.byref(s["match"]), m.ctypes.data, len(m), C.byref(n)))
    ctx.check(lib.psift_homography_estimate(ctx.handle, m.ctypes.data, n.value, C.byref(s["ransac"]),
                                            s["inliers"].ctypes.data, s["h"].ctypes.data, C.byref(has),
                                            C.byref(inliers)))
    rec = m.view(np.int32).reshape(-1, 10)
    return {"counts": [n.value, has.value, inliers.value], "index": rec[:, :2], "values": rec.view(np.float32)[:, 2:],
            "inliers": s["inliers"], "homography": s["h"]}


def _prepare_match_batch(case, seed):
    sizes = _match_sizes(case)
    n, cap = len(sizes), max(a for a, _ in sizes)
    keep, jobs = [], (psift.CMatchJob * n)()
    out = torch.zeros((n, cap, 10), dtype=torch.int32, device="cuda")
    counts = torch.zeros(n, dtype=torch.int32, device="cuda")
    for i, (nq, nt) in enumerate(sizes):
        g = _gen(seed, i)
        q, t, k = _pair_descriptors(nq, nt, g)
        qxy, txy = _pair_points(nq, nt, k, g)
        keep.append((q, t, qxy, txy))
        jobs[i] = psift.CMatchJob(q.data_ptr(), t.data_ptr(), qxy.data_ptr(), txy.data_ptr(), nq, nt,
                                  out[i].data_ptr(), cap, counts[i:].data_ptr())
    opt = psift.MatchOptions(case["ratio"], case["mutual"],
                             psift.PRECISION_FP32 if case["fp32"] else psift.PRECISION_BF16_RERANK)
    return {"kind": "match_batch", "ctx": psift.default_context(), "n": n, "jobs": jobs, "opt": opt.to_c(),
            "keep": keep, "out": {"counts": counts, "index": out[:, :, :2],
                                  "values": out.view(torch.float32)[:, :, 2:]}}


def _run_match_batch(s):
    ctx = s["ctx"]
    ctx.check(ctx.lib.psift_match_batch_dev(ctx.handle, s["jobs"], s["n"], C.byref(s["opt"])))
    return s["out"]


def _prepare_ransac_batch(case, seed):
    n = case["n"]
    recs, feats = [], []
    for i, (m, outliers) in enumerate(_set_sizes(case)):
        u = synth.SplitMix64(seed * 10007 + i).uniform(4)
        h = synth.perspective_h(1920, 1080, -30 + 60 * u[0], 0.7 + 0.7 * u[1], -2e-4 + 4e-4 * u[2],
                                -2e-4 + 4e-4 * u[3])
        rec, ft, _ = synth.putative_matches(m, outliers, h, 1920, 1080, seed * 10007 + 7 * i + 1)
        recs.append(rec)
        feats.append(ft)
    off = np.concatenate([[0], np.cumsum([len(r) for r in recs])])
    d = torch.from_numpy(np.concatenate(recs).view(np.uint8)).cuda()
    mask = torch.zeros(int(off[-1]), dtype=torch.uint8, device="cuda")
    info = torch.zeros((n, 16), dtype=torch.int32, device="cuda")  # count, has, iterations x 2, model
    weights = None
    if case["guided"]:  # a sampler's probabilities: falling with the Lowe ratio and the scale disagreement
        f = torch.from_numpy(np.concatenate(feats)).cuda()
        weights = torch.sigmoid(6.0 * (0.75 - f[:, 0]) - 2.0 * f[:, 1].abs()).clamp_(min=0.02).contiguous()
    jobs = (psift.CRansacJob * n)()
    for i in range(n):
        base = info[i].data_ptr()
        jobs[i] = psift.CRansacJob(d.data_ptr() + MATCH_BYTES * int(off[i]), len(recs[i]),
                                   mask.data_ptr() + int(off[i]), base + 16, base + 4, base,
                                   weights.data_ptr() + 4 * int(off[i]) if weights is not None else None, base + 8)
    model = info.view(torch.float32)[:, 4:13 if case["homography"] else 10]
    return {"kind": "ransac_batch", "ctx": psift.default_context(), "n": n, "jobs": jobs, "keep": (d, weights),
            "opt": psift.RansacOptions().to_c(), "homography": int(case["homography"]),
            "out": {"inliers": mask, "info": info[:, :4], "model": model}}


def _run_ransac_batch(s):
    ctx = s["ctx"]
    ctx.check(ctx.lib.psift_ransac_batch_dev(ctx.handle, s["jobs"], s["n"], C.byref(s["opt"]), s["homography"]))
    return s["out"]


def _prepare_fundamental(case, seed):
    n = case["n"]
    recs = [synth.epipolar_matches(m, o, seed * 20011 + i)[0] for i, (m, o) in enumerate(_set_sizes(case))]
    off = np.concatenate([[0], np.cumsum([len(r) for r in recs])])
    d = torch.from_numpy(np.concatenate(recs).view(np.uint8)).cuda()
    mask = torch.zeros(int(off[-1]), dtype=torch.uint8, device="cuda")
    f = torch.zeros((n, 9), dtype=torch.float64, device="cuda")
    info = torch.zeros((n, 4), dtype=torch.int32, device="cuda")  # has, count, iterations
    jobs = (psift.CFundamentalJob * n)()
    for i in range(n):
        base = info[i].data_ptr()
        jobs[i] = psift.CFundamentalJob(d.data_ptr() + MATCH_BYTES * int(off[i]), len(recs[i]),
                                        mask.data_ptr() + int(off[i]), f[i].data_ptr(), base, base + 4, base + 8)
    return {"kind": "fundamental", "ctx": psift.default_context(), "n": n, "jobs": jobs, "keep": d,
            "opt": psift.FundamentalRansacOptions().to_c(), "out": {"inliers": mask, "f": f, "info": info}}


def _run_fundamental(s):
    ctx = s["ctx"]
    ctx.check(ctx.lib.psift_fundamental_batch_dev(ctx.handle, s["jobs"], s["n"], C.byref(s["opt"])))
    return s["out"]


def _prepare_panorama(case, seed):
    n, h, w = case["n"], case["height"], case["width"]
    step = int(w * (1.0 - case["overlap"]))
    rgb = torch.stack([_scene(h, step * (n - 1) + w, _gen(seed, c), noise=0.0) for c in range(3)], dim=-1).float()
    tiles = []
    for i in range(n):
        v = (rgb[:, i * step:i * step + w] * (0.9, 1.0, 1.1, 0.95)[i]).round_().clamp_(0, 255).to(torch.uint8)
        a = torch.full((h, w, 1), 255, dtype=torch.uint8, device="cuda")
        tiles.append(torch.cat([v, a], dim=-1).cpu().numpy())
    blend = psift.PanoramaOptions.BLEND_MULTIBAND if case["multiband"] else psift.PanoramaOptions.BLEND_FEATHER
    arr = (psift.CRgbaImage * n)(*[psift.CRgbaImage(t.ctypes.data, h, w, 4 * w) for t in tiles])
    return {"kind": "panorama", "ctx": psift.default_context(), "n": n, "tiles": tiles, "arr": arr,
            "opt": psift.PanoramaOptions.default(blend=blend), "info": psift.CPanoramaInfo(),
            "out": {"canvas": np.zeros(8 * n * h * w, np.uint8), "registered": np.zeros(n, np.uint8),
                    "gains": np.zeros(n, np.float32), "homographies": np.zeros((n, 9), np.float32)}}


def _run_panorama(s):
    ctx, o, info = s["ctx"], s["out"], s["info"]
    ctx.check(ctx.lib.psift_stitch_panorama(ctx.handle, s["arr"], s["n"], C.byref(s["opt"]), o["canvas"].ctypes.data,
                                            o["canvas"].nbytes, C.byref(info), o["registered"].ctypes.data,
                                            o["gains"].ctypes.data, o["homographies"].ctypes.data))
    return {"size": [info.width, info.height], "reference": info.reference_index,
            "origin": [info.origin_x, info.origin_y], **o}


def _entry_sizes(case):
    r = random.Random(case["entries"] * 13 + case["per_entry"])
    return [r.randint(int(0.6 * case["per_entry"]), int(1.4 * case["per_entry"])) for _ in range(case["entries"])]


def _codes_of(d):
    """quantize_descriptor_u128's bits of device descriptors, as host (n, 2) u64."""
    bits = np.packbits((d > 0.065).cpu().numpy(), axis=1, bitorder="little")
    return np.ascontiguousarray(bits).view("<u8")


def _prepare_catalog_search(case, seed):
    g = _gen(seed)
    sizes = _entry_sizes(case)
    n = sum(sizes)
    off = np.concatenate([[0], np.cumsum(sizes)])
    d = _descriptors(n, g)
    span = torch.tensor([1920.0, 1080.0, 10.0, 0.09, 6.28], device="cuda")
    base = torch.tensor([0.0, 0.0, 1.6, 0.01, 0.0], device="cuda")
    meta = torch.rand((n, 5), generator=g, device="cuda") * span + base
    rec = np.zeros(n, np.dtype([("m", "<f4", 5), ("c", "<u8", 2), ("q", "u1", 128)]))  # PSIFTCAT v1 records
    rec["m"] = meta.cpu().numpy()
    rec["c"] = _codes_of(d)
    rec["q"] = (d * 512.0).round().clamp_(0, 255).to(torch.uint8).cpu().numpy()
    raw = memoryview(rec.tobytes())
    parts = [b"PSIFTCAT", struct.pack("<IIIfBQ", 1, 4, 3, 0.015, 0, len(sizes))]
    for e, m in enumerate(sizes):
        name = b"img%05d" % e
        parts += [struct.pack("<I", len(name)) + name + struct.pack("<IIQ", 1920, 1080, m),
                  raw[int(off[e]) * 164:int(off[e + 1]) * 164]]
    ctx = psift.default_context()
    with tempfile.TemporaryDirectory() as tmp:
        path = os.path.join(tmp, "catalog.psiftcat")
        with open(path, "wb") as fh:
            fh.writelines(parts)
        cat = psift.DeviceCatalog.load_binary(path, ctx)
    # The query: views of three catalog images under similarities, the rest clutter.
    nq = case["nq"]
    qd = _descriptors(nq, g)
    qm = torch.rand((nq, 5), generator=g, device="cuda") * span + base
    at = 0
    for j, share in enumerate((1.0, 0.6, 0.3)):
        e = (seed * 37 + 101 * j) % len(sizes)
        k = min(int(share * sizes[e]), nq // 4)
        o = int(off[e])
        th, sc = 0.17 + 0.1 * j, 1.1 + 0.05 * j
        x, y = meta[o:o + k, 0], meta[o:o + k, 1]
        qd[at:at + k] = d[o:o + k] + 0.01 * torch.randn((k, 128), generator=g, device="cuda").abs_()
        qm[at:at + k, 0] = sc * (math.cos(th) * x - math.sin(th) * y) + 30.0
        qm[at:at + k, 1] = sc * (math.sin(th) * x + math.cos(th) * y) - 20.0
        qm[at:at + k, 2] = sc * meta[o:o + k, 2]
        qm[at:at + k, 4] = meta[o:o + k, 4] + th
        at += k
    qd /= qd.norm(dim=1, keepdim=True)
    m = qm.T.contiguous().cpu().numpy()
    return {"kind": "catalog_search", "cat": cat,
            "query": psift.Features(m[0], m[1], m[2], m[3], m[4], qd.cpu().numpy())}


def _run_catalog_search(s):
    top = psift.DEFAULT_CATALOG_TOP_K
    hits = s["cat"].search_features(s["query"], top)
    counts, tracking = np.zeros((top, 4), np.int64), np.zeros((top, 6), np.float32)
    transform, homography = np.zeros((top, 6), np.float32), np.zeros((top, 3, 3), np.float32)
    for i, h in enumerate(hits):
        t = h.tracking
        counts[i] = int(h.id[3:]), h.coarse_votes, t.raw_match_count, t.match_count
        tracking[i] = *t.mean_displacement, *t.median_displacement, t.mean_scale_ratio, t.inlier_ratio
        if h.transform is not None:
            transform[i] = h.transform
        if h.homography is not None:
            homography[i] = h.homography
    return {"counts": counts, "tracking": tracking, "transform": transform, "homography": homography}


def _prepare_catalog_topk(case, seed):
    g = _gen(seed)
    ncat, nq, k = case["ncat"], case["nq"], case["k"]
    cat = _descriptors(ncat, g)
    pick = torch.randint(0, ncat, (nq,), generator=g, device="cuda")
    q = cat[pick] + 0.02 * torch.randn((nq, 128), generator=g, device="cuda").abs_()
    q /= q.norm(dim=1, keepdim=True)
    codes = torch.empty((ncat, 2), dtype=torch.int64, device="cuda")
    ctx = psift.default_context()
    torch.cuda.synchronize()
    ctx.check(ctx.lib.psift_quantize_u128_dev(ctx.handle, cat.data_ptr(), ncat, codes.data_ptr()))
    ctx.synchronize()
    z = lambda t: torch.zeros((nq, k), dtype=t, device="cuda")  # noqa: E731
    return {"kind": "catalog_topk", "ctx": ctx, "cat": cat, "codes": codes, "q": q, "nq": nq, "ncat": ncat, "k": k,
            "qcodes": torch.zeros((nq, 2), dtype=torch.int64, device="cuda"),
            "idx": z(torch.int32), "dist": z(torch.int32), "ridx": z(torch.int32), "d2": z(torch.float32)}


def _run_catalog_topk(s):
    ctx, lib = s["ctx"], s["ctx"].lib
    ctx.check(lib.psift_quantize_u128_dev(ctx.handle, s["q"].data_ptr(), s["nq"], s["qcodes"].data_ptr()))
    ctx.check(lib.psift_hamming_topk_dev(ctx.handle, s["qcodes"].data_ptr(), s["nq"], s["codes"].data_ptr(),
                                         s["ncat"], s["k"], s["idx"].data_ptr(), s["dist"].data_ptr()))
    ctx.check(lib.psift_l2_rerank_dev(ctx.handle, s["q"].data_ptr(), s["nq"], s["cat"].data_ptr(),
                                      s["idx"].data_ptr(), s["k"], s["ridx"].data_ptr(), s["d2"].data_ptr()))
    return {"codes": s["qcodes"], "index": s["idx"], "distance": s["dist"], "ranked": s["ridx"], "d2": s["d2"]}


def _prepare_sampler(case, seed):
    n = case["n"]
    g = _gen(seed)
    inl = torch.rand(n, generator=g, device="cuda") < 0.6
    u = torch.rand((n, 6), generator=g, device="cuda")
    z = torch.randn((n, 2), generator=g, device="cuda")
    col = lambda a, b: torch.where(inl, a, b)  # noqa: E731
    x = torch.stack([col(0.2 + 0.6 * u[:, 0], 0.5 + 0.5 * u[:, 0]), col(0.08 * z[:, 0], 0.7 * z[:, 0]),
                     col(0.08 * z[:, 1], -math.pi + 2 * math.pi * u[:, 1]),
                     col(0.1 + 0.3 * u[:, 1], 0.25 + 0.35 * u[:, 1]), u[:, 2], u[:, 3], u[:, 4], u[:, 5]], dim=1)
    return {"kind": "sampler", "ctx": psift.default_context(), "n": n, "steps": case["steps"], "batch": case["batch"],
            "x": x.contiguous(), "y": inl.float(),
            "params": torch.from_numpy(psift.InlierMLP(seed=seed % 1000).params).cuda(),
            "losses": torch.zeros(case["steps"], device="cuda"), "prob": torch.zeros(n, device="cuda")}


def _run_sampler(s):
    ctx, lib = s["ctx"], s["ctx"].lib
    ctx.check(lib.psift_mlp_train_dev(ctx.handle, s["params"].data_ptr(), s["x"].data_ptr(), s["y"].data_ptr(),
                                      s["n"], s["steps"], s["batch"], 3e-3, 12, s["losses"].data_ptr()))
    ctx.check(lib.psift_mlp_infer_dev(ctx.handle, s["params"].data_ptr(), s["x"].data_ptr(), s["n"],
                                      s["prob"].data_ptr()))
    return {"params": s["params"], "losses": s["losses"], "prob": s["prob"]}


# ---------------------------------------------------------------- work

def _detect_work(h, w, case, in_bytes):
    """The separable blurs' taps over the scale space (two passes, a multiply and an add per tap), and
    the image in and the features out once (blob images give about 0.75 features per 1000 pixels)."""
    s = case["scales"]
    k = 2.0 ** (1.0 / s)
    radius = lambda sigma: math.ceil(3.0 * sigma)  # noqa: E731
    sig = [1.6 * math.sqrt(k ** (2 * i) - k ** (2 * i - 2)) for i in range(1, s + 3)]
    oh, ow = (2 * h, 2 * w) if case["upsample"] else (h, w)
    flops = 4.0 * (2 * radius(1.25 if case["upsample"] else 1.52) + 1) * oh * ow
    for _ in range(case["octaves"]):
        if oh < 3 or ow < 3:
            break
        flops += sum(4.0 * (2 * radius(x) + 1) + 1.0 for x in sig) * oh * ow
        oh, ow = oh // 2, ow // 2
    feats = 7.5e-4 * h * w
    if case.get("max_features", 4096):
        feats = min(feats, case.get("max_features", 4096))
    return h * w * in_bytes + feats * FEATURE_BYTES, flops


def work(case):
    kind = case["kind"]
    if kind == "detect":
        b, f = _detect_work(case["height"], case["width"], case, 4 if case["f32"] else 1)
        return {"bytes": b, "flops": f}
    if kind == "detect_batch":
        per = [_detect_work(h, w, case, 1) for h, w in _image_shapes(case)]
        return {"bytes": sum(b for b, _ in per), "flops": sum(f for _, f in per)}
    if kind in ("pair", "match_batch"):
        sizes = [(case["nq"], case["nt"])] if kind == "pair" else _match_sizes(case)
        return {"bytes": sum((a + b) * (DESC_BYTES + 8) + a / 3 * MATCH_BYTES for a, b in sizes),
                "flops": sum(2.0 * 128 * a * b for a, b in sizes)}
    if kind in ("ransac_batch", "fundamental"):
        # hypotheses until a clean sample is 99 % likely, each scored against every match
        per, size = (20, 4) if kind == "ransac_batch" else (40, 8)
        sets = _set_sizes(case)
        hyp = [max(32.0, math.log(0.01) / math.log(1.0 - (1.0 - o) ** size)) for _, o in sets]
        return {"bytes": sum(m for m, _ in sets) * (MATCH_BYTES + 1.0),
                "flops": sum(per * m * t for (m, _), t in zip(sets, hyp))}
    if kind == "panorama":
        n, h, w = case["n"], case["height"], case["width"]
        b, f = _detect_work(h, w, {"scales": 3, "octaves": 4, "upsample": True}, 4)
        return {"bytes": n * b + 4.0 * h * (w + (n - 1) * w * (1 - case["overlap"])), "flops": n * f}
    if kind == "catalog_search":
        # the codes and the query read once, a popcount test of the code pairs that share a byte
        n = sum(_entry_sizes(case))
        return {"bytes": 16.0 * n + case["nq"] * (FEATURE_BYTES + 16), "flops": 12.0 * case["nq"] * n / 16}
    if kind == "catalog_topk":
        ncat, nq, k = case["ncat"], case["nq"], case["k"]
        return {"bytes": 16.0 * ncat + nq * (DESC_BYTES + 16) + nq * k * (DESC_BYTES + 16.0),
                "flops": 2.0 * 128 * nq * ncat + 3.0 * 128 * nq * k}
    per = 2.0 * (8 * 64 + 64 * 64 + 64)
    return {"bytes": case["n"] * 40.0 + case["steps"] * case["batch"] * 36.0,
            "flops": per * (3.0 * case["steps"] * case["batch"] + case["n"])}


# ---------------------------------------------------------------- 64-bit values

def exact(case, seed):
    """The 64-bit values of the outputs that are plain functions of the inputs: the match records and
    the re-ranked distances.  The others have none: which keypoints, samples and minibatches enter is
    decided by the 32-bit arithmetic itself, step by step."""
    kind = case["kind"]
    if kind == "pair":
        s = _prepare_pair(case, seed)
        rec = _exact_matches(*(torch.from_numpy(s[k]).cuda() for k in ("q", "t", "qxy", "txy")), case)
        out = torch.zeros((case["nq"], 8), dtype=torch.float64)
        out[:rec.shape[0]] = rec.cpu()
        return {"counts": None, "index": None, "values": out, "inliers": None, "homography": None}
    if kind == "match_batch":
        s = _prepare_match_batch(case, seed)
        out = torch.zeros((len(s["keep"]), s["out"]["index"].shape[1], 8), dtype=torch.float64)
        for i, (q, t, qxy, txy) in enumerate(s["keep"]):
            rec = _exact_matches(q, t, qxy, txy, case)
            out[i, :rec.shape[0]] = rec.cpu()
        return {"counts": None, "index": None, "values": out}
    if kind == "catalog_topk":
        s = _prepare_catalog_topk(case, seed)
        return {"codes": None, "index": None, "distance": None, "ranked": None, "d2": _exact_topk_d2(s)}
    return None


def _exact_matches(q, t, qxy, txy, case):
    q, t, qxy, txy = (x.double() for x in (q, t, qxy, txy))
    d2 = ((q * q).sum(1)[:, None] + (t * t).sum(1)[None] - 2.0 * (q @ t.T)).clamp_(min=0.0)
    best, idx = torch.topk(d2, 2, dim=1, largest=False)
    d = best.sqrt()
    ratio = d[:, 0] / d[:, 1]
    keep = (ratio < float(np.float32(case["ratio"]))) & (best[:, 1] > 1e-12)
    if case["mutual"]:
        keep &= d2.argmin(dim=0)[idx[:, 0]] == torch.arange(q.shape[0], device=q.device)
    a, b = qxy[keep], txy[idx[keep, 0]]
    return torch.cat([a, b, d[keep, :1], ratio[keep, None], b - a], dim=1)


def _exact_topk_d2(s):
    k = s["k"]
    signs = lambda d: torch.where(d > 0.065, 1.0, -1.0).to(torch.float16)  # noqa: E731
    cat = signs(s["cat"])
    index = torch.arange(s["ncat"], device="cuda", dtype=torch.int32)
    out = []
    for i in range(0, s["nq"], 64):
        q = s["q"][i:i + 64]
        dist = ((128 - (signs(q) @ cat.T).int()) // 2) * (1 << 22) + index  # (distance, index) order
        pick = torch.topk(dist, k, dim=1, largest=False).values & ((1 << 22) - 1)
        d2 = ((q.double()[:, None] - s["cat"][pick.long()].double()) ** 2).sum(2)
        out.append(d2.sort(dim=1).values)
    return torch.cat(out).cpu()


_PREPARE = {"detect": _prepare_detect, "detect_batch": _prepare_detect_batch, "pair": _prepare_pair,
            "match_batch": _prepare_match_batch, "ransac_batch": _prepare_ransac_batch,
            "fundamental": _prepare_fundamental, "panorama": _prepare_panorama,
            "catalog_search": _prepare_catalog_search, "catalog_topk": _prepare_catalog_topk,
            "sampler": _prepare_sampler}
_RUN = {"detect": _run_detect, "detect_batch": _run_detect_batch, "pair": _run_pair,
        "match_batch": _run_match_batch, "ransac_batch": _run_ransac_batch, "fundamental": _run_fundamental,
        "panorama": _run_panorama, "catalog_search": _run_catalog_search, "catalog_topk": _run_catalog_topk,
        "sampler": _run_sampler}
