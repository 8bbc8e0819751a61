"""The work this library does for its users, as cases that can be timed.

Each case is one kind of call with its sizes: a frame or several passes of
the path tracer, a batch of views, the reference-parity frame, a photon-map
or photon-beam pass, training and rendering with the radiance cache, the
radix sort, and the upload of a cloud.  `listed()` gives the fixed ones,
`draw(rng)` more of the same ranges, `prepare` what a program holds before
the call, `run` the call, `work` its indispensable bytes and operations and
`exact` its result in 64 bits where there is one.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (os.path.join(_ROOT, "cloudrendering-vulkan_gb300"), _ROOT):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import vcr  # noqa: E402
from vcr import configs  # noqa: E402

PRECISIONS = {"fp32": vcr.PREC_FP32, "fp16": vcr.PREC_FP16, "bf16": vcr.PREC_BF16}
TEXEL_BYTES = {"fp32": 4, "fp16": 2, "bf16": 2}
LOOKUPS_PER_PATH = 6.5   # density lookups of a camera path (the 1024x512x1024 cloud's mean)
FLOPS_PER_LOOKUP = 60    # trilinear filter, collision test and free flight
CACHE_FLOPS = 2 * (5 * 64 * 64 + 64 * 3)  # one forward of the cache network


def listed():
    return [
        # A thumbnail of a small cloud: the smallest frame, all latency and launches.
        {"name": "pt-thumbnail", "kind": "frame", "nx": 64, "ny": 64, "nz": 64, "precision": "fp32", "sigma": 8.0,
         "octaves": 5, "width": 64, "height": 64, "spp": 1, "level": 2, "steps": 4},
        # An interactive frame after a camera move on the 128^3 cloud: clear, one pass, display image.
        {"name": "pt-frame", "kind": "frame", "nx": 128, "ny": 128, "nz": 128, "precision": "fp32", "sigma": 8.0,
         "octaves": 6, "width": 512, "height": 512, "spp": 1, "level": 2, "steps": 4},
        # Final-quality rendering of the large cloud: consecutive passes in one launch at full HD.
        {"name": "pt-passes", "kind": "passes", "nx": 1024, "ny": 512, "nz": 1024, "precision": "fp16",
         "sigma": 32.0, "octaves": 8, "width": 1920, "height": 1080, "spp": 1, "passes": 8, "level": 3, "steps": 8},
        # Many cameras of uneven frames and sun directions in one launch (image-set rendering).
        {"name": "batch-views", "kind": "batch", "nx": 512, "ny": 512, "nz": 512, "precision": "bf16",
         "sigma": 16.0, "octaves": 6, "views": 12, "side_lo": 256, "side_hi": 1024, "spp": 4, "level": 2,
         "steps": 16},
        # The reference's own estimator: shadow volume for a new sun, then a parity frame at its window size.
        {"name": "parity-frame", "kind": "parity", "nx": 256, "ny": 256, "nz": 256, "precision": "fp32",
         "sigma": 16.0, "width": 800, "height": 600, "sv": 128},
        # One progressive photon-mapping pass (a million photons).
        {"name": "ppm-pass", "kind": "ppm", "nx": 256, "ny": 256, "nz": 256, "precision": "fp32", "sigma": 16.0,
         "octaves": 6, "width": 960, "height": 540, "photons": 1 << 20, "radius": 0.01},
        # One progressive photon-beam pass (about 262,144 beams): the longest single call.
        {"name": "ppb-pass", "kind": "ppb", "nx": 256, "ny": 256, "nz": 256, "precision": "fp32", "sigma": 16.0,
         "octaves": 6, "width": 1280, "height": 720, "photons": 60741, "radius": 0.015},
        # Training the radiance cache on records in hand (forward, backward, Adam).
        {"name": "cache-fit", "kind": "fit", "records": 65536, "steps": 8},
        # One online frame of the cached tracker: training paths, camera paths, cache queries, update.
        {"name": "cache-frame", "kind": "cached", "nx": 1024, "ny": 512, "nz": 1024, "precision": "fp16",
         "sigma": 32.0, "octaves": 8, "width": 1920, "height": 1080, "spp": 2, "train": 65536, "level": 3,
         "steps": 8},
        # Sorting a large set of 32-bit keys with their indices.
        {"name": "sort-large", "kind": "sort", "n": 1 << 26, "bits": 32},
        # Ordering the 30-bit Morton codes of a small scene: a few thousand keys.
        {"name": "sort-small", "kind": "sort", "n": 3001, "bits": 30},
        # Binding a cloud from host memory (a frame of an animated cloud) and reading densities from it.
        {"name": "grid-upload", "kind": "upload", "nx": 256, "ny": 256, "nz": 256, "precision": "fp16",
         "points": 1 << 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "passes", "batch", "parity", "ppm", "ppb", "fit", "cached", "sort", "upload"])
    prec = rng.choice(["fp32", "fp16", "bf16"])
    side = _log(rng, 40, 320)
    grid = {"nx": side, "ny": max(24, int(side * rng.uniform(0.5, 1.0))), "nz": side, "precision": prec,
            "sigma": rng.choice([8.0, 16.0, 32.0]), "octaves": rng.randint(4, 8)}
    width = _log(rng, 48, 1920)
    frame = {"width": width, "height": max(32, int(width * rng.uniform(0.5, 1.0)))}
    tuned = {"level": rng.randint(1, 3), "steps": rng.choice([4, 8, 16])}
    if kind == "frame":
        return {"kind": kind, **grid, **frame, "spp": rng.choice([1, 1, 2]), **tuned}
    if kind == "passes":
        return {"kind": kind, **grid, **frame, "spp": rng.choice([1, 2]), "passes": rng.randint(2, 8), **tuned}
    if kind == "batch":
        return {"kind": kind, **grid, "views": rng.randint(1, 12), "side_lo": 64, "side_hi": _log(rng, 128, 1024),
                "spp": rng.randint(1, 4), **tuned}
    if kind == "parity":
        del grid["octaves"]
        return {"kind": kind, **grid, "width": _log(rng, 64, 800), "height": _log(rng, 64, 600),
                "sv": rng.randint(32, 128)}
    if kind == "ppm":
        return {"kind": kind, **grid, "width": _log(rng, 64, 960), "height": _log(rng, 64, 540),
                "photons": _log(rng, 1 << 12, 1 << 20), "radius": rng.uniform(0.008, 0.02)}
    if kind == "ppb":
        return {"kind": kind, **grid, "width": _log(rng, 64, 960), "height": _log(rng, 64, 540),
                "photons": _log(rng, 300, 30000), "radius": rng.uniform(0.015, 0.03)}
    if kind == "fit":
        return {"kind": kind, "records": _log(rng, 1000, 131072), "steps": rng.randint(1, 8)}
    if kind == "cached":
        return {"kind": kind, **grid, **frame, "spp": rng.choice([1, 2]), "train": _log(rng, 4096, 65536), **tuned}
    if kind == "sort":
        return {"kind": kind, "n": _log(rng, 100, 1 << 26), "bits": rng.choice([24, 30, 32])}
    del grid["sigma"], grid["octaves"]
    return {"kind": kind, **grid, "points": _log(rng, 1 << 12, 1 << 20)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _size(case):
    return case["nx"], case["ny"], case["nz"]


def _scene(case, name="case", **kw):
    return configs.Scene(name, _size(case), case.get("octaves", 6), case["sigma"], case.get("width", 64),
                         case.get("height", 64), 1, precision=PRECISIONS[case["precision"]], **kw)


def _values(case, seed):
    """Cloud densities [Z, Y, X] on the GPU: value-noise octaves under a spherical falloff, clamped to [0, 1]."""
    nx, ny, nz = _size(case)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    v = torch.zeros((nz, ny, nx), device="cuda")
    amp, cells = 0.5, 4
    for _ in range(5):
        lattice = torch.rand((1, 1, cells + 1, cells + 1, cells + 1), device="cuda", generator=gen)
        v += amp * torch.nn.functional.interpolate(lattice, size=(nz, ny, nx), mode="trilinear",
                                                   align_corners=True)[0, 0]
        amp, cells = amp / 2, cells * 2
    ax = [torch.linspace(-1, 1, n, device="cuda") for n in (nz, ny, nx)]
    r = (ax[0][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[2][None, None, :] ** 2).sqrt()
    return ((v - 0.35) * 2.0 * (1.0 - r)).clamp(0.0, 1.0)


def _desc(case):
    n = max(_size(case))
    return vcr.grid_desc(_size(case), (1.0 / n,) * 3)


def _context(case, seed):
    """A context with the case's cloud (seeded), camera, parameters, frame and tuning bound."""
    sc = _scene(case, seed=seed % 100003 + 1)
    ctx = vcr.Context()
    if "level" in case:
        ctx.set_tuning(majorant_level=case["level"], dda_steps=case["steps"])
    configs.setup_context(ctx, sc)
    return ctx, sc


def _records(case, seed):
    """Cache records in the unit cloud box: positions, unit directions, sun, positive heavy-tailed targets."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 17)
    n = case["records"]
    r = torch.zeros((n, 16), device="cuda")
    r[:, 0:3] = torch.rand((n, 3), device="cuda", generator=gen) - torch.tensor([0.5, 0.5, 0.0], device="cuda")
    d = torch.randn((n, 3), device="cuda", generator=gen)
    r[:, 3:6] = d / d.norm(dim=1, keepdim=True)
    r[:, 6:9] = torch.tensor(configs.sun_travel_dir(), device="cuda")
    smooth = 0.1 + 0.4 * (1.0 + torch.sin(4.0 * r[:, 0:1] + 3.0 * r[:, 1:2])) * r[:, 2:3]
    r[:, 9:12] = smooth * torch.exp(0.8 * torch.randn((n, 3), device="cuda", generator=gen))
    return r


def _weights(seed):
    """Initial cache weights (uniform, fan-in scaled; the output layer's padding columns zero)."""
    rng = np.random.default_rng(seed)
    hidden = rng.uniform(-1, 1, (5, 64, 64)) * math.sqrt(6.0 / 64)
    out = np.zeros((64, 16))
    out[:, :3] = rng.uniform(-1, 1, (64, 3)) * math.sqrt(1.0 / 64)
    return np.concatenate([hidden.ravel(), out.ravel()]).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "seed": seed % 65521 + 1, "pass": 0}
    if kind in ("frame", "passes", "ppm", "ppb", "cached"):
        ctx, sc = _context(case, seed)
        px = sc.width * sc.height
        st.update(ctx=ctx, sum=torch.empty((sc.height, sc.width, 3), dtype=torch.float64, device="cuda"))
        if kind == "frame":
            st["rgba"] = torch.empty((sc.height, sc.width, 4), dtype=torch.uint8, device="cuda")
        elif kind == "ppm":
            ctx.ppm_setup(case["photons"], 8 * case["photons"], case["radius"], 0.7)
        elif kind == "ppb":
            ctx.ppb_setup(case["photons"], max(1 << 16, 276 * case["photons"]), case["radius"], 0.8)
        elif kind == "cached":
            prm = sc.params()
            prm.nrc_events = 2
            ctx.set_params(prm)
            ctx.nrc_setup(train_samples=case["train"], query_capacity=px * case["spp"], ema_decay=0.99,
                          seed=st["seed"])
            ctx.nrc_train_step(seed=st["seed"] + 5, pass_index=0)  # finds the path count of a training set
            ctx.nrc_set_weights(_weights(seed))
        ctx.synchronize()
    elif kind == "batch":
        ctx, sc = _context(case, seed)
        rng = np.random.default_rng(seed)
        views = []
        for v in range(case["views"]):
            a = 2.0 * math.pi * (v + rng.random()) / case["views"]
            pos = (1.4 * math.sin(a), 0.25, 0.5 - 1.4 * math.cos(a))
            fwd = (-pos[0], -pos[1], 0.5 - pos[2])
            # uneven sides, spread evenly over the range so that every seed asks for the same pixels
            s = int(round(case["side_lo"] + (case["side_hi"] - case["side_lo"]) * (v + 0.5) / case["views"]))
            views.append((vcr.camera_look(pos, fwd, 60.0, 0.1, s, s), s, s,
                          configs.sun_travel_dir(configs.C4_ELEVATIONS[v % 8])))
        ctx.batch_setup(views)
        st.update(ctx=ctx, images=[torch.empty((h, w, 3), dtype=torch.float64, device="cuda")
                                   for _, w, h, _ in views])
        ctx.synchronize()
    elif kind == "parity":
        w, h = case["width"], case["height"]
        ctx = vcr.Context()
        cloud = vcr.cloud_from_grid(_desc(case), 1.0, case["sigma"])
        ctx.grid_upload(_desc(case), _values(case, seed).cpu().numpy(), PRECISIONS[case["precision"]])
        ctx.set_cloud(cloud)
        ctx.set_camera(vcr.camera_look((0.0, 0.0, -0.4), (0.0, 0.0, 1.0), 90.0, 0.1, w, h))
        prm = _scene(case).params(vcr.TRACKER_GLOBAL)
        prm.albedo, prm.max_events = 1.0, 0
        prm.rng_mode, prm.nee_mode, prm.sky_mode = vcr.RNG_XORSHIFT, vcr.NEE_SHADOW_VOLUME, vcr.SKY_GRADIENT
        ctx.set_params(prm)
        ctx.set_frame(w, h)
        n = case["sv"]
        st.update(ctx=ctx, sv=vcr.shadow_volume_setup(_parity_sun(seed), cloud.bounds_min, cloud.bounds_max, n),
                  sum=torch.empty((h, w, 3), dtype=torch.float64, device="cuda"),
                  volume=torch.empty((n, n, n), device="cuda"))
        ctx.synchronize()
    elif kind == "fit":
        ctx = vcr.Context()
        ctx.set_cloud(_unit_cloud())
        ctx.nrc_setup(train_samples=max(case["records"], 1024), learning_rate=1e-3, query_capacity=1024,
                      seed=st["seed"], ema_decay=0.99)
        ctx.nrc_set_weights(_weights(seed))
        st.update(ctx=ctx, records=_records(case, seed))
    elif kind == "sort":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        n, bits = case["n"], case["bits"]
        keys = torch.randint(0, 1 << bits, (n,), dtype=torch.int64, device="cuda", generator=gen)
        keys = torch.where(keys >= 1 << 31, keys - (1 << 32), keys).to(torch.int32)  # the 32 bits of a uint32
        st.update(ctx=vcr.Context(), keys=keys, vals=torch.randperm(n, device="cuda", generator=gen).to(torch.int32),
                  keys_out=torch.empty_like(keys), vals_out=torch.empty_like(keys))
    elif kind == "upload":
        dense = _values(case, seed).cpu().pin_memory()
        cloud = vcr.cloud_from_grid(_desc(case), 1.0, 16.0)
        st.update(ctx=vcr.Context(), host=dense, dense=dense.numpy(), desc=_desc(case), cloud=cloud,
                  points=_points(case, seed), rho=torch.empty(case["points"], device="cuda"))
    else:
        raise ValueError(kind)
    return st


def _unit_cloud():
    c = vcr.cloud_from_grid(vcr.grid_desc((64, 64, 64), (1 / 64,) * 3), 1.0, 16.0)
    c.max_extinction = 1.0
    return c


def _parity_sun(seed):
    return configs.sun_travel_dir(20.0 + seed % 50, 90.0 + seed % 180)


def _points(case, seed):
    """Positions in the cloud's box (a unit along its longest axis), as floats."""
    nx, ny, nz = _size(case)
    n = max(nx, ny, nz)
    gen = torch.Generator(device="cuda").manual_seed(seed + 3)
    ext = torch.tensor([nx / n, ny / n, nz / n], device="cuda")
    return (torch.rand((case["points"], 3), device="cuda", generator=gen) - torch.tensor([0.5, 0.5, 0.0], device="cuda")) * ext


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def run(st):
    case, ctx, kind = st["case"], st["ctx"], st["case"]["kind"]
    seed, k = st["seed"], st["pass"]
    if kind == "frame":  # the camera moved: clear, one pass, the image to show and the sums
        ctx.reset()
        ctx.pt_pass(seed=seed, pass_index=0, spp=case["spp"])
        ctx.display_to(st["rgba"].data_ptr())
        ctx.readback_to(vcr.BUF_IMAGE_SUM, st["sum"].data_ptr(), st["sum"].nbytes)
        return st["rgba"], st["sum"]
    if kind == "passes":
        ctx.reset()
        ctx.pt_passes(seed=seed, first=0, count=case["passes"], spp=case["spp"])
        ctx.readback_to(vcr.BUF_IMAGE_SUM, st["sum"].data_ptr(), st["sum"].nbytes)
        return st["sum"]
    if kind == "batch":
        ctx.batch_reset()
        ctx.batch_pass(seed=seed, pass_index=0, spp=case["spp"])
        for v, image in enumerate(st["images"]):
            vcr.check(vcr.lib().vcr_batch_read(ctx.h, v, ctypes.c_void_p(image.data_ptr()), image.nbytes), ctx.h)
        return st["images"]
    if kind == "parity":
        ctx.shadow_volume_build(st["sv"])
        ctx.reset()
        ctx.pt_pass(seed=seed, pass_index=0)
        ctx.readback_to(vcr.BUF_IMAGE_SUM, st["sum"].data_ptr(), st["sum"].nbytes)
        ctx.readback_to(vcr.BUF_SHADOW_VOLUME, st["volume"].data_ptr(), st["volume"].nbytes)
        return st["sum"], st["volume"]
    if kind == "ppm":  # progressive: the statistics go on from pass to pass
        ctx.ppm_pass(seed=seed, pass_index=k)
        st["pass"] = k + 1
        ctx.readback_to(vcr.BUF_IMAGE_SUM, st["sum"].data_ptr(), st["sum"].nbytes)
        return st["sum"]
    if kind == "ppb":
        ctx.reset()
        ctx.ppb_pass(seed=seed, pass_index=0)
        ctx.readback_to(vcr.BUF_IMAGE_SUM, st["sum"].data_ptr(), st["sum"].nbytes)
        return st["sum"]
    if kind == "fit":
        ctx.nrc_fit(st["records"].data_ptr(), case["records"], case["steps"])
        return ctx.nrc_get_weights()
    if kind == "cached":
        ctx.reset()
        ctx.nrc_frame(seed=seed, pass_index=0, spp=case["spp"])
        ctx.readback_to(vcr.BUF_IMAGE_SUM, st["sum"].data_ptr(), st["sum"].nbytes)
        return st["sum"], ctx.nrc_get_weights()
    if kind == "sort":
        ctx.radix_sort_pairs(st["keys"].data_ptr(), st["vals"].data_ptr(), st["keys_out"].data_ptr(),
                             st["vals_out"].data_ptr(), case["n"], 0, case["bits"])
        return st["keys_out"], st["vals_out"]
    # upload
    ctx.grid_upload(st["desc"], st["dense"], PRECISIONS[case["precision"]])
    ctx.set_cloud(st["cloud"])
    ctx.grid_sample(st["points"].data_ptr(), st["rho"].data_ptr(), case["points"])
    return st["rho"], ctx.majorants(0)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "sort":  # pairs read once, written once
        return {"bytes": 16.0 * case["n"], "flops": 0.0}
    if kind == "fit":  # records read, weights and moments read and written each step
        return {"bytes": float(case["steps"] * (64 * case["records"] + 6 * 4 * 21504)),
                "flops": 3.0 * CACHE_FLOPS * case["records"] * case["steps"]}
    cells = case["nx"] * case["ny"] * case["nz"]
    grid = cells * TEXEL_BYTES[case["precision"]]
    if kind == "upload":  # the dense grid over the link and into memory, the stored grid and the samples out
        return {"bytes": float(cells * 4 + grid + 16 * case["points"]),
                "flops": float(cells + FLOPS_PER_LOOKUP * case["points"])}
    if kind == "batch":
        n = case["views"]
        px = sum(int(round(case["side_lo"] + (case["side_hi"] - case["side_lo"]) * (v + 0.5) / n)) ** 2
                 for v in range(n))
    else:
        px = case["width"] * case["height"]
    paths = px * case.get("spp", 1) * case.get("passes", 1)
    lookups = LOOKUPS_PER_PATH * paths
    flops = FLOPS_PER_LOOKUP * lookups
    out = 24.0 * px
    if kind == "parity":  # lookups of a column march, a sphere-traced frame and its volume
        lookups += case["sv"] ** 3
        flops = FLOPS_PER_LOOKUP * lookups
        out += 4.0 * case["sv"] ** 3
    elif kind == "ppm":  # emission, photons ordered and stored, one gather a pixel
        stored = 3.3 * case["photons"]
        lookups = 10.0 * case["photons"] + 4.0 * px
        flops = FLOPS_PER_LOOKUP * lookups
        out += stored * (48 + 2 * 16) + 64.0 * px
    elif kind == "ppb":  # beams with 16 transmittance samples, segments ordered, pairs of rays and segments
        beams = 4.3 * case["photons"]
        segs = beams * 0.58 / case["radius"]
        lookups = 17 * 5.0 * beams
        flops = FLOPS_PER_LOOKUP * lookups + 60.0 * px * segs * 2.75 * case["radius"] ** 2
        out += segs * (36 + 2 * 16 + 64)
    elif kind == "cached":
        lookups = 4.0 * paths + 20.0 * case["train"]
        flops = FLOPS_PER_LOOKUP * lookups + CACHE_FLOPS * (0.13 * paths + 3 * case["train"])
        out += 64.0 * (0.13 * paths + case["train"])
    return {"bytes": float(out + min(grid, 16.0 * lookups)), "flops": float(flops)}


# ---------------------------------------------------------------------------
# results in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "fit":
        return _exact_fit(case, seed)
    if kind == "upload":
        dense = _values(case, seed).double()
        rho = _trilinear64(dense, _points(case, seed).double(), _bounds64(case))
        nz, ny, nx = dense.shape
        up = [(-n) % 8 for n in (nx, ny, nz)]
        halo = torch.nn.functional.pad(dense[None, None], (1, up[0] + 1, 1, up[1] + 1, 1, up[2] + 1))
        maj = torch.nn.functional.max_pool3d(halo, 10, 8)[0, 0]
        return rho, maj.reshape(-1).cpu().numpy()
    if kind == "parity":
        return None, _exact_shadow_volume(case, seed)
    return None


def _bounds64(case):
    nx, ny, nz = _size(case)
    n = max(nx, ny, nz)
    b0 = torch.tensor([-0.5 * nx / n, -0.5 * ny / n, 0.0], dtype=torch.float64, device="cuda")
    return b0, torch.tensor([0.5 * nx / n, 0.5 * ny / n, nz / n], dtype=torch.float64, device="cuda")


def _trilinear64(dense, pos, bounds):
    """Clamp-to-edge trilinear filter with texel centres at (i + 1/2) / N."""
    b0, b1 = bounds
    grid = (2.0 * (pos - b0) / (b1 - b0) - 1.0).reshape(1, 1, 1, -1, 3)
    return torch.nn.functional.grid_sample(dense[None, None], grid, mode="bilinear", padding_mode="border",
                                           align_corners=False).reshape(-1)


def _exact_shadow_volume(case, seed):
    """exp(-(z + 1) voxel * mean extinction of the voxels up to z) along each light-aligned column."""
    n = case["sv"]
    d = np.array(_parity_sun(seed))
    d = d / np.linalg.norm(d)
    s = 1.0 if d[2] >= 0.0 else -1.0
    a = d[1] / (1.0 + abs(d[2]))
    b, c = d[1] * a, -d[0] * a
    right, up = np.array([d[2] + s * b, s * c, -d[0]]), np.array([c, 1.0 - b, -s * d[1]])
    b0, b1 = _bounds64(case)
    lo, hi = b0.cpu().numpy(), b1.cpu().numpy()
    radius = np.linalg.norm(hi - lo) / 2.0
    voxel = 2.0 * radius / (n - 1)
    origin = (lo + hi) / 2.0 + radius * (-d - right - up)
    t = lambda v: torch.tensor(v, dtype=torch.float64, device="cuda")  # noqa: E731
    i = torch.arange(n, dtype=torch.float64, device="cuda") * voxel
    dense = _values(case, seed).double()
    acc = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    out = torch.empty((n, n, n), dtype=torch.float64, device="cuda")
    plane = t(origin) + i[None, :, None] * t(right) + i[:, None, None] * t(up)
    for z in range(n):
        p = plane + z * voxel * t(d)
        inside = ((p >= b0) & (p <= b1)).all(dim=-1)
        rho = _trilinear64(dense, p.reshape(-1, 3), (b0, b1)).reshape(n, n)
        acc = acc + torch.where(inside, rho * case["sigma"], torch.zeros_like(rho))
        out[z] = torch.exp(-voxel * acc)
    return out


def _harmonics(v):
    """Real spherical harmonics of bands 0 .. 3 of unit vectors [n, 3]."""
    x, y, z = v[:, 0], v[:, 1], v[:, 2]
    xx, yy, zz = x * x, y * y, z * z
    c = [1 / math.sqrt(4 * math.pi), math.sqrt(3 / (4 * math.pi)), math.sqrt(15 / (4 * math.pi)),
         math.sqrt(5 / (16 * math.pi)), math.sqrt(35 / (32 * math.pi)), math.sqrt(105 / (4 * math.pi)),
         math.sqrt(21 / (32 * math.pi)), math.sqrt(7 / (16 * math.pi))]
    return torch.stack([
        torch.full_like(x, c[0]), -c[1] * y, c[1] * z, -c[1] * x,
        c[2] * x * y, -c[2] * y * z, c[3] * (3 * zz - 1), -c[2] * x * z, c[2] / 2 * (xx - yy),
        -c[4] * y * (3 * xx - yy), c[5] * x * y * z, -c[6] * y * (5 * zz - 1), c[7] * z * (5 * zz - 3),
        -c[6] * x * (5 * zz - 1), c[5] / 2 * z * (xx - yy), -c[4] * x * (xx - 3 * yy)], dim=1)


def _exact_fit(case, seed):
    """The network's training steps in 64 bits: encoding, five ReLU layers, relative L2 loss, Adam."""
    r = _records(case, seed).double()
    n = case["records"]
    p = r[:, 0:3] + torch.tensor([0.5, 0.5, 0.0], dtype=torch.float64, device="cuda")
    cols = []
    for level in range(16):
        z = 1.0 - (2.0 * level + 1.0) / 16.0
        turn = 2.0 * math.pi * 0.61803398875 * level
        rad = math.sqrt(1.0 - z * z)
        phase = 2.0 * math.pi * 2.0 ** (level / 2) * (rad * math.cos(turn) * p[:, 0] + rad * math.sin(turn) * p[:, 1]
                                                      + z * p[:, 2])
        cols += [torch.sin(phase), torch.cos(phase)]
    x0 = torch.cat([torch.stack(cols, dim=1), _harmonics(r[:, 3:6]), _harmonics(r[:, 6:9])], dim=1)
    w = torch.from_numpy(_weights(seed)).double().to("cuda")
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    shapes = [(64, 64)] * 5 + [(64, 16)]
    for step in range(1, case["steps"] + 1):
        layers = [t.reshape(s) for t, s in zip(torch.split(w, [a * b for a, b in shapes]), shapes)]
        xs = [x0]
        for layer in layers[:5]:
            xs.append((xs[-1] @ layer).clamp(min=0.0))
        y = (xs[-1] @ layers[5])[:, :3]
        dy = torch.zeros((n, 16), dtype=torch.float64, device="cuda")
        dy[:, :3] = 2.0 * (y - r[:, 9:12]) / (y * y + 0.01) / (3.0 * n)
        grads = []
        for layer in range(5, -1, -1):
            grads.append((xs[layer].T @ dy).reshape(-1))
            dy = (dy @ layers[layer].T) * (xs[layer] > 0)
        g = torch.cat(grads[::-1])
        m, v = 0.9 * m + 0.1 * g, 0.99 * v + 0.01 * g * g
        w = w - 1e-3 * (m / (1 - 0.9 ** step)) / ((v / (1 - 0.99 ** step)).sqrt() + 1e-8)
    return w.cpu().numpy()
