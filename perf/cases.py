"""The calls a user of the engine makes, as cases that can be timed and compared.

A case is a dict of plain values; `prepare` makes what a program has in hand before the
call (phantoms and inputs are made on the GPU from the seed), `run` makes the call through
the package's public entry points, `work` says what the call cannot do without, `exact`
gives the result in 64 bits where plain torch or numpy can.  Kinds of case:

  exposure   one beam on one built world, dose read back: GpuWorld.clear / run, then the
             dose, variance and event counts into pinned host or device memory
  patient    the same for a new patient: the voxel arrays handed over and the world built
             before the run, as the simulation worker does for every job
  batch      several small jobs in one Batch.run, each world's dose read into device memory
  forward    Denoiser.forward on prepared input channels
  train      Denoiser.train_step (loss, every gradient) on a batch of cubic patches
  denoise    a short run's dose through the trained network, into pinned host memory
  segment    CT numbers to material and density
"""
from __future__ import annotations

import ctypes as C
import math
import random
from pathlib import Path

import numpy as np
import torch

from opendxmc_gb300 import engine as G
from opendxmc_gb300 import native as N
from opendxmc_gb300 import phantoms as P

CHANNELS = (16, 32, 64, 128)
WEIGHTS = Path(G.__file__).parent / "weights" / "denoiser_torso_spiral.npy"


def listed() -> list[dict]:
    return [
        # a preview of a radiograph: the smallest call, bound by latency (1e5 histories)
        {"name": "dx_preview", "kind": "exposure", "phantom": "cylinder", "nx": 128, "ny": 128, "nz": 64,
         "sx": 0.1, "sy": 0.1, "sz": 0.25, "beam": "dx", "kvp": 70.0, "histories": 100_000, "correction": 1,
         "dose_to": "host"},
        # the small plain Monte Carlo job: 1e7 histories of a radiograph of the water cylinder
        {"name": "dx_exam", "kind": "exposure", "phantom": "cylinder", "nx": 128, "ny": 128, "nz": 64,
         "sx": 0.1, "sy": 0.1, "sz": 0.25, "beam": "dx", "kvp": 70.0, "histories": 10_000_000, "correction": 1,
         "dose_to": "host"},
        # spiral CT on the 256 x 256 x 200 torso, the benchmark's job with fewer histories
        {"name": "ct_torso", "kind": "exposure", "phantom": "torso", "nx": 256, "ny": 256, "nz": 200,
         "sx": 0.15, "sy": 0.15, "sz": 0.15, "beam": "spiral", "kvp": 120.0, "histories": 200_000_000,
         "correction": 1, "dose_to": "host"},
        # spiral CT at full size, 512 x 512 x 400; the dose stays on the device
        {"name": "ct_torso_full", "kind": "exposure", "phantom": "torso", "nx": 512, "ny": 512, "nz": 400,
         "sx": 0.08, "sy": 0.08, "sz": 0.1, "beam": "spiral_wide", "kvp": 120.0, "histories": 300_000_000,
         "correction": 1, "dose_to": "device"},
        # cone-beam CT of an odd-sized body with bound-electron Compton and fluorescence
        {"name": "cbct_bound", "kind": "exposure", "phantom": "body", "nx": 189, "ny": 117, "nz": 81,
         "sx": 0.2, "sy": 0.21, "sz": 0.27, "beam": "cbct", "kvp": 90.0, "histories": 10_000_000, "correction": 2,
         "dose_to": "host"},
        # a worker's job on a new patient: arrays in (FP64 densities), build, run, dose out
        {"name": "ct_patient", "kind": "patient", "phantom": "torso", "nx": 256, "ny": 256, "nz": 200,
         "sx": 0.15, "sy": 0.15, "sz": 0.15, "beam": "spiral", "kvp": 120.0, "histories": 30_000_000,
         "correction": 1, "dose_to": "host"},
        # a sweep of small exposures of small phantoms of uneven size in one launch
        {"name": "batch_small", "kind": "batch", "jobs": 8, "dim_lo": 64, "dim_hi": 128, "hist_lo": 100_000,
         "hist_hi": 2_000_000},
        # the network on one training-size patch: latency and launches
        {"name": "net_patch", "kind": "forward", "b": 1, "d": 64, "h": 64, "w": 64},
        # the network on a volume whose edges fill no whole brick
        {"name": "net_volume", "kind": "forward", "b": 1, "d": 200, "h": 264, "w": 232},
        # one training step as configured: 8 patches of 64^3, forward and backward
        {"name": "net_train", "kind": "train", "b": 8, "p": 64},
        # a short CT run's dose map denoised, scale from the map itself, and read back
        {"name": "denoise_torso", "kind": "denoise", "phantom": "torso", "nx": 256, "ny": 256, "nz": 200,
         "sx": 0.15, "sy": 0.15, "sz": 0.15},
        # a CT series to material and density
        {"name": "segment_ct", "kind": "segment", "n": 256 * 256 * 100},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _spacing(rng):
    return {k: round(rng.uniform(0.08, 0.3), 3) for k in ("sx", "sy", "sz")}


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["exposure", "exposure", "exposure", "patient", "batch", "forward", "forward", "train",
                       "denoise", "segment"])
    if kind == "exposure":
        return {"kind": kind, "phantom": rng.choice(["torso", "body", "cylinder"]), "nx": int(_log(rng, 64, 320)),
                "ny": int(_log(rng, 64, 320)), "nz": int(_log(rng, 48, 240)), **_spacing(rng),
                "beam": rng.choice(["dx", "spiral", "spiral_wide", "cbct", "sequential", "dual"]),
                "kvp": round(rng.uniform(60.0, 140.0), 1), "histories": int(_log(rng, 1e5, 2e8)),
                "correction": rng.choice([0, 1, 1, 1, 2]), "dose_to": rng.choice(["host", "device"])}
    if kind == "patient":
        return {"kind": kind, "phantom": rng.choice(["torso", "body"]), "nx": int(_log(rng, 64, 256)),
                "ny": int(_log(rng, 64, 256)), "nz": int(_log(rng, 48, 200)), **_spacing(rng),
                "beam": rng.choice(["dx", "spiral", "cbct"]), "kvp": round(rng.uniform(60.0, 140.0), 1),
                "histories": int(_log(rng, 1e6, 1e8)), "correction": 1, "dose_to": "host"}
    if kind == "batch":
        lo = int(_log(rng, 5e4, 2e6))
        return {"kind": kind, "jobs": rng.randint(3, 12), "dim_lo": 64, "dim_hi": rng.randint(80, 160),
                "hist_lo": lo, "hist_hi": int(lo * rng.uniform(1.0, 8.0))}
    if kind == "forward":
        return {"kind": kind, "b": rng.choice([1, 1, 1, 2]), "d": 8 * int(_log(rng, 4, 26)),
                "h": 8 * int(_log(rng, 4, 33)), "w": 8 * int(_log(rng, 4, 33))}
    if kind == "train":
        return {"kind": kind, "b": rng.randint(1, 8), "p": rng.choice([32, 40, 48, 56, 64])}
    if kind == "denoise":
        return {"kind": kind, "phantom": rng.choice(["torso", "body"]), "nx": 8 * rng.randint(12, 32),
                "ny": 8 * rng.randint(12, 32), "nz": 8 * rng.randint(8, 25), **_spacing(rng)}
    return {"kind": kind, "n": int(_log(rng, 2e5, 8e6))}


# ---------------------------------------------------------------- phantoms and beams
def _phantom(kind, dims, seed):
    """Seeded nested ellipsoids in the six materials (cylinder: air, water, bone) on a grid of
    `dims`, densities with +-2 % jitter: (float32 density, uint8 material) on the GPU."""
    nx, ny, nz = dims
    r = random.Random(seed)
    ax = [torch.linspace(-1.0 + 1.0 / n, 1.0 - 1.0 / n, n, device="cuda") for n in (nz, ny, nx)]
    Z, Y, X = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    mat = torch.zeros((nz, ny, nx), dtype=torch.uint8, device="cuda")

    def put(m, c, a, only=None):
        inside = ((X - c[0]) / a[0]) ** 2 + ((Y - c[1]) / a[1]) ** 2 + ((Z - c[2]) / a[2]) ** 2 < 1.0
        if only is not None:
            inside &= mat == only
        mat[inside] = m

    def near(*v, by=0.03):
        return [x + r.uniform(-by, by) for x in v]

    big = 1e3  # an axis along which the shape does not end
    if kind == "cylinder":
        put(1, near(0, 0, 0, by=0.01), (0.9, 0.9, big))
        put(2, near(0.5, 0, 0), (0.18, 0.18, big))
        mat[(Z.abs() > 0.94).expand_as(mat)] = 0
    else:
        if kind == "torso":
            scale, length = (0.76, 0.54), big
        else:
            scale, length = (r.uniform(0.8, 0.9), r.uniform(0.8, 0.9)), r.uniform(0.8, 0.9)
        a = (scale[0], scale[1], length)
        put(2, (0, 0, 0), a)
        put(4, (0, 0, 0), (0.91 * a[0], 0.88 * a[1], length))
        put(3, (0, 0.015, 0), (0.83 * a[0], 0.78 * a[1], length))
        for s in (-1, 1):
            put(1, near(0.4 * s * a[0], 0.07, 0.3), (0.3 * a[0], 0.55 * a[1], 0.6), only=3)
            put(5, near(0.57 * s * a[0], -0.14 * a[1], -0.7), (0.2 * a[0], 0.38 * a[1], 0.22))
        put(4, near(0.1 * a[0], -0.05 * a[1], 0.2), (0.27 * a[0], 0.34 * a[1], 0.33))
        put(2, near(0.2 * a[0], 0.2 * a[1], -0.6), (0.2 * a[0], 0.24 * a[1], 0.27))
        put(5, near(0, -0.65 * a[1], 0, by=0.01), (0.11 * a[0], 0.14 * a[1], big))
    nominal = [0.0012, 1.0, 1.92] if kind == "cylinder" else [d for _, _, d in P.SIX_MATERIALS]
    rho = torch.tensor(nominal, dtype=torch.float32, device="cuda")[mat.long()]
    g = torch.Generator(device="cuda").manual_seed(seed)
    rho *= 0.98 + 0.04 * torch.rand(mat.shape, generator=g, device="cuda")
    return rho, mat


def _materials(kind):
    return [P.AIR, P.WATER, P.BONE] if kind == "cylinder" else [c for _, c, _ in P.SIX_MATERIALS]


def _beam(case):
    """The beam of a case, sized to its grid, with the particles per exposure that make up its
    histories."""
    lx, ly, lz = case["nx"] * case["sx"], case["ny"] * case["sy"], case["nz"] * case["sz"]
    kvp, kind = case["kvp"], case["beam"]
    scan = min(20.0, 0.6 * lz)
    if kind == "dx":
        b = P.dx_beam_params(kvp=kvp, field_cm=min(40.0, max(2.0, 0.7 * min(lx, lz))), particles=1)
    elif kind == "spiral":
        b = P.ct_spiral_params(kvp=kvp, scan_cm=scan, particles=1)
    elif kind == "spiral_wide":
        b = P.ct_spiral_params(kvp=kvp, pitch=0.8, collimation_cm=8.0, scan_cm=scan, particles=1)
    elif kind == "cbct":
        b = P.cbct_params(kvp=kvp, half_angles=(math.atan(0.4 * max(lx, ly) / 60.0), math.atan(0.4 * lz / 60.0)),
                          particles=1)
    elif kind == "sequential":
        b = P.ct_sequential_params(kvp=kvp, n_slices=3, slice_spacing_cm=scan / 3, position=(0.0, 0.0, -scan / 3),
                                   particles=1)
    else:
        b = P.ct_dual_energy_params(kvp_a=kvp, scan_cm=scan, particles=1)
    b["particles_per_exposure"] = max(1, case["histories"] // len(G.beam_exposures(b)))
    return b


def _outputs(n, where):
    """Dose, variance and event counts of n voxels, in pinned host or device memory."""
    at = {"pin_memory": True} if where == "host" else {"device": "cuda"}
    return (torch.zeros(n, dtype=torch.float64, **at), torch.zeros(n, dtype=torch.float64, **at),
            torch.zeros(n, dtype=torch.int64, **at))


def _read_dose(world, out):
    """dxmcg_world_read_dose into torch memory the GPU can write (pinned or device)."""
    d, v, c = (x.data_ptr() for x in out)
    N.check(N.lib().dxmcg_world_read_dose(world._h, C.cast(d, C.POINTER(C.c_double)),
                                          C.cast(v, C.POINTER(C.c_double)), C.cast(c, C.POINTER(C.c_uint64))))


def _counts(st):
    return [int(st[k]) for k in ("n_histories", "n_missed", "n_photo", "n_compton", "n_rayleigh", "n_cutoff",
                                 "n_fluorescence", "n_errors")]


# ---------------------------------------------------------------- network inputs
def _volume(b, d, h, w, seed):
    """A noisy short run's dose over a smooth one in a torso, as (noisy, smooth, rho, mat)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    parts = []
    for k in range(b):
        rho, mat = _phantom("torso", (w, h, d), 7 * seed + k)
        z, y, x = (torch.linspace(-1, 1, n, device="cuda") for n in (d, h, w))
        ph = torch.rand(4, generator=g, device="cuda") * 3.0
        smooth = (1.2 + 0.4 * torch.sin(2 * x + ph[0])[None, None, :] + 0.3 * torch.cos(2 * y + ph[1])[None, :, None]
                  + 0.2 * torch.sin(3 * z + ph[2])[:, None, None]) * (1.0 + (mat == 5))
        hits = torch.poisson(torch.full_like(smooth, 2.0), generator=g)
        noisy = smooth * hits * (0.25 + 0.5 * torch.rand(smooth.shape, generator=g, device="cuda"))
        noisy[mat == 0] = 0.0
        parts.append((noisy, smooth, rho, mat))
    return [torch.stack(p) for p in zip(*parts)]


def _network():
    net = G.Denoiser(CHANNELS, seed=0)
    net.set_params(np.load(WEIGHTS))
    return net


def _seg_table():
    """A segmentation table of five materials at 120 kVp, written out."""
    t = N.Segmentation()
    t.n_materials = 5
    t.water_attenuation, t.water_density = 0.2059, 1.0
    t.air_attenuation, t.air_density = 0.1855, 0.001205
    for k, v in enumerate((0.1855, 0.1934, 0.2047, 0.2051, 0.2796)):
        t.attenuation[k] = v
    for k, v in enumerate((-1000.0, -107.4, 24.1, 36.0, 480.2)):
        t.hu[k] = v
    for k in range(4):
        t.separator[k] = 0.5 * (t.hu[k] + t.hu[k + 1])
    return t


# ---------------------------------------------------------------- the four entry points
def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind in ("exposure", "patient", "denoise"):
        dims, sp = (case["nx"], case["ny"], case["nz"]), (case["sx"], case["sy"], case["sz"])
        rho, mat = _phantom(case["phantom"], dims, seed)
        world = G.GpuWorld(dims, sp, _materials(case["phantom"]), case.get("correction", 1))
        if kind == "denoise":
            case = dict(case, beam="spiral_wide", kvp=120.0, histories=20_000_000, dose_to="host")
        rho_h = rho.double().cpu().numpy() if kind == "patient" else rho.cpu().numpy()
        mat_h = mat.cpu().numpy()
        del rho, mat
        torch.cuda.empty_cache()
        s = {"kind": kind, "world": world, "beam": _beam(case), "seed": seed}
        if kind == "patient":
            s.update(rho=rho_h, mat=mat_h)
        else:
            world.set_data(rho_h, mat_h)
            world.build()
        if kind == "denoise":
            world.run(s["beam"], G.run_options(seed=seed))
            s.update(net=_network(), out=torch.zeros(world.N, dtype=torch.float64, pin_memory=True))
        else:
            s["out"] = _outputs(world.N, case["dose_to"])
        return s
    if kind == "batch":
        r = random.Random(seed)
        jobs, outs = [], []
        for j in range(case["jobs"]):
            # grid sizes and history counts belong to the case, phantoms and streams to the seed
            q = random.Random(1000 * case["jobs"] + j)
            dims = tuple(q.randint(case["dim_lo"], case["dim_hi"]) for _ in range(3))
            sp = tuple(round(q.uniform(0.1, 0.3), 3) for _ in range(3))
            c = {"nx": dims[0], "ny": dims[1], "nz": dims[2], "sx": sp[0], "sy": sp[1], "sz": sp[2],
                 "kvp": round(q.uniform(60.0, 140.0), 1), "beam": "dx" if j % 2 == 0 else "cbct",
                 "histories": int(_log(q, case["hist_lo"], case["hist_hi"] + 1))}
            rho, mat = _phantom("body", dims, seed * 100 + j)
            w = G.GpuWorld(dims, sp, _materials("body"))
            w.set_data(rho.cpu().numpy(), mat.cpu().numpy())
            w.build()
            jobs.append((w, _beam(c), G.run_options(seed=r.randrange(1 << 30))))
            outs.append(_outputs(w.N, "device"))
        return {"kind": kind, "batch": G.Batch(jobs), "worlds": [w for w, _, _ in jobs], "out": outs}
    if kind == "segment":
        rng = np.random.default_rng(seed)
        hu = rng.choice([-1000.0, -850.0, -105.0, 30.0, 45.0, 600.0], case["n"]) + rng.normal(0, 25.0, case["n"])
        return {"kind": kind, "table": _seg_table(), "hu": np.clip(np.rint(hu), -1024.0, 3071.0)}
    b, d, h, w = (case["b"], case["d"], case["h"], case["w"]) if kind == "forward" else (case["b"],) + (case["p"],) * 3
    noisy, smooth, rho, mat = _volume(b, d, h, w, seed)
    x = G.prepare_input(noisy, rho, mat, 1.2)
    s = {"kind": kind, "net": _network(), "x": x}
    if kind == "train":
        s["target"] = (smooth / 1.2).float().contiguous()
    torch.cuda.synchronize()
    return s


def run(s: dict):
    kind = s["kind"]
    if kind in ("exposure", "patient"):
        world = s["world"]
        if kind == "patient":
            world.set_data(s["rho"], s["mat"])
            world.build()
        else:
            world.clear()
        st = world.run(s["beam"], G.run_options(seed=s["seed"]))
        _read_dose(world, s["out"])
        return {"dose": list(s["out"]), "counts": _counts(st)}
    if kind == "batch":
        for w in s["worlds"]:
            w.clear()
        st = s["batch"].run()
        for w, out in zip(s["worlds"], s["out"]):
            _read_dose(w, out)
        return {"dose": [list(o) for o in s["out"]], "counts": _counts(st)}
    if kind == "forward":
        return s["net"].forward(s["x"])
    if kind == "train":
        # learning rate 0, the first step of a warm-up: the step's whole work on the same weights
        loss = s["net"].train_step(s["x"], s["target"], 0.0)
        return {"loss": loss, "grads": s["net"].grads()}
    if kind == "denoise":
        scale = C.c_double(0)
        N.check(N.lib().dxmcg_world_denoise(s["world"]._h, s["net"]._h, 0.0,
                                            C.cast(s["out"].data_ptr(), C.POINTER(C.c_double)), C.byref(scale)))
        return {"dose": s["out"], "scale": scale.value}
    m, d = G.ct_segment(s["table"], s["hu"])
    return {"material": m, "density": d}


def _net_work(voxels, train):
    """Multiply-add FLOPs of the network's convolutions per pass."""
    prev, fwd, dgrad = 16, 0.0, 0.0
    for l, c in enumerate(CHANNELS):
        f = [54 * prev * c / 8 ** l, 54 * c * c / 8 ** l]
        fwd += sum(f)
        dgrad += f[1] + (f[0] if l else 0.0)
        prev = c
    for l in range(len(CHANNELS) - 1):
        c = CHANNELS[l]
        f = (54 * (CHANNELS[l + 1] + c) * c + 54 * c * c) / 8 ** l
        fwd += f
        dgrad += f
    return voxels * (2 * fwd + dgrad if train else fwd)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "segment":
        return {"bytes": 17.0 * case["n"], "flops": 5.0 * case["n"]}
    if kind in ("forward", "train"):
        v = case["b"] * case["d"] * case["h"] * case["w"] if kind == "forward" else case["b"] * case["p"] ** 3
        out = 4.0 * v if kind == "forward" else 8.0 * v + 4.0 * 1.5e6  # prediction; target, gradients
        return {"bytes": 32.0 * v + out, "flops": _net_work(v, kind == "train")}
    if kind == "denoise":
        v = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 44.0 * v, "flops": 0.4 * _net_work(v, False)}  # layers on the tissue's part of the grid
    # transport: per history about 1.4 deposits of 24 bytes read and written, 8 voxel reads of
    # 4 bytes and 200 arithmetic operations of its thread; per voxel the tally cleared and read
    # with the voxel word, and the dose, variance and count written
    if kind == "batch":
        hist, v = 0.0, 0.0
        for j in range(case["jobs"]):
            q = random.Random(1000 * case["jobs"] + j)
            v += float(np.prod([q.randint(case["dim_lo"], case["dim_hi"]) for _ in range(3)]))
            hist += math.sqrt(case["hist_lo"] * case["hist_hi"])
    else:
        hist, v = case["histories"], case["nx"] * case["ny"] * case["nz"]
    per_voxel = 24.0 + 24.0 + 4.0 + 24.0 + (9.0 + 4.0 if kind == "patient" else 0.0)
    return {"bytes": 100.0 * hist + per_voxel * v, "flops": 400.0 * hist}


# ---------------------------------------------------------------- results in 64 bits
def _exact_net(x, params, target=None):
    """The network in FP64 on the bf16-rounded weights: the prediction, or with a target the
    loss and the gradient of every parameter."""
    F = torch.nn.functional
    p = torch.tensor(params, device="cuda")
    n_conv = p.numel() - (CHANNELS[0] + 1)
    shapes, prev = [], 16
    for c in CHANNELS:
        shapes += [(c, prev), (c, c)]
        prev = c
    for l in range(len(CHANNELS) - 2, -1, -1):
        shapes += [(CHANNELS[l], CHANNELS[l + 1] + CHANNELS[l]), (CHANNELS[l], CHANNELS[l])]
    leaves, o = [], 0
    for co, ci in shapes:
        leaves.append(p[o:o + co * 27 * ci].bfloat16().double().requires_grad_(target is not None))
        o += co * 27 * ci
        leaves.append(p[o:o + co].double().requires_grad_(target is not None))
        o += co
    assert o == n_conv
    head = p[o:].double().requires_grad_(target is not None)

    def conv(k, t):
        co, ci = shapes[k]
        w = leaves[2 * k].view(co, 3, 3, 3, ci).permute(0, 4, 1, 2, 3)
        t = F.pad(t, (1, 1, 1, 1, 1, 1))
        dims = [s - 2 for s in t.shape[2:]]
        acc = leaves[2 * k + 1].view(1, -1, 1, 1, 1)
        for z in range(3):
            for y in range(3):
                for xx in range(3):
                    part = t[:, :, z:z + dims[0], y:y + dims[1], xx:xx + dims[2]]
                    acc = acc + torch.einsum("bczyx,oc->bozyx", part, w[:, :, z, y, xx])
        return torch.relu(acc)

    L = len(CHANNELS)

    def network(t):
        skips = []
        for l in range(L):
            t = conv(2 * l + 1, conv(2 * l, t))
            if l < L - 1:
                skips.append(t)
                t = F.avg_pool3d(t, 2)
        for l in range(L - 2, -1, -1):
            k = 2 * L + 2 * (L - 2 - l)
            up = t.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
            t = conv(k + 1, conv(k, torch.cat([up, skips[l]], 1)))
        return torch.einsum("bczyx,c->bzyx", t, head[:-1]) + head[-1]

    t = x.permute(0, 4, 1, 2, 3).double()
    if target is None:
        with torch.no_grad():
            return torch.cat([network(t[k:k + 1]) for k in range(t.shape[0])])
    loss = 0.0
    for k in range(t.shape[0]):  # one patch at a time: the gradients add up
        part = (network(t[k:k + 1]) - target[k:k + 1].double()).abs().sum() / target.numel()
        part.backward()
        loss += float(part)
    return {"loss": loss, "grads": torch.cat([v.grad for v in leaves] + [head.grad])}


def exact(case: dict, seed: int):
    """Segmentation and the network; the transport's histories have no other 64-bit form than
    the engine's own random streams, and a denoised map starts from such a run."""
    if case["kind"] == "segment":
        s = prepare(case, seed)
        t, hu = s["table"], s["hu"]
        sep, att = np.array(t.separator[:4]), np.array(t.attenuation[:5])
        m = np.searchsorted(sep, hu, side="right").astype(np.uint8)
        w, a = t.water_attenuation * t.water_density, t.air_attenuation * t.air_density
        return {"material": m, "density": np.maximum(((w - a) * hu / 1000.0 + w) / att[m], 0.0)}
    if case["kind"] == "forward":
        s = prepare(case, seed)
        return _exact_net(s["x"], s["net"].get_params())
    if case["kind"] == "train":
        s = prepare(case, seed)
        return _exact_net(s["x"], s["net"].get_params(), s["target"])
    return None
