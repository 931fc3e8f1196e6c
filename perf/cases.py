"""The work this framework is timed on: its public entry points over the sizes that its users have.

Most cases are adjoint gridding reconstructions (`gpu.Gridding.run`, `gpu.Gridding3.run`) from a
single small slice to a dynamic series and a 3-D volume; the others are the steps around it: the
forward NUFFT, density weights, coil calibration, coil combination and Cartesian coil images.
Trajectories are golden-angle radial (2-D) and Fibonacci-sphere kooshball (3-D) with a rotation
drawn from the seed; k-space is that of an ellipse phantom with smooth coil maps and noise at about
30 dB, so the signal is concentrated at the k-space centre as in a scan.
"""
import math

import numpy as np
import torch

from kspacejet_gb300 import gpu

DEVICE = "cuda"
GOLDEN_ANGLE = math.pi / ((1.0 + math.sqrt(5.0)) / 2.0)


# ---------------------------------------------------------------- the cases


def listed():
    return [
        # one small slice of a served stream, submitted alone: launches and latency
        {"name": "slice_small", "kind": "adjoint2", "image": 64, "grid": 128, "readout": 128, "spokes": 64, "coils": 8,
         "frames": 1, "width": 4, "kernel": "kb", "dcf": "ramp", "output": "rss", "samples": "cf32"},
        # one frame of a dynamic series, reconstructed as it arrives
        {"name": "frame_32coils", "kind": "adjoint2", "image": 192, "grid": 384, "readout": 384, "spokes": 34,
         "coils": 32, "frames": 1, "width": 4, "kernel": "kb", "dcf": "ramp", "output": "rss", "samples": "cf32"},
        # a fully sampled radial slice with a small coil array
        {"name": "plain_radial", "kind": "adjoint2", "image": 256, "grid": 512, "readout": 512, "spokes": 402,
         "coils": 8, "frames": 1, "width": 4, "kernel": "kb", "dcf": "ramp", "output": "rss", "samples": "cf32"},
        # the drop-in linear operator at the largest frame its envelope admits, coil images out
        {"name": "linear_dropin", "kind": "adjoint2", "image": 256, "grid": 256, "readout": 256, "spokes": 256,
         "coils": 8, "frames": 1, "width": 2, "kernel": "linear", "dcf": "ramp", "output": "coil_last",
         "samples": "cf32"},
        # odd sizes: a sigma = 1.5 grid with factors 3 and 5, a wide kernel, iterative density weights, 11 coils
        {"name": "odd_series", "kind": "adjoint2", "image": 200, "grid": 300, "readout": 301, "spokes": 77, "coils": 11,
         "frames": 7, "width": 6, "kernel": "kb", "dcf": "external", "output": "coil_last", "samples": "cf32"},
        # the batched dynamic series
        {"name": "dynamic_series", "kind": "adjoint2", "image": 192, "grid": 384, "readout": 384, "spokes": 34,
         "coils": 32, "frames": 96, "width": 4, "kernel": "kb", "dcf": "ramp", "output": "rss", "samples": "cf32"},
        # the mixed-precision 3-D kooshball volume: bfloat16 sample storage, iterative density weights
        {"name": "kooshball3d", "kind": "adjoint3", "image": 256, "grid": 384, "readout": 256, "spokes": 40000,
         "coils": 20, "width": 4, "dcf": "external", "output": "rss", "samples": "bf16"},
        # coil images -> samples, the other half of an iterative reconstruction's step
        {"name": "forward_series", "kind": "forward2", "image": 192, "grid": 384, "readout": 384, "spokes": 34,
         "coils": 32, "frames": 24, "width": 4},
        # density weights of a dynamic series' trajectories
        {"name": "density_weights", "kind": "weights2", "image": 192, "grid": 384, "readout": 384, "spokes": 34,
         "frames": 96, "width": 4, "iterations": 10},
        # whitening, covariance and 32 -> 8 compression of one acquisition (512 readout x 805 spokes)
        {"name": "coil_preparation", "kind": "coils", "coils": 32, "virtual": 8, "samples": 412160},
        # adaptive combination of the compressed coil images
        {"name": "adaptive_combine", "kind": "walsh", "rows": 256, "cols": 256, "coils": 8, "window": 7,
         "iterations": 24},
        # Cartesian coil images of a multi-slice scan
        {"name": "cartesian_images", "kind": "cartesian", "rows": 256, "cols": 256, "coils": 32, "frames": 8,
         "output": "coil_last"},
    ]


def _spread(rng, low, high):
    """A whole number between low and high, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["adjoint2", "adjoint2", "adjoint2", "adjoint2", "linear", "adjoint3", "forward2", "weights2",
                       "coils", "walsh", "cartesian"])
    if kind == "adjoint2":
        image = rng.choice([64, 80, 84, 90, 96, 128, 150, 160, 168, 192, 200, 224, 256])
        grid = rng.choice([g for g in (image * 3 // 2, image * 2) if _grid_length(g)])
        readout = image + rng.randrange(image + 1)
        spokes, coils = _spread(rng, 24, 805), rng.randint(4, 32)
        frames = _spread(rng, 1, max(1.0, min(96.0, 40e6 / (readout * spokes * coils))))
        return {"kind": "adjoint2", "image": image, "grid": grid, "readout": readout, "spokes": spokes, "coils": coils,
                "frames": frames, "width": rng.choice([4, 4, 4, 6]), "kernel": "kb",
                "dcf": rng.choice(["ramp", "ramp", "external"]), "output": rng.choice(["rss", "rss", "coil_last",
                                                                                      "coil_major"]),
                "samples": rng.choice(["cf32", "cf32", "bf16"])}
    if kind == "linear":
        image = rng.choice([64, 128, 192, 256])
        return {"kind": "adjoint2", "image": image, "grid": image, "readout": image,
                "spokes": _spread(rng, 24, 65536 // image), "coils": rng.randint(4, 32), "frames": rng.randint(1, 4),
                "width": 2, "kernel": "linear", "dcf": "ramp", "output": "coil_last", "samples": "cf32"}
    if kind == "adjoint3":
        image = rng.choice([64, 80, 96, 112, 128, 144])
        return {"kind": "adjoint3", "image": image, "grid": image * 3 // 2, "readout": image + rng.randrange(33),
                "spokes": _spread(rng, 1000, 16000), "coils": rng.randint(4, 20), "width": 4,
                "dcf": rng.choice(["ramp", "external"]), "output": rng.choice(["rss", "coil_last"]),
                "samples": rng.choice(["cf32", "bf16"])}
    if kind == "forward2":
        image = rng.choice([64, 96, 120, 128, 160, 192])
        coils, spokes = rng.randint(4, 32), _spread(rng, 24, 402)
        return {"kind": "forward2", "image": image, "grid": 2 * image, "readout": 2 * image, "spokes": spokes,
                "coils": coils, "frames": _spread(rng, 1, max(1.0, min(24.0, 10e6 / (2 * image * spokes * coils)))),
                "width": rng.choice([4, 4, 6])}
    if kind == "weights2":
        image = rng.choice([64, 96, 128, 150, 192, 256])
        readout, spokes = 2 * image - rng.randrange(image // 2), _spread(rng, 24, 402)
        return {"kind": "weights2", "image": image, "grid": 2 * image, "readout": readout, "spokes": spokes,
                "frames": _spread(rng, 1, max(1.0, min(96.0, 1.25e6 / (readout * spokes)))), "width": 4,
                "iterations": 10}
    if kind == "coils":
        coils = rng.randint(12, 32)
        return {"kind": "coils", "coils": coils, "virtual": rng.randint(4, min(12, coils)),
                "samples": _spread(rng, 8192, 412160)}
    if kind == "walsh":
        return {"kind": "walsh", "rows": _spread(rng, 64, 400), "cols": _spread(rng, 64, 400),
                "coils": rng.randint(4, 8), "window": rng.choice([5, 7, 7, 9]), "iterations": 24}
    coils = rng.randint(4, 32)
    rows, cols = rng.choice([96, 128, 160, 192, 240, 256, 320]), rng.choice([96, 128, 160, 192, 240, 256, 320])
    return {"kind": "cartesian", "rows": rows, "cols": cols, "coils": coils,
            "frames": _spread(rng, 1, max(1.0, min(8.0, 16.7e6 / (rows * cols * coils)))),
            "output": rng.choice(["coil_last", "rss"])}


def _grid_length(n):
    """A length with a mixed-radix transform whose last 16 columns, where there are fewer, still hold a stencil."""
    smooth = n
    for p in (2, 3, 5, 7):
        while smooth % p == 0:
            smooth //= p
    return smooth == 1 and (n % 16 == 0 or n % 16 > 4)


# ---------------------------------------------------------------- inputs


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(0x6B53 + int(seed))
    return g


def _noise(g, *shape):
    return torch.complex(torch.randn(*shape, generator=g, device=DEVICE), torch.randn(*shape, generator=g, device=DEVICE))


def _radial(case, frames, g):
    """[frames, spokes * readout, 2] (k_row, k_col), radians per pixel; spokes run on from frame to frame."""
    readout, spokes = case["readout"], case["spokes"]
    first = float(torch.rand(1, generator=g, device=DEVICE, dtype=torch.float64)) * 2.0 * math.pi
    k = (torch.arange(readout, device=DEVICE, dtype=torch.float64) - readout // 2) * (2.0 * math.pi / readout)
    a = torch.arange(frames * spokes, device=DEVICE, dtype=torch.float64) * GOLDEN_ANGLE + first
    t = torch.stack([torch.sin(a)[:, None] * k, torch.cos(a)[:, None] * k], dim=-1).float()
    return t.clamp_(-math.pi, math.pi).reshape(frames, spokes * readout, 2).contiguous()


def _kooshball(case, g):
    """[spokes * readout, 3] (k_z, k_y, k_x), radians per voxel."""
    readout, spokes = case["readout"], case["spokes"]
    first = float(torch.rand(1, generator=g, device=DEVICE, dtype=torch.float64)) * 2.0 * math.pi
    i = torch.arange(spokes, device=DEVICE, dtype=torch.float64)
    z = 1.0 - (2.0 * i + 1.0) / spokes
    r, phi = torch.sqrt(1.0 - z * z), i * (math.pi * (3.0 - math.sqrt(5.0))) + first
    d = torch.stack([z, r * torch.sin(phi), r * torch.cos(phi)], dim=-1)
    k = (torch.arange(readout, device=DEVICE, dtype=torch.float64) - readout // 2) * (2.0 * math.pi / readout)
    return (d[:, None, :] * k[None, :, None]).float().reshape(-1, 3).contiguous()


def _phantom(k, image):
    """Fourier transform of two ellipses (discs in 2-D, balls in 3-D, stretched) at k [..., dims]."""
    out = 0.0
    for centre, size, value in ((0.0, 0.7, 1.0), (0.12, 0.17, 0.5)):
        axes = torch.tensor([size, 0.75 * size, 0.9 * size][: k.shape[-1]], device=DEVICE) * (image / 2.0)
        q = torch.linalg.vector_norm(k * axes, dim=-1).clamp_min(1e-3)
        if k.shape[-1] == 2:
            shape = 2.0 * math.pi * torch.special.bessel_j1(q) / q
        else:
            shape = 4.0 * math.pi * (torch.sin(q) - q * torch.cos(q)) / (q * q * q)
        turn = k.sum(-1) * (centre * image / 2.0)
        out = out + value * float(axes.prod()) * shape * torch.complex(torch.cos(turn), -torch.sin(turn))
    return out


def _kspace(traj, case, g):
    """[frames, coils, samples] of the phantom seen through smooth coil maps, with noise; traj [frames, samples, d]."""
    coils, image, d = case["coils"], case["image"], traj.shape[-1]
    gain = _noise(g, coils) + 1.0
    slope = (torch.rand(coils, d, generator=g, device=DEVICE) * 6.0 - 3.0) * (2.0 * math.pi / image)
    out = torch.empty(traj.shape[0], coils, traj.shape[1], dtype=torch.complex64, device=DEVICE)
    for c in range(coils):
        for f0 in range(0, traj.shape[0], 32):
            out[f0:f0 + 32, c] = gain[c] * _phantom(traj[f0:f0 + 32] - slope[c], image)
    level = float(out[:1].abs().square().mean().sqrt()) * 10.0 ** (-30.0 / 20.0) / math.sqrt(2.0)
    for f in range(traj.shape[0]):
        for c0 in range(0, coils, 8):
            part = out[f, c0:c0 + 8]
            part += level * _noise(g, *part.shape)
    return out


def _smooth_images(g, frames, rows, cols, coils):
    """Coil-last images: an ellipse with texture, times smooth complex coil maps, plus weak noise."""
    y = torch.linspace(-1, 1, rows, device=DEVICE)[:, None]
    x = torch.linspace(-1, 1, cols, device=DEVICE)[None, :]
    body = ((x / 0.7) ** 2 + (y / 0.9) ** 2 < 1).float() * (1.0 + 0.3 * torch.cos(9 * x) * torch.cos(7 * y))
    a = torch.rand(4, coils, generator=g, device=DEVICE) * 2.0 - 1.0
    maps = torch.exp(-((y[..., None] - a[0]) ** 2 + (x[..., None] - a[1]) ** 2))
    turn = 2.0 * (a[2] * y[..., None] + a[3] * x[..., None])
    image = torch.complex(body[..., None] * maps * torch.cos(turn), body[..., None] * maps * torch.sin(turn))
    return (image[None] + 0.02 * _noise(g, frames, rows, cols, coils)).contiguous()


def _inputs(case, seed):
    """The tensors a user's program has in hand: what prepare() and exact() both start from."""
    g = _generator(seed)
    kind = case["kind"]
    if kind in ("adjoint2", "adjoint3"):
        traj = _radial(case, case["frames"], g) if kind == "adjoint2" else _kooshball(case, g)[None]
        k = _kspace(traj, case, g)
        if case["samples"] == "bf16":
            k = torch.view_as_real(k).to(torch.bfloat16).contiguous()
        dcf = None
        if case["dcf"] == "external":  # smooth positive weights of a radial scan
            r = torch.linalg.vector_norm(traj, dim=-1)
            dcf = ((r + 0.05) ** (traj.shape[-1] - 1) * (0.9 + 0.2 * torch.rand(r.shape, generator=g, device=DEVICE)))
            dcf = dcf.contiguous()
        return {"traj": traj, "k": k, "dcf": dcf}
    if kind == "forward2":
        return {"traj": _radial(case, case["frames"], g),
                "image": _smooth_images(g, case["frames"], case["image"], case["image"], case["coils"])}
    if kind == "weights2":
        return {"traj": _radial(case, case["frames"], g)}
    if kind == "coils":
        c, m, v = case["coils"], case["samples"], case["virtual"]
        mix = 0.3 * _noise(g, c, c) + torch.eye(c, device=DEVICE)
        decay = torch.exp(-6.0 * torch.rand(m, generator=g, device=DEVICE))
        signal = _noise(g, c, 6) @ (_noise(g, 6, m) * decay)
        q = torch.linalg.qr(_noise(g, c, v).to(torch.complex128))[0]
        return {"whitening": torch.linalg.inv(mix.to(torch.complex128)).to(torch.complex64).contiguous(),
                "basis": q.mH.to(torch.complex64).contiguous(),
                "k": (signal + 0.05 * (mix @ _noise(g, c, m))).contiguous()}
    if kind == "walsh":
        return {"image": _smooth_images(g, 1, case["rows"], case["cols"], case["coils"])[0].contiguous()}
    image = _smooth_images(g, case["frames"], case["rows"], case["cols"], case["coils"]).permute(0, 3, 1, 2)
    return {"k": torch.fft.fft2(image).contiguous()}


# ---------------------------------------------------------------- the passes

_OUTPUT = {"rss": gpu.OUTPUT_RSS, "coil_last": gpu.OUTPUT_COIL_LAST, "coil_major": gpu.OUTPUT_COIL_MAJOR}
_DCF = {"ramp": gpu.DCF_ANALYTIC_RAMP, "external": gpu.DCF_EXTERNAL}
_FORMAT = {"cf32": gpu.SAMPLES_CF32, "bf16": gpu.SAMPLES_BF16}


def prepare(case, seed):
    s = dict(_inputs(case, seed), case=case)
    kind = case["kind"]
    if kind == "adjoint2":
        if case["kernel"] == "kb":
            s["plan"] = gpu.kb_gridding(case["image"], case["grid"], case["coils"], case["readout"] * case["spokes"],
                                        frames=case["frames"], width=case["width"], output=_OUTPUT[case["output"]],
                                        dcf=_DCF[case["dcf"]], sample_format=_FORMAT[case["samples"]])
        else:
            s["plan"] = gpu.Gridding(image=(case["image"], case["image"]), channels=case["coils"],
                                     samples=case["readout"] * case["spokes"], frames=case["frames"],
                                     dcf=_DCF[case["dcf"]], output=_OUTPUT[case["output"]])
    elif kind == "adjoint3":
        s["plan"] = gpu.Gridding3(image=case["image"], grid=case["grid"], channels=case["coils"],
                                  samples=case["readout"] * case["spokes"], width=case["width"], dcf=_DCF[case["dcf"]],
                                  output=_OUTPUT[case["output"]], sample_format=_FORMAT[case["samples"]])
    elif kind == "forward2":
        s["plan"] = gpu.kb_gridding(case["image"], case["grid"], case["coils"], case["readout"] * case["spokes"],
                                    frames=case["frames"], width=case["width"])
        s["workspace"] = torch.empty(s["plan"].forward_workspace_bytes(), dtype=torch.uint8, device=DEVICE)
    if kind in ("adjoint2", "adjoint3"):
        s["workspace"], s["out"] = s["plan"].new_workspace(DEVICE), s["plan"].new_output(DEVICE)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("adjoint2", "adjoint3"):
        state["plan"].run(state["k"], state["traj"], state["out"], state["workspace"], dcf=state["dcf"])
        return state["out"]
    if kind == "forward2":
        return state["plan"].forward(state["image"], state["traj"], workspace=state["workspace"])
    if kind == "weights2":
        return gpu.pipe_menon_dcf(state["traj"], case["image"], case["grid"], width=case["width"],
                                  iterations=case["iterations"])
    if kind == "coils":
        white = gpu.noise_prewhiten(state["whitening"], state["k"])
        return {"white": white, "covariance": gpu.coil_covariance(white),
                "compressed": gpu.coil_compress(state["basis"], white)}
    if kind == "walsh":
        return gpu.walsh_combine(state["image"], window=case["window"], iterations=case["iterations"])
    return gpu.cartesian_ifft2(state["k"], output=_OUTPUT[case["output"]])


def work(case):
    """Bytes: inputs read once, results written once.  Flops: the taps, 5 N log2 N per transform of the oversampled
    grid, and the sums that define the other steps."""
    kind = case["kind"]
    if kind in ("adjoint2", "adjoint3", "forward2"):
        d = 3 if kind == "adjoint3" else 2
        frames, c, m = case.get("frames", 1), case["coils"], case["readout"] * case["spokes"]
        pixels, cells = case["image"] ** d, case["grid"] ** d
        element = 4 if case.get("samples") == "bf16" else 8
        out = 8 * pixels * c if case.get("output") != "rss" else 4 * pixels
        moved = element * m * c + 4 * d * m + out + (4 * m if case.get("dcf") == "external" else 0)
        flops = c * (4.0 * m * case["width"] ** d + 5.0 * cells * math.log2(cells))
        return {"bytes": float(frames * moved), "flops": float(frames * flops)}
    if kind == "weights2":
        m = case["frames"] * case["readout"] * case["spokes"]
        return {"bytes": 12.0 * m, "flops": 4.0 * m * case["width"] ** 2 * case["iterations"]}
    if kind == "coils":
        c, v, m = case["coils"], case["virtual"], case["samples"]
        return {"bytes": 8.0 * m * (2 * c + v) + 8.0 * (2 * c * c + v * c), "flops": 8.0 * m * c * (1.5 * c + v)}
    if kind == "walsh":
        p, c = case["rows"] * case["cols"], case["coils"]
        return {"bytes": 8.0 * p * (c + 1),
                "flops": p * (4.0 * c * c * 2 * case["window"] + 8.0 * c * c * case["iterations"])}
    p, c = case["frames"] * case["rows"] * case["cols"], case["coils"]
    return {"bytes": p * (8.0 * c + (8.0 * c if case["output"] == "coil_last" else 4.0)),
            "flops": 5.0 * p * c * math.log2(case["rows"] * case["cols"])}


# ---------------------------------------------------------------- the same in 64 bits


def _taps(u, width, beta):
    """First tap and the width weights [..., width] of the Kaiser-Bessel kernel at u (grid cells)."""
    first = torch.floor(u) - width // 2 + 1
    d = first[..., None] + torch.arange(width, device=DEVICE, dtype=torch.float64) - u[..., None]
    arg = (1.0 - (2.0 * d / width) ** 2).clamp_min(0.0)
    return first.long(), torch.special.i0(beta * torch.sqrt(arg)) / float(np.i0(beta))


def _beta(width, sigma):
    return math.pi * math.sqrt((width / sigma * (sigma - 0.5)) ** 2 - 0.8)


def _deapodise(n, g, width, beta):
    q = torch.arange(n, device=DEVICE, dtype=torch.float64) - n // 2
    z2 = beta ** 2 - (math.pi * width * q / g) ** 2
    z = torch.sqrt(z2.abs()).clamp_min(1e-6)
    return float(np.i0(beta)) / (width * torch.where(z2 > 0, torch.sinh(z), torch.sin(z)) * (1.0 / z))


def _cells(first, weights, grid):
    """Every tap of one frame as (cell index, weight) pairs; first, weights: one per axis."""
    out = [(0, 1.0)]
    for f, w in zip(first, weights):
        out = [(i * grid + (f + j) % grid, v * w[..., j]) for i, v in out for j in range(w.shape[-1])]
    return out


def _stencil(traj, case):
    """Per axis first taps and weights of one frame's trajectory [samples, dims]."""
    u = traj.double() * case["grid"] / (2.0 * math.pi)
    if case.get("kernel") == "linear":
        first = torch.floor(u)
        return list(first.long().unbind(-1)), [torch.stack([1.0 - f, f], -1) for f in (u - first).unbind(-1)]
    beta = _beta(case["width"], case["grid"] / case["image"])
    taps = [_taps(x, case["width"], beta) for x in u.unbind(-1)]
    return [t[0] for t in taps], [t[1] for t in taps]


def _phase(traj, case, sign=1.0):
    n = case["image"]
    delta = n // 2 - (n - 1) / 2.0 if case.get("kernel") != "linear" else -(n - 1) / 2.0
    turn = traj.double().sum(-1) * (delta * sign)
    return torch.complex(torch.cos(turn), torch.sin(turn))


def _exact_adjoint(case, x):
    d = x["traj"].shape[-1]
    n, g, c = case["image"], case["grid"], case["coils"]
    keep = (torch.arange(n, device=DEVICE) - n // 2) % g
    result = []
    for f in range(x["traj"].shape[0]):
        traj = x["traj"][f]
        if case["dcf"] == "external":
            w = x["dcf"][f].double()
        else:
            w = torch.linalg.vector_norm(traj.double(), dim=-1) ** (d - 1)
        w = w * _phase(traj, case)
        cells = _cells(*_stencil(traj, case), g)
        images = torch.zeros([n] * d, dtype=torch.float64, device=DEVICE) if case["output"] == "rss" else []
        step = c if d == 2 else 1
        for c0 in range(0, c, step):
            k = x["k"][f, c0:c0 + step]
            k = (torch.view_as_complex(k.double()) if k.dtype == torch.bfloat16 else k.to(torch.complex128)) * w
            grid = torch.zeros(k.shape[0], g ** d, dtype=torch.complex128, device=DEVICE)
            for index, weight in cells:
                grid.index_add_(1, index, k * weight)
            image = torch.fft.ifftn(grid.reshape([-1] + [g] * d), dim=tuple(range(1, d + 1)), norm="forward")
            if case.get("kernel") != "linear":
                factor = _deapodise(n, g, case["width"], _beta(case["width"], g / n))
                for axis in range(1, d + 1):
                    image = image.index_select(axis, keep) * factor.reshape([-1] + [1] * (d - axis))
            if case["output"] == "rss":
                images += image.abs().square().sum(0)
            else:
                images.append(image)
        if case["output"] == "rss":
            result.append(images.sqrt())
        else:
            images = torch.cat(images)
            result.append(images if case["output"] == "coil_major" else images.movedim(0, -1))
    return torch.stack(result) if d == 2 else result[0]


def _exact_forward(case, x):
    n, g, width = case["image"], case["grid"], case["width"]
    factor = _deapodise(n, g, width, _beta(width, g / n))
    keep = (torch.arange(n, device=DEVICE) - n // 2) % g
    result = []
    for f in range(case["frames"]):
        image = x["image"][f].to(torch.complex128).movedim(-1, 0) * factor[:, None] * factor
        grid = torch.zeros(image.shape[0], g, g, dtype=torch.complex128, device=DEVICE)
        grid[:, keep[:, None], keep[None, :]] = image
        grid = torch.fft.fft2(grid).reshape(image.shape[0], -1)
        y = 0.0
        for index, weight in _cells(*_stencil(x["traj"][f], case), g):
            y = y + grid[:, index] * weight
        result.append(y * _phase(x["traj"][f], case, -1.0))
    return torch.stack(result)


def _exact_weights(case, x):
    g, frames = case["grid"], case["frames"]
    first, weights = _stencil(x["traj"], case)
    base = torch.arange(frames, device=DEVICE)[:, None] * (g * g)
    cells = [(base + i, v) for i, v in _cells(first, weights, g)]
    w = torch.ones(x["traj"].shape[:2], dtype=torch.float64, device=DEVICE)
    for _ in range(case["iterations"]):
        grid = torch.zeros(frames * g * g, dtype=torch.float64, device=DEVICE)
        for index, v in cells:
            grid.index_add_(0, index.reshape(-1), (w * v).reshape(-1))
        d = 0.0
        for index, v in cells:
            d = d + grid[index] * v
        w = torch.where(d > 0, w / d, torch.zeros_like(w))
    return w


def _exact_walsh(case, x):
    image = x["image"].to(torch.complex128)
    rows, cols, c = image.shape
    h = case["window"] // 2
    full = torch.zeros(rows + 2 * h, cols + 2 * h, c, dtype=torch.complex128, device=DEVICE)
    full[h:h + rows, h:h + cols] = image
    pair = full[..., :, None] * full[..., None, :].conj()
    tall = sum(pair[i:i + rows] for i in range(2 * h + 1))
    r = sum(tall[:, i:i + cols] for i in range(2 * h + 1))
    v = image[..., None]
    for _ in range(case["iterations"]):
        u = r @ v
        v = u / torch.linalg.vector_norm(u, dim=-2, keepdim=True)
    v = v[..., 0]
    v = v * torch.exp(-1j * torch.angle(v[..., :1]))
    return (v.conj() * image).sum(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "adjoint3" and case["readout"] * case["spokes"] * case["coils"] > 50e6:
        return None  # 64 double-precision atomic additions for each of its 200 million samples
    x = _inputs(case, seed)
    if kind in ("adjoint2", "adjoint3"):
        return _exact_adjoint(case, x)
    if kind == "forward2":
        return _exact_forward(case, x)
    if kind == "weights2":
        return _exact_weights(case, x)
    if kind == "coils":
        white = x["whitening"].to(torch.complex128) @ x["k"].to(torch.complex128)
        return {"white": white, "covariance": white @ white.mH / case["samples"],
                "compressed": x["basis"].to(torch.complex128) @ white}
    if kind == "walsh":
        return _exact_walsh(case, x)
    image = torch.fft.ifft2(x["k"].to(torch.complex128)).permute(0, 2, 3, 1)
    return image if case["output"] == "coil_last" else image.abs().square().sum(-1).sqrt()
