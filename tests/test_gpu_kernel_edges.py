"""The kernels at the sizes where their tiling can go wrong: edges of blocks,
remainders, the smallest sizes they accept, and every lane grouping.

Tolerances: list order, coil groupings and copies exactly; float32 forms 1e-5
rel L2 against the double-precision restatements (the bar of the gridding
tests); float32 sums of C products 4 C eps of the sums of absolute values;
Cartesian transforms 3e-6; density weights 1e-7 (float32 rounding of the
result); covariance 1e-4 Frobenius (the split's stated bound).
"""
import numpy as np
import pytest

import oracle
from binning_reference import binning

pytestmark = pytest.mark.gpu

TOL = 1e-5
EPS = 2.0 ** -24


def _torch():
    import torch

    return torch


def _scattered(samples, frames, dims, seed):
    """Trajectories that revisit cells: half radial-like around the centre, half uniform."""
    rng = np.random.default_rng(seed)
    t = rng.uniform(-np.pi, np.pi, size=(frames, samples, dims))
    t[:, ::2] *= rng.uniform(0, 0.2, size=(frames, (samples + 1) // 2, 1))
    return t.astype(np.float32)


def _complex(rng, *shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


# ------------------------------------------------------------------ binning


@pytest.mark.parametrize("image,grid,width,samples,frames", [
    (4, 8, 8, 513, 2),      # every stencil covers the whole grid, both ends of it in one chunk
    (8, 16, 4, 1, 1),       # one sample
    (16, 24, 6, 511, 3),    # two chunks, the last one partial
    (12, 24, 4, 512, 1),    # one whole turn of a block
    (32, 64, 4, 1025, 5),   # turns and a remainder
    (32, 64, 2, 40000, 1),  # several blocks of samples per frame, long lists
    (48, 96, 4, 700, 250),  # one block per frame
])
def test_lists_are_in_sample_order(native, cuda, image, grid, width, samples, frames):
    from kspacejet_gb300 import gpu

    torch = _torch()
    tr = _scattered(samples, frames, 2, seed=grid + samples)
    g = gpu.kb_gridding(image=image, grid=grid, channels=1, samples=samples, frames=frames, width=width)
    k = torch.ones(frames, 1, samples, dtype=torch.complex64, device=cuda)
    ws = g.new_workspace(cuda)
    g.run(k, torch.from_numpy(tr).to(cuda), g.new_output(cuda), ws)
    cw, off, smp = g.binning(ws)
    ref_off, ref_smp = binning(tr, grid, grid, width, True, chunk=cw)
    np.testing.assert_array_equal(off, ref_off)
    np.testing.assert_array_equal(smp, ref_smp)


# ------------------------------------------------- row pass: lane groups


@pytest.mark.parametrize("image,grid,width,samples", [(64, 128, 4, 3000), (4, 8, 8, 700), (24, 40, 6, 9000),
                                                      (96, 192, 2, 5000)])
def test_every_coil_count_gives_the_single_coil_image(native, cuda, image, grid, width, samples):
    from kspacejet_gb300 import gpu

    torch = _torch()
    tr = torch.from_numpy(_scattered(samples, 1, 2, seed=grid)).to(cuda)
    rng = np.random.default_rng(3)
    k = torch.from_numpy(_complex(rng, 1, 40, samples)).to(cuda)
    single = []
    g = gpu.kb_gridding(image=image, grid=grid, channels=1, samples=samples, width=width, output=gpu.OUTPUT_COIL_MAJOR)
    ws = g.new_workspace(cuda)
    for c in range(40):
        out = g.new_output(cuda)
        g.run(k[:, c:c + 1].contiguous(), tr, out, ws)
        single.append(out)
    single = torch.cat(single, dim=1)
    for coils in (2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 40):
        g = gpu.kb_gridding(image=image, grid=grid, channels=coils, samples=samples, width=width,
                            output=gpu.OUTPUT_COIL_MAJOR)
        out = g.new_output(cuda)
        g.run(k[:, :coils].contiguous(), tr, out, g.new_workspace(cuda))
        assert torch.equal(out, single[:, :coils]), coils


@pytest.mark.parametrize("width,samples", [(4, 20000), (6, 3000)])
def test_gridding_of_crowded_rows_matches_fp64(native, cuda, orc, width, samples):
    """Rows of thousands of entries (segments longer than the smallest unit), 16-bit samples too."""
    from kspacejet_gb300 import gpu

    torch = _torch()
    tr = _scattered(samples, 1, 2, seed=samples)
    k = _complex(np.random.default_rng(1), 1, 3, samples)
    d = np.ones(samples)
    for fmt in (gpu.SAMPLES_CF32, gpu.SAMPLES_BF16):
        x = torch.from_numpy(k).to(cuda)
        ref_k = k
        if fmt == gpu.SAMPLES_BF16:
            x = torch.view_as_real(x).to(torch.bfloat16).contiguous()
            ref_k = torch.view_as_complex(x.float()).cpu().numpy()
        g = gpu.kb_gridding(image=16, grid=32, channels=3, samples=samples, width=width, dcf=gpu.DCF_NONE,
                            output=gpu.OUTPUT_COIL_MAJOR, sample_format=fmt)
        out = g.new_output(cuda)
        g.run(x, torch.from_numpy(tr).to(cuda), out, g.new_workspace(cuda))
        for c in range(3):
            ref = orc.kb_gridding(32, 16, ref_k[0, c].astype(np.complex128), tr[0].astype(np.float64), d, width=width)
            assert oracle.rel_l2(out[0, c].cpu().numpy(), ref) <= TOL


# ------------------------------------------------------------------ 3-D


@pytest.mark.parametrize("image,grid,width,samples,coils", [(8, 12, 4, 30000, 3), (10, 20, 2, 513, 1),
                                                            (8, 16, 6, 1500, 9)])
def test_3d_lists_in_order(native, cuda, orc, image, grid, width, samples, coils):
    """Against FP64, and byte-identical however often it is run (the lists' order is the samples')."""
    from kspacejet_gb300 import gpu

    torch = _torch()
    tr = _scattered(samples, 1, 3, seed=samples)[0]
    k = _complex(np.random.default_rng(2), coils, samples)
    g = gpu.Gridding3(image=image, grid=grid, channels=coils, samples=samples, width=width,
                      output=gpu.OUTPUT_COIL_LAST)
    ws = g.new_workspace(cuda)
    outs = []
    for _ in range(3):
        out = g.new_output(cuda)
        g.run(torch.from_numpy(k).to(cuda), torch.from_numpy(tr).to(cuda), out, ws)
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    got = outs[0].cpu().numpy()
    for c in {0, coils - 1}:
        ref = orc.kb_gridding3(grid, image, k[c].astype(np.complex128), tr.astype(np.float64), np.ones(samples),
                               width=width)
        assert oracle.rel_l2(got[..., c], ref) <= TOL


@pytest.mark.parametrize("samples,channels", [(127, 31), (128, 32), (129, 33), (1000, 5)])
def test_samples_moved_beside_the_scan_and_alone(native, cuda, samples, channels):
    """A frame alone (its samples are reordered in the scan's launch) gives the bytes it has in a
    batch of 160 (a launch of their own)."""
    from kspacejet_gb300 import gpu

    torch = _torch()
    frames = 160
    rng = np.random.default_rng(samples)
    tr = torch.from_numpy(_scattered(samples, frames, 2, seed=channels)).to(cuda)
    k = torch.from_numpy(_complex(rng, frames, channels, samples)).to(cuda)
    outs = []
    for n in (1, frames):
        g = gpu.kb_gridding(16, 32, channels, samples, frames=n, output=gpu.OUTPUT_COIL_LAST)
        out = g.new_output(cuda)
        g.run(k[:n].contiguous(), tr[:n].contiguous(), out, g.new_workspace(cuda))
        outs.append(out[0].cpu().numpy())
    assert outs[0].tobytes() == outs[1].tobytes()


@pytest.mark.parametrize("image,grid,coils", [(12, 24, 20), (2, 12, 11), (16, 24, 24), (10, 20, 40), (10, 20, 17)])
def test_3d_coils_in_parts(native, cuda, orc, image, grid, coils):
    """Coil counts whose columns are transformed in parts of 4 or 8 coils, and one that is not."""
    from kspacejet_gb300 import gpu

    torch = _torch()
    samples = 600
    tr = _scattered(samples, 1, 3, seed=coils)[0]
    k = _complex(np.random.default_rng(coils), coils, samples)
    outs = {}
    for output in (gpu.OUTPUT_COIL_LAST, gpu.OUTPUT_RSS):
        g = gpu.Gridding3(image=image, grid=grid, channels=coils, samples=samples, width=4, output=output,
                          dcf=gpu.DCF_NONE)
        ws = g.new_workspace(cuda).fill_(255)  # coils past the last one start as NaN
        outs[output] = g.new_output(cuda)
        g.run(torch.from_numpy(k).to(cuda), torch.from_numpy(tr).to(cuda), outs[output], ws)
    images = outs[gpu.OUTPUT_COIL_LAST].cpu().numpy().reshape(image, image, image, coils)
    for c in range(0, coils, 3):
        ref = orc.kb_gridding3(grid, image, k[c].astype(np.complex128), tr.astype(np.float64), np.ones(samples), width=4)
        assert oracle.rel_l2(images[..., c], ref) <= TOL
    rss = np.sqrt((np.abs(images.astype(np.complex128)) ** 2).sum(-1))
    assert oracle.rel_l2(outs[gpu.OUTPUT_RSS].cpu().numpy().reshape(rss.shape), rss) <= 4 * coils * EPS


# -------------------------------------------------------- density weights


@pytest.mark.parametrize("image,grid,width,samples", [(8, 16, 4, 700), (16, 32, 2, 513), (16, 32, 8, 1500),
                                                      (24, 40, 6, 2000)])
def test_density_weights_of_every_width(native, cuda, orc, image, grid, width, samples):
    from kspacejet_gb300 import gpu

    torch = _torch()
    tr = _scattered(samples, 2, 2, seed=samples + width)
    got = gpu.pipe_menon_dcf(torch.from_numpy(tr).to(cuda), image, grid, width=width, iterations=6).cpu().numpy()
    for f in range(2):
        want = orc.pipe_menon_dcf(tr[f], grid, grid, width, sigma=grid / image, iterations=6)
        assert oracle.rel_l2(got[f].astype(np.float64), want) <= 1e-7


def test_density_weights_in_passes_of_frames(native, cuda):
    """Two frames whose entries (2 M samples x 16 x 80 bytes each) exceed one pass together."""
    from kspacejet_gb300 import gpu

    torch = _torch()
    rng = np.random.default_rng(5)
    tr = torch.from_numpy(rng.uniform(-np.pi, np.pi, size=(2, 2_000_000, 2)).astype(np.float32)).to(cuda)
    both = gpu.pipe_menon_dcf(tr, 128, 256, width=8, iterations=2)
    for f in range(2):
        assert torch.equal(both[f], gpu.pipe_menon_dcf(tr[f].contiguous(), 128, 256, width=8, iterations=2))


@pytest.mark.parametrize("width,beta", [(2, 27.0), (2, 31.0), (4, 12.5), (4, 60.0), (8, 39.0), (8, 120.0)])
def test_density_weights_of_a_given_beta(native, cuda, orc, width, beta):
    """Both sides of what the tap polynomials resolve (the rest takes the Bessel function)."""
    import ctypes

    from kspacejet_gb300 import gpu

    torch = _torch()
    tr = _scattered(900, 1, 2, seed=width)
    g = gpu.kb_gridding(16, 32, 1, 900, width=width)
    d = g.desc()
    d.kb_beta = beta
    lib = gpu.lib()
    n = int(lib.ksj_gpu_pipe_menon_workspace_bytes(ctypes.byref(d)))
    ws = torch.empty(n, dtype=torch.uint8, device=cuda)
    out = torch.empty(900, dtype=torch.float32, device=cuda)
    t = torch.from_numpy(tr).to(cuda)
    torch.cuda.synchronize()
    assert lib.ksj_gpu_pipe_menon_dcf(ctypes.byref(d), 3, t.data_ptr(), out.data_ptr(), ws.data_ptr(), n, None) == 0
    torch.cuda.synchronize()
    want = orc.pipe_menon_dcf(tr[0], 32, 32, width, beta=float(np.float32(beta)), iterations=3)
    assert oracle.rel_l2(out.cpu().numpy().astype(np.float64), want) <= 1e-7


# ------------------------------------------------------------ coil steps


@pytest.mark.parametrize("coils", [1, 8, 31, 32])
@pytest.mark.parametrize("samples", [1, 63, 64, 65, 129, 20001])
def test_covariance_tiles(native, cuda, coils, samples):
    from kspacejet_gb300 import gpu

    torch = _torch()
    x = _complex(np.random.default_rng(samples + coils), coils, samples)
    got = gpu.coil_covariance(torch.from_numpy(x).to(cuda)).cpu().numpy()
    xd = x.astype(np.complex128)
    want = xd @ xd.conj().T / samples
    assert np.linalg.norm(got - want) <= 1e-4 * np.linalg.norm(want)
    noise = gpu.noise_covariance(torch.from_numpy(x).to(cuda)).cpu().numpy()
    xm = xd - xd.mean(axis=1, keepdims=True)
    want_n = (xm @ xm.conj().T / samples).conj()
    assert np.linalg.norm(noise - want_n) <= 1e-4 * np.linalg.norm(want)


@pytest.mark.parametrize("virtual,coils", [(1, 1), (1, 32), (2, 3), (7, 9), (8, 32), (16, 17), (16, 32)])
@pytest.mark.parametrize("samples,shift", [(1, 0), (2, 0), (513, 0), (514, 0), (514, 1)])
def test_compression_samples_together_and_alone(native, cuda, virtual, coils, samples, shift):
    """Even counts on 16-byte rows go several samples a thread, others one."""
    from kspacejet_gb300 import gpu

    torch = _torch()
    rng = np.random.default_rng(virtual * coils + samples)
    b, x = _complex(rng, virtual, coils), _complex(rng, coils, samples)
    held = torch.zeros(coils * samples + 1, dtype=torch.complex64, device=cuda)
    k = held[shift:shift + coils * samples].view(coils, samples)  # off a 16-byte boundary when shifted
    k.copy_(torch.from_numpy(x))
    got = gpu.coil_compress(torch.from_numpy(b).to(cuda), k).cpu().numpy()
    want = b.astype(np.complex128) @ x.astype(np.complex128)
    assert np.all(np.abs(got - want) <= 4 * coils * EPS * (np.abs(b) @ np.abs(x)) + 1e-30)


@pytest.mark.parametrize("coils", [1, 17, 32])
@pytest.mark.parametrize("samples", [3, 1000, 1002])
def test_prewhitening_sizes(native, cuda, coils, samples):
    from kspacejet_gb300 import gpu

    torch = _torch()
    rng = np.random.default_rng(coils)
    w, x = _complex(rng, coils, coils), _complex(rng, coils, samples)
    got = gpu.noise_prewhiten(torch.from_numpy(w).to(cuda), torch.from_numpy(x).to(cuda)).cpu().numpy()
    want = w.astype(np.complex128) @ x.astype(np.complex128)
    assert np.all(np.abs(got - want) <= 4 * coils * EPS * (np.abs(w) @ np.abs(x)))


@pytest.mark.parametrize("rows,cols,coils,window,iterations", [
    (1, 1, 8, 9, 24), (8, 32, 4, 1, 5), (9, 33, 8, 7, 24), (7, 70, 5, 9, 13), (17, 31, 2, 3, 14), (40, 40, 1, 7, 24),
    (33, 65, 7, 5, 0)])
def test_walsh_tiles_and_iterations(native, cuda, rows, cols, coils, window, iterations):
    """Against the same number of power iterations in double precision."""
    from kspacejet_gb300 import gpu

    torch = _torch()
    rng = np.random.default_rng(rows * cols)
    maps = _complex(rng, coils)
    x = (maps * (1.0 + rng.random((rows, cols, 1))) + 0.1 * _complex(rng, rows, cols, coils)).astype(np.complex64)
    if rows > 8:
        x[-3:, -3:] = 0  # pixels of nothing: window and own vector
    got = gpu.walsh_combine(torch.from_numpy(x).to(cuda), window=window, iterations=iterations).cpu().numpy()
    h, xd = window // 2, x.astype(np.complex128)
    pad = np.pad(xd, ((h, h), (h, h), (0, 0)))
    outer = pad[..., :, None] * pad[..., None, :].conj()
    r = sum(outer[i:i + rows, j:j + cols] for i in range(window) for j in range(window))
    v = xd.copy()
    v[np.abs(v).sum(-1) == 0] = np.eye(coils)[0]
    for _ in range(iterations):
        u = np.einsum("rcij,rcj->rci", r, v)
        n = np.linalg.norm(u, axis=-1, keepdims=True)
        v = np.where(n > 0, u / np.where(n > 0, n, 1), v)
    m = np.abs(v[..., :1])
    v = v * np.where(m > 0, v[..., :1].conj() / np.where(m > 0, m, 1), 1)
    want = (v.conj() * xd).sum(-1)
    assert np.linalg.norm(got - want) <= TOL * np.linalg.norm(want)


# ------------------------------------------------------------ transforms


@pytest.mark.parametrize("image,grid", [(64, 128), (60, 128), (96, 192), (128, 192), (128, 256), (192, 384), (255, 384),
                                        (256, 512), (300, 512), (20, 30), (33, 70)])
@pytest.mark.parametrize("coils", [1, 9, 33])
def test_forward_placement(native, cuda, orc, image, grid, coils):
    """Images that fill half the grid and others, on every two-step length and mixed-radix ones."""
    from kspacejet_gb300 import gpu

    torch = _torch()
    rng = np.random.default_rng(grid + coils)
    img = _complex(rng, 1, image, image, coils)
    tr = _scattered(77, 1, 2, seed=grid)
    g = gpu.kb_gridding(image=image, grid=grid, channels=coils, samples=77, width=4)
    got = g.forward(torch.from_numpy(img).to(cuda), torch.from_numpy(tr).to(cuda)).cpu().numpy()
    for c in {0, coils - 1}:
        want = orc.kb_forward(grid, image, img[0, :, :, c], tr[0].astype(np.float64), width=4)
        assert oracle.rel_l2(got[0, c], want) <= TOL


@pytest.mark.parametrize("rows,cols,coils", [(2, 2, 1), (128, 192, 3), (16, 128, 33), (384, 10, 5), (30, 256, 64),
                                             (13, 512, 2), (12, 11, 9), (96, 45, 17)])
def test_cartesian_rows_from_channel_major(native, cuda, rows, cols, coils):
    from kspacejet_gb300 import gpu
    from oracle.cartesian import ifft2_coil_images

    torch = _torch()
    k = _complex(np.random.default_rng(rows + cols), 2, coils, rows, cols)
    want = ifft2_coil_images(k)
    got = gpu.cartesian_ifft2(torch.from_numpy(k).to(cuda)).cpu().numpy()
    assert oracle.rel_l2(got, want) <= 3e-6
    rss = gpu.cartesian_ifft2(torch.from_numpy(k).to(cuda), output=gpu.OUTPUT_RSS).cpu().numpy()
    assert oracle.rel_l2(rss, np.sqrt((np.abs(want) ** 2).sum(-1))) <= 3e-6
