"""Column passes over more than 256 rows with few lines a tile (one or two coils and
narrow images, or a tuned column block of one): the tile is copied in several boxes, which have to
start on 128 bytes of shared memory.

Tuned blocks give the bytes of the default one.  Narrow images: Cartesian ones against the
double-precision transform (3e-6, the bar of its tests), gridded ones against the same frame with rows and
columns exchanged, whose column pass has few rows (two float32 transforms, 2e-6)."""
import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _complex(rng, *shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


@pytest.mark.parametrize("output", ["OUTPUT_RSS", "OUTPUT_COIL_LAST"])
@pytest.mark.parametrize("rows,cols,coils", [(315, 36, 5), (270, 48, 1), (441, 30, 3), (500, 40, 2), (294, 64, 8),
                                             (343, 20, 33), (486, 32, 1)])
def test_tuned_column_blocks(native, cuda, rows, cols, coils, output):
    import torch
    from kspacejet_gb300 import gpu

    samples = 700
    rng = np.random.default_rng(rows + coils)
    g = gpu.Gridding(image=(rows, cols), channels=coils, samples=samples, frames=2, output=getattr(gpu, output))
    k = torch.from_numpy(_complex(rng, 2, coils, samples)).to(cuda)
    t = torch.from_numpy(rng.uniform(-3.1, 3.1, (2, samples, 2)).astype(np.float32)).to(cuda)
    ws, want = g.new_workspace(cuda), g.new_output(cuda)
    g.run(k, t, want, ws)
    assert g.flags(ws) == 0
    group = max(2, 1 << (min(coils, 32) - 1).bit_length())  # coils of a tile; two tiles where that is not all of them
    for block in (1, 2, 4):
        if rows * block * group * 8 * (2 if coils > 32 else 1) > 200 * 1024:
            continue  # refused: the tile does not fit
        tuning = gpu.GriddingTuning(ctypes.sizeof(gpu.GriddingTuning), 0, block, 0, 0, 0, 0, 0, 0)
        out = g.new_output(cuda)
        g.run(k, t, out, ws, tuning=tuning)
        assert g.flags(ws) == 0
        assert torch.equal(out, want), block


@pytest.mark.parametrize("rows,cols,coils", [(315, 2, 1), (315, 4, 1), (270, 3, 2), (441, 7, 1), (500, 2, 3), (294, 5, 2)])
def test_narrow_images(native, cuda, rows, cols, coils):
    import torch
    from kspacejet_gb300 import gpu
    from oracle.cartesian import ifft2_coil_images

    rng = np.random.default_rng(rows * cols)
    x = _complex(rng, 2, coils, rows, cols)
    got = gpu.cartesian_ifft2(torch.from_numpy(x).to(cuda)).cpu().numpy()
    assert oracle.rel_l2(got, ifft2_coil_images(x)) <= 3e-6

    samples = 300
    k = torch.from_numpy(_complex(rng, 1, coils, samples)).to(cuda)
    t = torch.from_numpy(rng.uniform(-3.1, 3.1, (1, samples, 2)).astype(np.float32)).to(cuda)
    images = []
    for shape, tr in (((rows, cols), t), ((cols, rows), t.flip(-1).contiguous())):
        if not all(_smooth(n) for n in shape):
            return
        g = gpu.Gridding(image=shape, channels=coils, samples=samples, output=gpu.OUTPUT_COIL_MAJOR)
        out, ws = g.new_output(cuda), g.new_workspace(cuda)
        g.run(k, tr, out, ws)
        assert g.flags(ws) == 0
        images.append(out.cpu().numpy())
    assert oracle.rel_l2(images[0], images[1].transpose(0, 1, 3, 2)) <= 2e-6


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1
