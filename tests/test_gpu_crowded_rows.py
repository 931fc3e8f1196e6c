"""Accuracy of rows whose lists hold very many samples.

All samples lie at one place and have one value a coil, so each cell is the sum
of n equal terms, where the roundings of a running sum add up instead of
cancelling.  A cell's sum is taken in partial sums of at most 512 entries
that are then added up in turn: 512 + n / 512 additions deep, each off by at most 2^-24 of the sum.  The image is that of one sample of n times
the value; its relative error is that of the cells."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SAMPLES = 1 << 17
COILS = 32
TOL = (512 + SAMPLES // 512) * 2.0 ** -24  # 4.6e-5


@pytest.mark.parametrize("dims", [2, 3])
def test_sum_of_equal_samples(native, cuda, orc, dims):
    import torch
    from kspacejet_gb300 import gpu

    image, grid = 16, 24
    rng = np.random.default_rng(dims)
    place = np.array([0.7, -0.4, 15.5 / grid * 2 * np.pi - np.pi][3 - dims:], np.float32)
    value = rng.uniform(0.5, 1.5, (COILS, 2)).astype(np.float32).view(np.complex64)[:, 0]
    k = torch.from_numpy(value).to(cuda)[:, None].expand(COILS, SAMPLES).contiguous()
    tr = torch.from_numpy(place).to(cuda).expand(SAMPLES, dims).contiguous()
    if dims == 2:
        g = gpu.kb_gridding(image, grid, COILS, SAMPLES, dcf=gpu.DCF_NONE, output=gpu.OUTPUT_COIL_LAST)
        k, tr = k[None], tr[None]
    else:
        g = gpu.Gridding3(image=image, grid=grid, channels=COILS, samples=SAMPLES, output=gpu.OUTPUT_COIL_LAST)
    out = g.new_output(cuda)
    g.run(k, tr, out, g.new_workspace(cuda))
    got = out.cpu().numpy().reshape(-1, COILS)
    one = orc.kb_gridding if dims == 2 else orc.kb_gridding3
    want = one(grid, image, np.ones(1, np.complex128), place[None].astype(np.float64), np.ones(1), width=4).reshape(-1)
    for c in range(COILS):
        assert oracle.rel_l2(got[:, c], want * (SAMPLES * complex(value[c]))) <= TOL
