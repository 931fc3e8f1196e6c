"""Binning lists of millions of entries: every one of them reaches the image.

All samples lie at one place, whose stencil falls into two lists of every row it
covers.  They are zero but for 1000 of them spread over the whole range, positive, so
that the sums are of 1000 terms whatever the lists' lengths; the image is that of
their sum at the place (1e-5, the bar of the gridding tests)."""
import math

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize("samples", [(1 << 22) - 1, 1 << 22, (1 << 22) + 5, 5 << 20, 1 << 23])
def test_every_entry_of_a_long_list_counts(native, cuda, orc, samples):
    import torch
    from kspacejet_gb300 import gpu

    image, grid = 16, 32
    place = np.array([0.3, 15.5 / grid * 2 * math.pi], np.float32)  # columns 14 to 17
    rng = np.random.default_rng(samples)
    at = np.sort(rng.choice(samples, 1000, replace=False))
    at[0], at[-1] = 0, samples - 1
    value = (rng.uniform(0.5, 1.5, 1000) + 1j * rng.uniform(0.5, 1.5, 1000)).astype(np.complex64)
    k = torch.zeros(1, 1, samples, dtype=torch.complex64, device=cuda)
    k[0, 0, torch.from_numpy(at).to(cuda)] = torch.from_numpy(value).to(cuda)
    tr = torch.from_numpy(place).to(cuda).expand(1, samples, 2).contiguous()
    g = gpu.kb_gridding(image, grid, 1, samples, width=4, dcf=gpu.DCF_NONE, output=gpu.OUTPUT_COIL_MAJOR)
    out = g.new_output(cuda)
    g.run(k, tr, out, g.new_workspace(cuda))
    want = orc.kb_gridding(grid, image, np.array([value.astype(np.complex128).sum()]), place[None].astype(np.float64),
                           np.ones(1), width=4)
    assert oracle.rel_l2(out[0, 0].cpu().numpy(), want) <= TOL
