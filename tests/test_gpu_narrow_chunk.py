"""Grids whose last 16-column chunk is narrower than a stencil's inner columns: a
stencil that wraps reaches over that chunk into the first, so its sample stands
in three lists of a row.

The lists are compared exactly with those of the chunks of all W wrapped columns;
images 1e-5 rel L2 and weights 1e-7 against the double-precision restatements (the bars of the
gridding and density-weight tests)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

TOL = 1e-5
TOL_WEIGHTS = 1e-7


def _trajectory(samples, frames, dims, grid, seed):
    """Uniform, a third of it with the columns near the edge between the last and the first."""
    rng = np.random.default_rng(seed)
    t = rng.uniform(-np.pi, np.pi, size=(frames, samples, dims))
    t[:, ::3, -1] = rng.uniform(-9, 9, size=t[:, ::3, -1].shape) * 2 * np.pi / grid
    return t.astype(np.float32)


def _lists(traj, grid, width, chunk):
    """A frame's lists as sample indices, from the set of chunks of the W columns of every row."""
    u = np.floor(traj.astype(np.float64) * grid / (2 * np.pi)).astype(np.int64) - width // 2 + 1
    chunks = (grid + chunk - 1) // chunk
    lists = [[] for _ in range(grid * chunks)]
    for s, (r, c) in enumerate(u):
        touched = sorted({(c + j) % grid // chunk for j in range(width)})
        for j in range(width):
            for k in touched:
                lists[(r + j) % grid * chunks + k].append(s)
    return lists


# (image, grid, width): two chunks (both ends of a wrapped stencil in the first one), four and fifteen
SHAPES = [(9, 18, 4), (9, 18, 6), (9, 18, 8), (12, 20, 6), (12, 20, 8), (12, 21, 8), (25, 49, 4), (33, 50, 4), (25, 50, 8),
          (56, 84, 6), (150, 225, 4), (150, 225, 8)]


@pytest.mark.parametrize("image,grid,width", SHAPES)
def test_lists_name_every_chunk(native, cuda, image, grid, width):
    import torch
    from kspacejet_gb300 import gpu

    samples, frames = 1100, 2
    tr = _trajectory(samples, frames, 2, grid, seed=grid + width)
    g = gpu.kb_gridding(image, grid, 1, samples, frames=frames, width=width)
    ws = g.new_workspace(cuda)
    g.run(torch.ones(frames, 1, samples, dtype=torch.complex64, device=cuda), torch.from_numpy(tr).to(cuda),
          g.new_output(cuda), ws)
    chunk, off, smp = g.binning(ws)
    want = [x for f in range(frames) for x in _lists(tr[f], grid, width, chunk)]
    np.testing.assert_array_equal(off, np.cumsum([0] + [len(x) for x in want]))
    np.testing.assert_array_equal(smp, np.concatenate([np.array(x, np.uint32) for x in want]))


@pytest.mark.parametrize("coils", [1, 5, 32])
@pytest.mark.parametrize("image,grid,width", SHAPES)
def test_adjoint(native, cuda, orc, image, grid, width, coils):
    import torch
    from kspacejet_gb300 import gpu

    samples = 3000
    tr = _trajectory(samples, 1, 2, grid, seed=grid * width)
    rng = np.random.default_rng(coils)
    k = (rng.standard_normal((1, coils, samples)) + 1j * rng.standard_normal((1, coils, samples))).astype(np.complex64)
    g = gpu.kb_gridding(image, grid, coils, samples, width=width, dcf=gpu.DCF_NONE, output=gpu.OUTPUT_COIL_MAJOR)
    out = g.new_output(cuda)
    g.run(torch.from_numpy(k).to(cuda), torch.from_numpy(tr).to(cuda), out, g.new_workspace(cuda))
    for c in {0, coils - 1}:
        want = orc.kb_gridding(grid, image, k[0, c].astype(np.complex128), tr[0].astype(np.float64), np.ones(samples),
                               width=width)
        assert oracle.rel_l2(out[0, c].cpu().numpy(), want) <= TOL


@pytest.mark.parametrize("image,grid,width", SHAPES)
def test_density_weights(native, cuda, orc, image, grid, width):
    import torch
    from kspacejet_gb300 import gpu

    tr = _trajectory(1500, 2, 2, grid, seed=grid - width)
    got = gpu.pipe_menon_dcf(torch.from_numpy(tr).to(cuda), image, grid, width=width, iterations=4).cpu().numpy()
    for f in range(2):
        want = orc.pipe_menon_dcf(tr[f], grid, grid, width, sigma=grid / image, iterations=4)
        assert oracle.rel_l2(got[f].astype(np.float64), want) <= TOL_WEIGHTS


@pytest.mark.parametrize("image,grid,width", [(9, 18, 4), (9, 18, 8), (12, 20, 6), (25, 49, 4)])
def test_3d(native, cuda, orc, image, grid, width):
    import torch
    from kspacejet_gb300 import gpu

    samples = 1500
    tr = _trajectory(samples, 1, 3, grid, seed=grid)[0]
    rng = np.random.default_rng(width)
    k = (rng.standard_normal((2, samples)) + 1j * rng.standard_normal((2, samples))).astype(np.complex64)
    g = gpu.Gridding3(image=image, grid=grid, channels=2, samples=samples, width=width, output=gpu.OUTPUT_COIL_LAST)
    out = g.new_output(cuda)
    g.run(torch.from_numpy(k).to(cuda), torch.from_numpy(tr).to(cuda), out, g.new_workspace(cuda))
    for c in range(2):
        want = orc.kb_gridding3(grid, image, k[c].astype(np.complex128), tr.astype(np.float64), np.ones(samples),
                                width=width)
        assert oracle.rel_l2(out[..., c].cpu().numpy(), want) <= TOL
    got = gpu.pipe_menon_dcf3(torch.from_numpy(tr).to(cuda), image, grid, width=width, iterations=3).cpu().numpy()
    beta = float(np.float32(orc.kb_beta(width, grid / image)))
    want = orc.pipe_menon_dcf3(tr, grid, width, beta=beta, iterations=3)
    assert oracle.rel_l2(got.astype(np.float64), want) <= TOL_WEIGHTS
