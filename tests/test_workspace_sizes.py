"""Workspace sizes grow with the problem: a workspace of the largest call a
program makes serves each of its smaller ones (and the shorter last pass of a
call that goes over its frames in passes).  Sizes are host arithmetic."""
import ctypes

import pytest


@pytest.fixture(scope="module")
def gpu(native):
    from kspacejet_gb300 import gpu

    return gpu


def _adjoint(gpu, grid, width, channels, samples, frames):
    return gpu.kb_gridding(grid // 2, grid, channels, samples, frames=frames, width=width).workspace_bytes()


def _host(gpu, grid, width, channels, samples, frames):
    return gpu.kb_gridding(grid // 2, grid, channels, samples, frames=frames, width=width).host_workspace_bytes()


def _weights(gpu, grid, width, channels, samples, frames):
    d = gpu.kb_gridding(grid // 2, grid, 1, samples, frames=frames, width=width).desc()
    return int(gpu.lib().ksj_gpu_pipe_menon_workspace_bytes(ctypes.byref(d)))


def _grows(sizes):
    sizes = list(sizes)
    assert all(s > 0 for s in sizes)
    assert sizes == sorted(sizes)


@pytest.mark.parametrize("size", [_adjoint, _host, _weights])
@pytest.mark.parametrize("grid,width,channels", [(32, 2, 1), (384, 4, 1), (512, 8, 1)])
def test_size_grows_with_frames(gpu, size, grid, width, channels):
    for samples in (1, 1536, 13312):
        _grows(size(gpu, grid, width, channels, samples, f) for f in range(1, 310))


@pytest.mark.parametrize("size", [_adjoint, _host, _weights])
@pytest.mark.parametrize("grid,width,channels", [(32, 2, 1), (384, 4, 1), (512, 2, 1)])
def test_size_grows_with_samples(gpu, size, grid, width, channels):
    steps = [512 * t + d for t in range(1, 160) for d in (0, 1)]
    for frames in (1, 5, 77):
        _grows(size(gpu, grid, width, channels, m, frames) for m in steps if m * frames < 3_000_000)


@pytest.mark.parametrize("grid,samples,frames", [(256, 41216, 541), (448, 40768, 547), (384, 79488, 279)])
def test_weights_of_a_series_hold_every_shorter_pass(gpu, grid, samples, frames):
    whole = _weights(gpu, grid, 4, 1, samples, frames)
    assert all(_weights(gpu, grid, 4, 1, samples, f) <= whole for f in range(frames // 2 - 40, frames))


@pytest.mark.parametrize("grid", [24, 384, 512])
def test_3d_size_grows_with_samples(gpu, grid):
    sizes3, sizes3w = [], []
    for turns in list(range(1, 40)) + list(range(600, 620)) + list(range(1210, 1220)):
        for samples in (512 * turns, 512 * turns + 1):
            g = gpu.Gridding3(image=grid // 2, grid=grid, channels=1, samples=samples)
            sizes3.append(g.workspace_bytes())
            d = g.desc()
            sizes3w.append(int(gpu.lib().ksj_gpu_pipe_menon3_workspace_bytes(ctypes.byref(d))))
    _grows(sizes3)
    _grows(sizes3w)


@pytest.mark.parametrize("grid,width", [(64, 4), (512, 8)])
def test_weights_size_grows_across_the_passes(gpu, grid, width):
    """Frames of one to several passes of 4 GB of entries; frames of a few samples by the thousand."""
    for frames in (1, 2, 3, 7, 5000, 65535):
        _grows(_weights(gpu, grid, width, 1, m, frames) for m in
               [1, 700, 40_000, 800_000, 1_100_000, 1_118_481, 1_118_482, 1_677_721, 1_677_722, 3_355_443, 3_355_444,
                5_592_405, 5_592_406, 11_184_810, 11_184_811, 1 << 26])
    for m in (1, 40_000, 1_118_482, 5_592_406):
        _grows(_weights(gpu, grid, width, 1, m, f) for f in [1, 2, 3, 4, 5, 10, 83, 84, 2047, 2048, 2049, 65535])
