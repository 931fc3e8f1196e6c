"""Density weights of a series that goes through its workspace in passes, the last of them shorter."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GUARD = 1 << 20


def test_passes_of_three_and_two_frames(native, cuda):
    """Five frames whose entries (1.1 M samples x 16 x 80 bytes a frame) fill 4 GB with three:
    the bytes of each frame alone, and nothing past the workspace is written."""
    import torch
    from kspacejet_gb300 import gpu

    frames, samples, image, grid, width = 5, 1_100_000, 64, 128, 8
    rng = np.random.default_rng(11)
    tr = torch.from_numpy(rng.uniform(-np.pi, np.pi, size=(frames, samples, 2)).astype(np.float32)).to(cuda)
    lib = gpu.lib()
    d = gpu.kb_gridding(image, grid, 1, samples, frames=frames, width=width).desc()
    n = int(lib.ksj_gpu_pipe_menon_workspace_bytes(ctypes.byref(d)))
    ws = torch.full((n + GUARD,), 0xA5, dtype=torch.uint8, device=cuda)
    out = torch.empty((frames, samples), dtype=torch.float32, device=cuda)
    torch.cuda.synchronize()
    assert lib.ksj_gpu_pipe_menon_dcf(ctypes.byref(d), 2, tr.data_ptr(), out.data_ptr(), ws.data_ptr(), n, None) == 0
    torch.cuda.synchronize()
    assert bool((ws[n:] == 0xA5).all())
    for f in range(frames):
        assert torch.equal(out[f], gpu.pipe_menon_dcf(tr[f].contiguous(), image, grid, width=width, iterations=2))
    # the workspace of the whole series serves any part of it
    for part in (1, 2, 4):
        p = gpu.kb_gridding(image, grid, 1, samples, frames=part, width=width).desc()
        got = torch.empty((part, samples), dtype=torch.float32, device=cuda)
        torch.cuda.synchronize()
        assert lib.ksj_gpu_pipe_menon_dcf(ctypes.byref(p), 2, tr.data_ptr(), got.data_ptr(), ws.data_ptr(), n, None) == 0
        torch.cuda.synchronize()
        assert torch.equal(got, out[:part])
