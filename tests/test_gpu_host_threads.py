"""Calls of different sizes from several host threads at once.

A kernel's dynamic shared memory limit belongs to the process, so a small
call must not lower it under a large one: every thread's calls are accepted
and give the bytes they give alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CALLS = 60


def _jobs(gpu, torch, cuda):
    """(name, call) pairs; call() launches on the current stream and returns a new output."""
    rng = np.random.default_rng(4)

    def tensor(*shape, complex_=True):
        x = rng.standard_normal(shape)
        if complex_:
            return torch.from_numpy((x + 1j * rng.standard_normal(shape)).astype(np.complex64)).to(cuda)
        return torch.from_numpy(np.clip(x, -3.1, 3.1).astype(np.float32)).to(cuda)

    jobs = []

    def adjoint(grid, channels, samples, frames, width):
        g = gpu.kb_gridding(grid // 2, grid, channels, samples, frames=frames, width=width)
        k, t = tensor(frames, channels, samples), tensor(frames, samples, 2, complex_=False)
        ws = g.new_workspace(cuda)

        def call(stream):
            out = g.new_output(cuda)
            g.run(k, t, out, ws, stream=stream)
            return out

        jobs.append((f"adjoint {grid}", call))

    def adjoint3(grid, channels, samples):
        g = gpu.Gridding3(image=grid // 2, grid=grid, channels=channels, samples=samples)
        k, t = tensor(channels, samples), tensor(samples, 3, complex_=False)
        ws = g.new_workspace(cuda)

        def call(stream):
            out = g.new_output(cuda)
            g.run(k, t, out, ws, stream=stream)
            return out

        jobs.append((f"3-D {grid}", call))

    def forward(grid, channels):
        g = gpu.kb_gridding(grid // 2, grid, channels, 500, width=4)
        x, t = tensor(1, grid // 2, grid // 2, channels), tensor(1, 500, 2, complex_=False)
        ws = torch.empty(g.forward_workspace_bytes(), dtype=torch.uint8, device=cuda)
        jobs.append((f"forward {grid}", lambda stream: g.forward(x, t, workspace=ws, stream=stream)))

    adjoint(16, 1, 300, 1, 4)
    adjoint(512, 2, 20000, 1, 4)
    adjoint(128, 8, 4000, 5, 4)
    adjoint(64, 32, 4000, 1, 4)
    adjoint3(12, 2, 500)
    adjoint3(128, 1, 20000)
    forward(128, 2)
    forward(128, 32)
    small, large = tensor(40, 40, 8), tensor(64, 64, 8)
    jobs.append(("walsh 1", lambda stream: gpu.walsh_combine(small, window=1, iterations=4, stream=stream)))
    jobs.append(("walsh 9", lambda stream: gpu.walsh_combine(large, window=9, iterations=4, stream=stream)))
    return jobs


def test_calls_of_different_sizes_from_several_threads(native, cuda):
    import torch
    from kspacejet_gb300 import gpu

    jobs = _jobs(gpu, torch, cuda)
    torch.cuda.synchronize()
    want = [call(None) for _, call in jobs]
    torch.cuda.synchronize()
    start = threading.Barrier(len(jobs))
    failures = []

    def work(i):
        name, call = jobs[i]
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                stream = torch.cuda.current_stream()
                start.wait(timeout=60)
                for n in range(CALLS):
                    out = call(stream)
                    if n % 10 == 9:
                        stream.synchronize()
                        if not torch.equal(out, want[i]):
                            failures.append(f"{name}: call {n} differs")
                            return
        except Exception as e:  # noqa: BLE001 (reported by the test)
            failures.append(f"{name}: {e}")

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert failures == []
