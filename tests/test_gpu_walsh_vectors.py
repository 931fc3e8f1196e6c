"""Adaptive combination where a pixel's own coil vector lies in the space of a
small eigenvalue of its window: coils that share no pixel, one far weaker than the
other.  Each power iteration then has to keep the vector at unit length.

The reference is the same number of power iterations in double precision; the
vectors are exact here (the products of coils without a common pixel are zero), so the
bound is a few roundings of the norm and the product, 1e-5 as for other images."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _combine64(x, window, iterations):
    rows, cols, coils = x.shape
    h, xd = window // 2, x.astype(np.complex128)
    pad = np.pad(xd, ((h, h), (h, h), (0, 0)))
    outer = pad[..., :, None] * pad[..., None, :].conj()
    r = sum(outer[i:i + rows, j:j + cols] for i in range(window) for j in range(window))
    v = xd / np.linalg.norm(xd, axis=-1, keepdims=True)
    for _ in range(iterations):
        u = np.einsum("rcij,rcj->rci", r, v)
        v = u / np.linalg.norm(u, axis=-1, keepdims=True)
    m = np.abs(v[..., :1])
    v = v * np.where(m > 0, v[..., :1].conj() / np.where(m > 0, m, 1), 1)
    return (v.conj() * xd).sum(-1)


@pytest.mark.parametrize("iterations", [1, 12, 13, 24, 100])
@pytest.mark.parametrize("ratio", [1.0, 0.5, 0.3, 0.1, 3e-2, 1e-2, 3e-3, 2e-3, 1e-3, 3e-4, 1e-5, 1e-6, 1e-9, 1e-12])
def test_disjoint_coils(native, cuda, ratio, iterations):
    import torch
    from kspacejet_gb300 import gpu

    rows, cols = 20, 37
    yy, xx = np.mgrid[:rows, :cols]
    x = np.zeros((rows, cols, 2), np.complex64)
    even = (yy + xx) % 2 == 0
    x[even, 0] = 1.0
    x[~even, 1] = ratio * np.exp(0.3j)
    got = gpu.walsh_combine(torch.from_numpy(x).to(cuda), window=7, iterations=iterations).cpu().numpy()
    want = _combine64(x, 7, iterations)
    assert np.all(np.abs(got - want) <= TOL * np.abs(want))


@pytest.mark.parametrize("scale", [1e-6, 1.0, 1e6])
def test_own_vector_orthogonal_to_the_dominant_one(native, cuda, scale):
    """Eight coils in groups of two that share pixels within a group only, each group 30 times weaker."""
    import torch
    from kspacejet_gb300 import gpu

    rng = np.random.default_rng(8)
    rows, cols = 24, 40
    yy, xx = np.mgrid[:rows, :cols]
    group = (yy + 2 * xx) % 4
    x = np.zeros((rows, cols, 8), np.complex64)
    for g in range(4):
        m = group == g
        a, b = 30.0 ** -g, 30.0 ** -g * np.exp(1j * g)
        wiggle = 1 + 0.01 * rng.standard_normal((m.sum(), 2))
        x[m, 2 * g] = scale * a * wiggle[:, 0]
        x[m, 2 * g + 1] = scale * b * wiggle[:, 1]
    got = gpu.walsh_combine(torch.from_numpy(x).to(cuda), window=7, iterations=24).cpu().numpy()
    want = _combine64(x, 7, 24)
    assert np.all(np.abs(got - want) <= TOL * np.abs(want))
