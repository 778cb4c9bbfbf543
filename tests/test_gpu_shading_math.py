"""Edges of the shading transcendentals' domains against the CPU restatement: rough lobes past the angle where the
half vector's cosine changes formula, grazing and aligned half vectors, sample angles at the quadrants' ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dirs(r, n):
    d = r.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _close(g, c, frac):
    # the lobe's value amplifies a float's rounding of the angle by 2 tan / m^2: 1e-5 relative, but for a
    # fraction of records at the clamps
    bad = ~np.isclose(g, c, rtol=1e-5, atol=1e-5, equal_nan=True)
    assert bad.any(-1).mean() <= frac, bad.any(-1).mean()


# tan of the half-vector angle is roughness * sqrt(-log(1 - r1)): 256 and above at 64 to 1000
@pytest.mark.parametrize("rough", [1e-3, 0.05, 1.0, 63.0, 64.0, 200.0, 1000.0])
def test_half_vector_sampling(ctx, oracle_lib, rough):
    r = np.random.default_rng(int(rough * 1000))
    n = 4000
    N = _dirs(r, n)
    V = N + 0.7 * _dirs(r, n)
    V /= np.linalg.norm(V, axis=1, keepdims=True)
    r1 = np.concatenate([r.integers(0, 1 << 24, n // 2) / 2.0 ** 24, 1.0 - r.integers(1, 64, n // 2) / 2.0 ** 24])
    rec = np.concatenate([np.ones((n, 1)), r.uniform(0.1, 1, (n, 3)), np.full((n, 1), rough), V, N, r1[:, None],
                          r.integers(0, 1 << 24, (n, 1)) / 2.0 ** 24], 1).astype(np.float32)
    g, c = ctx.probe(0, rec), oracle_lib.probe(0, rec)
    _close(g[:, :3], c[:, :3], 2e-3)


def test_hemisphere_angles(ctx, oracle_lib):
    """The azimuth at and beside the multiples of a quarter turn, and over the whole range."""
    k = np.concatenate([q * (1 << 22) + np.arange(-200, 201) for q in range(5)] + [np.arange(0, 1 << 24, 4099)])
    r2 = np.clip(k, 0, (1 << 24) - 1) / 2.0 ** 24
    n = len(r2)
    r = np.random.default_rng(1)
    N = _dirs(r, n)
    rec = np.concatenate([np.zeros((n, 1)), np.ones((n, 3)), np.zeros((n, 1)), N, N, r.uniform(0, 1, (n, 1)), r2[:, None]],
                         1).astype(np.float32)
    g, c = ctx.probe(0, rec), oracle_lib.probe(0, rec)
    np.testing.assert_allclose(g, c, rtol=1e-5, atol=1e-6)


def test_lobe_values_at_aligned_and_grazing_half_vectors(ctx, oracle_lib):
    """Half vectors from the normal itself (cosine 1) to beyond the horizon (negative cosine)."""
    r = np.random.default_rng(2)
    n = 6000
    N = _dirs(r, n)
    t = np.cross(N, _dirs(r, n))
    t /= np.linalg.norm(t, axis=1, keepdims=True)
    a = np.concatenate([np.zeros(100), r.uniform(0, 3e-3, 900), r.uniform(0, np.pi, n - 1000)])[:, None]
    H = N * np.cos(a) + t * np.sin(a)
    s = np.cross(H, _dirs(r, n))
    s /= np.linalg.norm(s, axis=1, keepdims=True)
    b = r.uniform(0.05, 1.2, (n, 1))
    V, L = H * np.cos(b) + s * np.sin(b), H * np.cos(b) - s * np.sin(b)
    rec = np.concatenate([np.ones((n, 1)), r.uniform(0.1, 1, (n, 3)), r.uniform(0.05, 1, (n, 1)), L, V, N], 1).astype(np.float32)
    for kind in (1, 2):
        g, c = ctx.probe(kind, rec), oracle_lib.probe(kind, rec)
        scale = np.maximum(np.abs(c).max(-1, keepdims=True), 1.0)
        _close(g / scale, c / scale, 1e-2)
