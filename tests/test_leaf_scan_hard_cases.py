"""The cooperative leaf phase (tuning kernel 45: packed arithmetic, leaves
located by reduction) against the kernels whose lanes scan their own leaves
(13, and 0, which also walks the nodes themselves), bit for bit, on what is
hard for the watertight test: slivers and flat leaves, triangles seen
edge-on, rays aimed at vertices and along edges, rays in the triangles' own
plane, meshes far from the origin or of extreme scale, rays from far away, and
degenerate or huge triangles among ordinary ones.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
OUT = ("prim", "t", "u", "v", "w")
N = 120_000


def _soup(scenes):
    return scenes.triangle_soup(6000, 21, edge=0.03)[0].reshape(-1, 3, 3)


def _slivers(scenes):
    v = _soup(scenes).astype(np.float64)
    c = v.mean(1, keepdims=True)
    k = np.exp(np.linspace(0, 14, v.shape[0]))[:, None, None]
    d = v - c
    d[:, 1:] = d[:, :1] * np.array([0.4, -0.9])[None, :, None] + d[:, 1:] / k  # flattened onto one direction
    return (c + d).astype(np.float32)


def _grid(scenes, lift=0.0):
    n = 48
    x, y = np.meshgrid(np.arange(n + 1) / n, np.arange(n + 1) / n, indexing="ij")
    z = lift * np.sin(7 * x) * np.cos(5 * y)
    p = np.stack([x, y, z], 2)
    a, b, c, d = p[:-1, :-1], p[1:, :-1], p[1:, 1:], p[:-1, 1:]
    return np.concatenate([np.stack([a, b, c], 2).reshape(-1, 3, 3), np.stack([a, c, d], 2).reshape(-1, 3, 3)])


def _mixed(scenes):
    v = _soup(scenes).copy()
    v[::11, 1] = v[::11, 0]                     # two equal vertices
    v[1::11, 2] = 0.5 * (v[1::11, 0] + v[1::11, 1])  # collinear
    v[2::13] = v[2::13, :1]                     # a point
    v[3::97] = v[3::97, :1] + (v[3::97] - v[3::97, :1]) * 40  # large ones
    v[5::601] *= 1e3
    return v


MESHES = {
    "soup": _soup,
    "slivers": _slivers,
    "flat grid": lambda s: _grid(s),
    "wavy grid": lambda s: _grid(s, 0.05),
    "tilted grid": lambda s: _grid(s) @ np.array([[0.8, 0.6, 0.0], [-0.48, 0.64, 0.6], [0.36, -0.48, 0.8]]),
    "far": lambda s: _soup(s) + np.array([3e3, -2e3, 7e3]),
    "tiny": lambda s: _soup(s) * 1e-8,
    "huge": lambda s: _soup(s).astype(np.float64) * 1e9,
    "mixed": _mixed,
}


def _rays(v, seed):
    rng = np.random.default_rng(seed)
    lo, hi = v.reshape(-1, 3).min(0), v.reshape(-1, 3).max(0)
    ext = np.maximum(hi - lo, 1e-3 * (hi - lo).max())
    tri = rng.integers(0, v.shape[0], N)
    w = rng.dirichlet((1, 1, 1), N)
    w[0::6] = np.eye(3)[rng.integers(0, 3, w[0::6].shape[0])]           # vertices
    w[1::6, 2] = 0
    w[1::6] /= w[1::6].sum(1, keepdims=True) + 1e-30                     # edge points
    p = (v[tri] * w[:, :, None]).sum(1)
    d = rng.standard_normal((N, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    e1, e2 = v[tri, 1] - v[tri, 0], v[tri, 2] - v[tri, 0]
    m = rng.standard_normal((N, 2))
    inpl = e1 * m[:, :1] + e2 * m[:, 1:]
    norm = np.linalg.norm(inpl, axis=1, keepdims=True)
    inpl = np.where(norm > 0, inpl / np.maximum(norm, 1e-300), d)
    k = slice(2, None, 6)
    d[k] = inpl[k]                                                       # in the triangle's plane
    k = slice(3, None, 6)
    d[k] = inpl[k] + 10.0 ** rng.uniform(-8, -1, (d[k].shape[0], 1)) * d[k]  # nearly in it
    dist = ext.max() * 10.0 ** rng.uniform(-3, 0.3, (N, 1))
    dist[4::30] = ext.max() * 10.0 ** rng.uniform(1, 5, dist[4::30].shape)
    r = np.empty((N, 8), np.float32)
    r[:, 0:3] = p - d * dist
    r[:, 3:6] = d
    s = slice(5, None, 12)
    r[s, 3:6] = (d * dist)[s]                                            # shadow rays: the target at t = 1
    r[:, 6] = np.inf
    r[s, 6] = 1.0
    r[7::24, 6] = (dist[7::24, 0]).astype(np.float32)                   # reach ends at the target
    r[:, 7] = 0.0
    return r


@pytest.mark.parametrize("mesh", list(MESHES))
@pytest.mark.parametrize("bias", [0.0, 1e-3])
def test_leaf_phases_agree(ctx, mesh, bias):
    from vermeer_gb300 import scenes
    v = np.asarray(MESHES[mesh](scenes), np.float32)
    g = ctx.mesh_build(v.reshape(-1, 3), np.arange(3 * v.shape[0], dtype=np.uint32), ray_bias=bias)
    rays = _rays(v.astype(np.float64), 31)
    try:
        for shadow in (False, True):
            got = {}
            for k in (0, 13, 45):
                ctx.set_tuning(kernel=k)
                got[k] = ctx.trace_mesh(g, rays, shadow=shadow)
            assert (got[0]["prim"] >= 0).sum() > N // 50
            for k in (13, 45):
                for o in OUT:
                    a, b = (x[o].view(np.uint32) if x[o].dtype == np.float32 else x[o] for x in (got[k], got[0]))
                    bad = np.nonzero(a != b)[0]
                    assert bad.size == 0, (o, k, shadow, bad.size, bad[:4] % 6, rays[bad[:2]])
    finally:
        ctx.set_tuning()
