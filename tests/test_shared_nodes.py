"""Uploaded trees that reach a node more than once.

A tree of n nodes has at most 4n + 1 entries (nodes and leaves); a ray that takes
more than 4n + 2 ends the call with VMR_ERR_TIMEOUT, whatever the tuning, and one
that takes exactly that many does not.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TIMEOUT = -4
KERNELS = (0, 1, 13, 29, 37, 45)


def _leaf(k):
    return -(1 << 31) | (k << 4)


def _tree(shared, leaves, n_leaf_ids):
    """Two nodes: the root holds the second one `shared` times, which holds
    `leaves` leaves of one element each.  Entries: 1 + shared * (1 + leaves)."""
    inner = [1] * shared + [-1] * (4 - shared)
    leaf = [_leaf(k % n_leaf_ids) for k in range(leaves)] + [-1] * (4 - leaves)
    return np.array([inner, leaf], np.int64).astype(np.int32)


def _boxes(nodes, keys=1):
    b = np.empty((keys, nodes, 24), np.float32)
    b[..., :12], b[..., 12:] = -10, 10
    return b


def _nodes(children, dtype):
    n = np.zeros(len(children), dtype)
    n["children"] = children
    n["axis"] = (0, 1, 2)
    if "boxes" in n.dtype.names:
        n["boxes"] = _boxes(len(children))[0]
    return n


def _mesh(ctx, children, keys):
    """Four triangles that no ray of _rays meets, under the given tree."""
    import vermeer_gb300 as vg
    v = np.tile(np.array([[9, 9, 9], [9.01, 9, 9], [9, 9.01, 9]], np.float32), (4 * keys, 1))
    idx, acc = np.arange(12, dtype=np.uint32), np.arange(4, dtype=np.int32)
    bounds = np.array([[-10] * 3 + [10] * 3] * keys, np.float32)
    if keys == 1:
        return ctx.mesh_upload(v, idx, acc, nodes=_nodes(children, vg.NODE_DTYPE), bounds=bounds)
    return ctx.mesh_upload(v, idx, acc, mnodes=_nodes(children, vg.MNODE_DTYPE), mboxes=_boxes(len(children), keys),
                           bounds=bounds, keys=keys, motion_mode=1)


def _rays(n):
    from vermeer_gb300 import scenes
    r = scenes.incoherent_rays(n, 5)
    r[:, 5] = -np.abs(r[:, 5])
    r[:, 7] = 0.5
    return r


def _codes(ctx, trace):
    import vermeer_gb300 as vg
    out = []
    try:
        for k in KERNELS:
            ctx.set_tuning(kernel=k)
            for shadow in (False, True):
                try:
                    r = trace(shadow)
                    assert (r["prim"] == -1).all()
                    out.append(0)
                except vg.VmrError as e:
                    out.append(e.code)
    finally:
        ctx.set_tuning()
    return out


# 10 is the cap of two nodes
@pytest.mark.parametrize("shared,leaves,refused", [(1, 4, False), (3, 2, False), (2, 4, True), (3, 3, True),
                                                   (4, 4, True)])
@pytest.mark.parametrize("keys", [1, 2])
@pytest.mark.parametrize("n", [1, 5000])
def test_entries_beyond_the_cap_are_refused(ctx, shared, leaves, refused, keys, n):
    import vermeer_gb300 as vg
    from vermeer_gb300 import scenes
    g = _mesh(ctx, _tree(shared, leaves, 4), keys)
    rays = _rays(n)
    want = [TIMEOUT if refused else 0] * (2 * len(KERNELS))
    assert _codes(ctx, lambda s: ctx.trace_mesh(g, rays, shadow=s)) == want
    other = ctx.mesh_build(*scenes.triangle_soup(3, 4, lo=20, hi=21, edge=0.01))
    ctx.scene_build([g, other])
    assert _codes(ctx, lambda s: ctx.trace_scene(rays, shadow=s)) == want
    # the same tree as the top level, its leaves whole meshes that are not met
    geoms = [_mesh(ctx, _tree(1, 1, 4), keys) for _ in range(4)]
    if keys == 1:
        ctx.scene_upload(np.array(geoms, np.uint32), nodes=_nodes(_tree(shared, leaves, 4), vg.NODE_DTYPE))
    else:
        ctx.scene_upload(np.array(geoms, np.uint32), mnodes=_nodes(_tree(shared, leaves, 4), vg.MNODE_DTYPE),
                         mboxes=_boxes(2, keys), keys=keys)
    assert _codes(ctx, lambda s: ctx.trace_scene(rays, shadow=s)) == want
