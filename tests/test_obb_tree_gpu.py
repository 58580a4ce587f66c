"""GPU parity of the AABB-BVH -> OBB-tree transform and of the node collapse
against the oracle restatement, through the reference entry points
kr_cuda_bvh_obb_tree and kr_cuda_bvh_collapse."""
import numpy as np
import pytest

from conftest import contained, same_bits, uncontained_leaves
from oracle import bvh as ref
from obvh_b200 import bvh, workloads
from test_build_gpu import _shapes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def builder():
    import torch
    assert torch.cuda.is_available()
    return bvh.LbvhBuilder()


def _lbvh(builder, v, f):
    mesh = bvh.Mesh(v, f)
    tree = builder.build(mesh)
    return mesh, tree


def _tree_numpy(tree):
    return bvh.nodes_numpy(tree["nodes"]), tree["parents"].cpu().numpy().view(np.uint32)


def _check_obbs(mesh, tree, v, f, sample_leaves=None):
    obbs, xfs = bvh.obb_tree(mesh, tree)
    nodes, parents = _tree_numpy(tree)
    want_o, want_x, _ = ref.obb_tree(nodes, parents, v, f)
    got_o, got_x = obbs.cpu().numpy(), xfs.cpu().numpy()
    assert same_bits(got_o, want_o)
    assert same_bits(got_x, want_x)
    # every vertex lies in its leaf's box and in every ancestor's box
    n = (len(parents) + 1) // 2
    f4 = bvh.as_faces4(f)
    if sample_leaves is None:
        assert uncontained_leaves(v, f4, nodes["left"][n - 1:], parents, got_o) == 0
        return got_o
    for j in np.random.default_rng(0).choice(n, sample_leaves, replace=False):
        tri = v[f4[nodes["left"][n - 1 + j], :3]]
        node = n - 1 + j
        while node != 0xFFFFFFFF:
            assert contained(tri, got_o[node]), (j, node)
            node = parents[node]
    return got_o


@pytest.mark.parametrize("n", [1, 2, 3, 9, 100, 5000, 100_003])
def test_obb_tree_soup(builder, n):
    v, f = workloads.triangle_soup(n, seed=100 + n)
    mesh, tree = _lbvh(builder, v, f)
    _check_obbs(mesh, tree, v, f)


def test_obb_tree_full_size(builder):
    """The 2M-triangle LBVH + OBB-tree workload: every vertex of every leaf
    inside its leaf's box and every ancestor's box (FP64)."""
    v, f = workloads.triangle_soup(2_000_000, seed=1)
    mesh, tree = _lbvh(builder, v, f)
    _check_obbs(mesh, tree, v, f)


def test_obb_tree_mesh(builder):
    v, f = workloads.torus_knot_mesh(segments=256, around=112)
    mesh, tree = _lbvh(builder, v, f)
    _check_obbs(mesh, tree, v, f)


def _random_tree(n, rng):
    """A binary tree whose depth-first leaf order is not the leaf index order."""
    ni = n - 1
    nodes = np.zeros(2 * n - 1, ref.NODE)
    parents = np.full(2 * n - 1, 0xFFFFFFFF, np.uint32)
    leaf_ids = list(rng.permutation(n) + ni)
    nodes["left"][ni:] = rng.permutation(n)
    nodes["n_prims"][ni:] = 1
    nxt = [1]

    def build_at(idx, items):
        if len(items) == 2:
            l, r = items
        else:
            cut = int(rng.integers(1, len(items)))
            kids = []
            for part in (items[:cut], items[cut:]):
                if len(part) == 1:
                    kids.append(part[0])
                else:
                    kids.append(nxt[0])
                    nxt[0] += 1
                    build_at(kids[-1], part)
            l, r = kids
        nodes["left"][idx], nodes["right"][idx] = l, r
        parents[l] = parents[r] = idx

    import sys
    sys.setrecursionlimit(100000)
    build_at(0, leaf_ids)
    return nodes, parents


def test_obb_tree_on_a_non_morton_tree():
    """kr_cuda_bvh_obb_tree on a tree not built by the LBVH (e.g. a restructured one)."""
    import torch
    rng = np.random.default_rng(3)
    n = 3000
    v, f = workloads.triangle_soup(n, seed=8)
    nodes, parents = _random_tree(n, rng)
    f4 = bvh.as_faces4(f)
    for j in range(n):  # leaf bounds (unused by the transform, kept valid)
        tri = v[f4[nodes["left"][n - 1 + j], :3]]
        nodes["b"][n - 1 + j] = np.concatenate([tri.min(0), tri.max(0)])
    mesh = bvh.Mesh(v, f)
    tree = {"nodes": torch.from_numpy(nodes.view(np.uint8).copy()).cuda(),
            "parents": torch.from_numpy(parents.view(np.int32).copy()).cuda()}
    obbs, xfs = bvh.obb_tree(mesh, tree)
    want_o, want_x, _ = ref.obb_tree(nodes, parents, v, f)
    assert same_bits(obbs.cpu().numpy(), want_o)
    assert same_bits(xfs.cpu().numpy(), want_x)


@pytest.mark.parametrize("n", [2, 31, 32, 33, 255, 257, 1000])
@pytest.mark.parametrize("spread", [0, 3, 100])
def test_obb_tree_where_siblings_meet_in_a_warp_and_across(n, spread):
    """Neighbours in depth-first order `spread` leaf numbers apart on average:
    from walks that all meet within a warp to walks that never do."""
    import torch
    rng = np.random.default_rng(1000 * spread + n)
    v, f = workloads.triangle_soup(n, seed=n)
    nodes, parents = _random_tree(n, rng)
    # leaves renumbered: depth-first rank, jittered by `spread`
    order, stack = [], [0]
    while stack:
        k = stack.pop()
        if k >= n - 1:
            order.append(k)
        else:
            stack += [int(nodes["right"][k]), int(nodes["left"][k])]
    new = np.empty(n, np.int64)
    rank = np.argsort(np.argsort(np.arange(n) + rng.uniform(0, spread, n), kind="stable"), kind="stable")
    new[np.array(order) - (n - 1)] = n - 1 + rank
    for side in ("left", "right"):
        kids = nodes[side][:n - 1].astype(np.int64)
        nodes[side][:n - 1] = np.where(kids >= n - 1, new[np.maximum(kids, n - 1) - (n - 1)], kids)
    nodes["left"][n - 1:] = rng.permutation(n)
    parents[:] = 0xFFFFFFFF
    for k in range(n - 1):
        parents[nodes["left"][k]] = parents[nodes["right"][k]] = k
    mesh = bvh.Mesh(v, f)
    tree = {"nodes": torch.from_numpy(nodes.view(np.uint8).copy()).cuda(),
            "parents": torch.from_numpy(parents.view(np.int32).copy()).cuda()}
    obbs, xfs = bvh.obb_tree(mesh, tree)
    want_o, want_x, _ = ref.obb_tree(nodes, parents, v, f)
    assert same_bits(obbs.cpu().numpy(), want_o)
    assert same_bits(xfs.cpu().numpy(), want_x)


@pytest.mark.parametrize("kind", ["sheet", "turned", "shell", "large"])
@pytest.mark.parametrize("n", [8, 9, 32, 33, 511, 513, 5000])
def test_obb_tree_extents_by_groups_units_and_blocks(builder, kind, n):
    """Around the sizes of a thread's, a group's and a unit's nodes."""
    v, f = _shapes(kind, n, n)
    mesh, tree = _lbvh(builder, v, f)
    obbs, xfs = bvh.obb_tree(mesh, tree)
    nodes, parents = _tree_numpy(tree)
    want_o, want_x, _ = ref.obb_tree(nodes, parents, v, f)
    assert same_bits(obbs.cpu().numpy(), want_o)
    assert same_bits(xfs.cpu().numpy(), want_x)


def _chain(n):
    """A tree as deep as it has leaves: internal node k holds leaf k and node k + 1."""
    nodes = np.zeros(2 * n - 1, ref.NODE)
    parents = np.full(2 * n - 1, 0xFFFFFFFF, np.uint32)
    k = np.arange(n - 1)
    nodes["left"][:n - 1], nodes["right"][:n - 1] = n - 1 + k, np.append(k[1:], 2 * n - 2)
    nodes["left"][n - 1:], nodes["n_prims"][n - 1:] = np.arange(n), 1
    parents[nodes["left"][:n - 1]] = parents[nodes["right"][:n - 1]] = k
    return nodes, parents


def test_obb_tree_of_a_chain_costs_little_more_than_its_collapse():
    """One walk a level all the way up, every sibling a leaf.  The collapse of the
    same tree is such a walk too, without slabs: the transform took 1.19 times
    its time with a lane for a walk, and 1.50 where a group's lanes took turns
    at a leaf's slabs."""
    import torch
    n = 5000
    v, f = workloads.triangle_soup(n, seed=8)
    nodes, parents = _chain(n)
    tri = v[bvh.as_faces4(f)[:, :3]]
    nodes["b"][n - 1:] = np.concatenate([tri.min(1), tri.max(1)], 1)
    mesh = bvh.Mesh(v, f)
    tree = {"nodes": torch.from_numpy(nodes.view(np.uint8).copy()).cuda(),
            "parents": torch.from_numpy(parents.view(np.int32).copy()).cuda(),
            "counts": torch.zeros(2 * n - 1, dtype=torch.int32, device="cuda"),
            "costs": torch.zeros(2 * n - 1, device="cuda")}
    obbs, xfs = bvh.obb_tree(mesh, tree)
    want_o, want_x, _ = ref.obb_tree(nodes, parents, v, f)
    assert same_bits(obbs.cpu().numpy(), want_o)
    assert same_bits(xfs.cpu().numpy(), want_x)
    times = ([], [])
    for _ in range(7):  # in turn, the medians compared
        for k, call in enumerate((lambda: bvh.obb_tree(mesh, tree, obbs, xfs), lambda: bvh.collapse(tree))):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call()
            b.record()
            b.synchronize()
            times[k].append(a.elapsed_time(b))
    assert np.median(times[0]) < 1.35 * np.median(times[1]), (np.median(times[0]), np.median(times[1]))


def test_obb_tree_rejects_a_parent_cycle():
    """A malformed tree ends with an error from the bounded walks, not a hang."""
    import torch
    from obvh_b200 import ObvhError
    n = 64
    v, f = workloads.triangle_soup(n, seed=9)
    rng = np.random.default_rng(4)
    nodes, parents = _random_tree(n, rng)
    parents[5] = 5  # internal node 5 is its own parent
    mesh = bvh.Mesh(v, f)
    tree = {"nodes": torch.from_numpy(nodes.view(np.uint8).copy()).cuda(),
            "parents": torch.from_numpy(parents.view(np.int32).copy()).cuda()}
    with pytest.raises(ObvhError, match="cycle|malformed"):
        bvh.obb_tree(mesh, tree)
    # the library stays usable afterwards
    v2, f2 = workloads.triangle_soup(100, seed=10)
    b = bvh.LbvhBuilder()
    mesh2 = bvh.Mesh(v2, f2)
    bvh.obb_tree(mesh2, b.build(mesh2))


@pytest.mark.parametrize("n", [2, 3, 50, 5000, 200_003])
def test_collapse(builder, n):
    v, f = workloads.triangle_soup(n, seed=200 + n)
    mesh, tree = _lbvh(builder, v, f)
    nodes, parents = _tree_numpy(tree)
    counts0 = tree["counts"].cpu().numpy().view(np.uint32).copy()
    costs0 = tree["costs"].cpu().numpy().copy()
    out = bvh.collapse(tree, 1.2, 1.0, metrics=True)
    col_w, cnt_w, prim_w, cost_w, used = ref.collapse(nodes, parents, counts0, costs0, 1.2, 1.0)
    col = bvh.nodes_numpy(out["collapsed"])
    assert same_bits(col["b"], col_w["b"])
    assert np.array_equal(col["left"], col_w["left"])
    assert np.array_equal(col["right"][: n - 1], col_w["right"][: n - 1])
    assert np.array_equal(col["n_prims"], col_w["n_prims"])
    assert np.array_equal(tree["counts"].cpu().numpy().view(np.uint32), cnt_w)
    assert same_bits(tree["costs"].cpu().numpy(), cost_w)
    assert np.array_equal(out["primitives"].cpu().numpy().view(np.uint32)[:used], prim_w[:used])
    assert out["metrics"][0] >= 0 and out["metrics"][1] >= 0


def test_collapse_full_size(builder):
    v, f = workloads.triangle_soup(2_000_000, seed=1)
    mesh, tree = _lbvh(builder, v, f)
    nodes, parents = _tree_numpy(tree)
    counts0 = tree["counts"].cpu().numpy().view(np.uint32).copy()
    costs0 = tree["costs"].cpu().numpy().copy()
    out = bvh.collapse(tree)
    col_w, cnt_w, prim_w, cost_w, used = ref.collapse(nodes, parents, counts0, costs0)
    col = bvh.nodes_numpy(out["collapsed"])
    assert np.array_equal(col["n_prims"], col_w["n_prims"]) and np.array_equal(col["left"], col_w["left"])
    assert np.array_equal(out["primitives"].cpu().numpy().view(np.uint32)[:used], prim_w[:used])
    assert same_bits(tree["costs"].cpu().numpy(), cost_w)
