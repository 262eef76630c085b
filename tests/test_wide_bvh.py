"""The four-wide form of the mesh BVHs (csrc/wide_bvh.cpp) on the CPU: every
leaf once, and rays reach the same leaves through it as through the binary
BVH, for meshes from a few triangles to a ragged grid, flat ones and ones
with leaves of more than two triangles."""
import subprocess

import numpy as np
import pytest

from slimtracincpp_b200 import build as B
from slimtracincpp_b200 import layout as L
from slimtracincpp_b200 import scenes
from slimtracincpp_b200.scene import MeshAsset
from conftest import ROOT


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = tmp_path_factory.mktemp("wide") / "wide_bvh_check"
    subprocess.run(["g++", *B.CXX_FLAGS, "-mfma", str(ROOT / "tests" / "wide_bvh_check.cpp"), str(B.CSRC / "wide_bvh.cpp"),
                    "-o", str(exe)], check=True, capture_output=True)
    return exe


def nodes_of(name):
    if name == "icosphere":
        pos, idx, _ = scenes.icosphere(4)
    elif name == "grid":
        pos, idx, _ = scenes.heightfield(np.random.default_rng(3), 47, 0.3)
    elif name == "flat":
        pos, idx, _ = scenes.heightfield(np.random.default_rng(3), 12, 0.0)
    elif name == "tiny":
        pos, idx, _ = scenes.icosphere(3)
        pos = pos * np.float32(1e-3)
    else:
        pos, idx, _ = scenes.icosphere(0)
        idx = idx[:3]
    m = MeshAsset.build(pos, idx)
    return m.nodes.copy(), m.triangle_count


def run(checker, tmp_path, nodes, triangles, stack=64):
    path = tmp_path / "nodes.bin"
    path.write_bytes(np.array([len(nodes), triangles], np.uint32).tobytes() + nodes.tobytes())
    return subprocess.run([str(checker), str(path), str(stack)], capture_output=True, text=True)


@pytest.mark.parametrize("name", ["three", "icosphere", "grid", "flat", "tiny"])
def test_rays_reach_the_same_leaves(checker, tmp_path, name):
    nodes, triangles = nodes_of(name)
    assert nodes.dtype == L.BVH_NODE
    r = run(checker, tmp_path, nodes, triangles)
    assert r.returncode == 0 and "leaf hits" in r.stdout, (r.returncode, r.stdout)


def test_wide_leaves(checker, tmp_path):
    """Leaves of up to eight triangles: the bottom of an icosphere's BVH merged."""
    nodes, triangles = nodes_of("icosphere")
    merged, stack = [nodes[0].copy()], [(0, 0)]

    def span(i):
        n = nodes[i]
        if n["leaf_count"]:
            return int(n["first_index"]), int(n["leaf_count"])
        (a, ca), (b, cb) = span(int(n["first_index"])), span(int(n["first_index"]) + 1)
        return min(a, b), ca + cb

    while stack:
        src, dst = stack.pop()
        first, count = span(src)
        if count <= 8:
            merged[dst]["first_index"], merged[dst]["leaf_count"] = first, count
            continue
        merged[dst]["first_index"] = len(merged)
        for c in (int(nodes[src]["first_index"]), int(nodes[src]["first_index"]) + 1):
            merged.append(nodes[c].copy())
            stack.append((c, len(merged) - 1))
    r = run(checker, tmp_path, np.array(merged, L.BVH_NODE), triangles)
    assert r.returncode == 0 and "leaf hits" in r.stdout, (r.returncode, r.stdout)


@pytest.mark.parametrize("fault", ["not nested", "nan", "huge"])
def test_refused_boxes(checker, tmp_path, fault):
    nodes, triangles = nodes_of("grid")
    k = len(nodes) // 2
    nodes[k]["max"][1] = {"not nested": 50.0, "nan": np.nan, "huge": 3e30}[fault]
    r = run(checker, tmp_path, nodes, triangles)
    assert r.returncode == 0 and r.stdout.strip() == "none", (r.returncode, r.stdout)


def test_refused_when_the_stack_is_too_small(checker, tmp_path):
    nodes, triangles = nodes_of("grid")
    out = [run(checker, tmp_path, nodes, triangles, stack).stdout.strip() == "none" for stack in (4, 12, 64)]
    assert out[0] and not out[2], out
