"""The four-wide form of mesh BVHs (csrc/wide_bvh.cpp) on the CPU: BVHs that it
is not built for -- nodes that share their children, which a tree walk reaches
many times over -- and how large it gets at most."""
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


def run(checker, tmp_path, nodes, triangles):
    path = tmp_path / "nodes.bin"
    path.write_bytes(np.array([len(nodes), triangles], np.uint32).tobytes() + nodes.tobytes())
    return subprocess.run([str(checker), str(path)], capture_output=True, text=True, timeout=60)


@pytest.mark.parametrize("levels", [2, 3, 20])
def test_shared_children_have_no_wide_form(checker, tmp_path, levels):
    """Both nodes of a pair have the next pair as their children."""
    nodes = np.zeros(2 * levels + 1, L.BVH_NODE)
    nodes["min"], nodes["max"] = -1.0, 1.0
    for level in range(levels):
        for i in ([0] if level == 0 else [2 * level - 1, 2 * level]):
            nodes[i]["first_index"] = 2 * level + 1
    nodes[-2:]["leaf_count"] = 1
    nodes[-1]["first_index"] = 1
    r = run(checker, tmp_path, nodes, 2)
    assert r.returncode == 0 and r.stdout == "none\n", (r.returncode, r.stdout)


@pytest.mark.parametrize("seed", range(6))
def test_most_wide_nodes(checker, tmp_path, seed):
    rng = np.random.default_rng(seed)
    positions = rng.normal(size=(3 * rng.integers(3, 900), 3)).astype(np.float32)
    indices = np.arange(len(positions), dtype=np.uint32).reshape(-1, 3)
    if seed < 2:
        positions, indices, _ = (scenes.icosphere, scenes.icosphere)[seed](2 + seed)
    m = MeshAsset.build(positions, indices)
    r = run(checker, tmp_path, m.nodes.copy(), m.triangle_count)
    assert r.returncode == 0 and "leaf hits" in r.stdout, (r.returncode, r.stdout)
    inner = int((m.nodes["leaf_count"] == 0).sum())
    assert int(r.stdout.split()[0]) <= (2 * inner + 1) // 3
