"""Edge and bisector searches over the regions that bound them, against the oracle's stores record for
record, on clouds whose trisectors take every kind of region: equal radii (an arc adds nothing to
its ends), radii over two orders of magnitude (elliptic arcs, and sites of very different size
under the same box), a flat slab (edges of hull cells, whose ends lie far apart), and a shell of small
spheres around a large one (radii far below the edge's own)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cloud(kind: str, n: int, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    side = 6.0 * n ** (1 / 3)
    xyz = rng.uniform(0, side, (n, 3))
    r = np.full(n, 1.0)
    if kind == "wide":
        r = 10 ** rng.uniform(-1.5, 0.7, n)
    elif kind == "slab":
        xyz[:, 2] *= 0.05
        r = rng.uniform(0.2, 1.5, n)
    elif kind == "shell":
        d = rng.normal(size=(n, 3))
        xyz = d / np.linalg.norm(d, axis=1)[:, None] * rng.uniform(32, 40, n)[:, None]
        xyz[0] = 0
        r = rng.uniform(0.3, 1.0, n)
        r[0] = 30.0
    return np.concatenate([xyz, r[:, None]], axis=1).astype(np.float32)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind,n,seed", [("equal", 700, 1), ("wide", 900, 2), ("slab", 700, 3), ("shell", 60, 4)])
def test_stores_match_the_oracle(kind, n, seed, precision):
    import apo_b200
    from oracle import oracle
    sites = cloud(kind, n, seed)
    ref = oracle.build(sites)
    assert ref["flags"] == 0
    algo = apo_b200.AlgorithmGPU(sites, precision=precision)
    algo.build()
    for name in ("indices", "status", "vertex_nb", "edge_nb", "vertices", "edges"):
        assert np.array_equal(algo.debug_array(name), ref[name]), name
    assert np.array_equal(algo.toHost().verticesId, ref["out_vertices_id"])
    algo.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_searches_handed_to_a_warp(precision):
    """Long searches (edges of hull cells whose bounds cover much of the cloud): set up again by the warp
    that they go to, whichever way it would decide whether the security radius covers them."""
    import apo_b200
    from apo_b200 import generators
    from oracle import oracle
    sites = generators.uniform_random(3000, 66.9, 0.5, 2.0, 5)
    ref = oracle.build(sites)
    assert ref["flags"] == 0
    algo = apo_b200.AlgorithmGPU(sites, precision=precision)
    algo.build()
    for name in ("indices", "status", "vertex_nb", "edge_nb", "vertices", "edges"):
        assert np.array_equal(algo.debug_array(name), ref[name]), name
    algo.close()
