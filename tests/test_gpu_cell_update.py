"""Cell update at the edges of its fast paths, against the oracle's stores record for record:

- updates that give about 32 new-edge candidates (two per new vertex), the most a warp handles with
  one candidate per lane; more are sorted: a ring of small spheres around the face of two large
  ones, which is then cut by one of them;
- cells with about 80 neighbours, the slots of the neighbour list; more are read from the edges: a
  large sphere surrounded by small ones, with tiny ones between it and a second large sphere (each
  adds a neighbour with a closed edge and no vertex, so the store's limits are not reached).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ringed(ring: int) -> np.ndarray:
    rng = np.random.default_rng(3)
    radius, gap = 10.0, 2.2
    s = [[-(radius + gap / 2), 0, 0, radius], [radius + gap / 2, 0, 0, radius]]
    for a in 2 * np.pi * (np.arange(ring) + rng.uniform(-.2, .2, ring)) / ring:
        s.append([rng.uniform(-.2, .2), 6 * np.cos(a), 6 * np.sin(a), 0.8 + rng.uniform(0, .05)])
    return np.array(s, dtype=np.float32)


def crowded(around: int, between: int) -> np.ndarray:
    rng = np.random.default_rng(3)
    s = [[0, 0, 0, 10], [20.3, 0, 0, 10]]
    for t in range(around):
        a, b = -1 + 1.75 * (t + 0.5) / around, np.pi * (1 + 5 ** .5) * t
        r, d = np.sqrt(1 - a * a), 11.6 + rng.uniform(0, .3)
        s.append([d * a, d * r * np.cos(b), d * r * np.sin(b), 0.6 + rng.uniform(0, .2)])
    side = int(np.ceil(np.sqrt(between)))
    for q in range(between):
        y, z = (q // side - (side - 1) / 2) * .62, (q % side - (side - 1) / 2) * .62
        s.append([10.15 + rng.uniform(-.01, .01), y + rng.uniform(-.03, .03), z + rng.uniform(-.03, .03), 0.05])
    return np.array(s, dtype=np.float32)


def check(sites, steps, precision):
    import apo_b200
    from oracle import oracle
    ref = oracle.build(sites, knn_steps=steps)
    assert ref["flags"] == 0
    algo = apo_b200.AlgorithmGPU(sites, knnValidationStep=steps, precision=precision)
    algo.build()
    for name in ("indices", "status", "vertex_nb", "edge_nb", "vertices", "edges"):
        assert np.array_equal(algo.debug_array(name), ref[name]), name
    assert np.array_equal(algo.toHost().verticesId, ref["out_vertices_id"])
    algo.close()
    return ref


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("ring", [8, 9, 11, 13])
def test_updates_around_32_candidates(ring, precision):
    check(ringed(ring), 1, precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("around,between,steps", [(60, 16, 1), (60, 16, 8), (64, 20, 8)])
def test_cells_around_80_neighbours(around, between, steps, precision):
    ref = check(crowded(around, between), steps, precision)
    most = 0
    at = 0
    for n in ref["edge_nb"].astype(int):
        most = max(most, np.unique(ref["edges"].reshape(-1, 4)[at:at + n, :2]).size)
        at += n
    assert (most > 80) == (around == 64) and most > 75
