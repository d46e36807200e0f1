"""kNN cells with small slots first (96 vertices, 160 edges; sets of more than 4096 cells): a cell
that outgrows them is done again with the full slots. Large spheres, each among 55 to 70 smaller
ones, have cells of 106 to 136 vertices and 159 to 204 edges after six kNN steps; the stores are
compared with the oracle's record for record."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def clusters(around: int, lo: float, hi: float) -> np.ndarray:
    rng = np.random.default_rng(around)
    s = [[0, 0, 0, 10]]
    for t in range(around):
        a, b = -1 + 2 * (t + 0.5) / around, np.pi * (1 + 5 ** .5) * t
        r, rad = np.sqrt(1 - a * a), rng.uniform(lo, hi)
        d = 10 + rad + rng.uniform(.2, .5)
        s.append([d * a, d * r * np.cos(b), d * r * np.sin(b), rad])
    for _ in range(100):
        p = rng.normal(size=3)
        p *= rng.uniform(20, 24) / np.linalg.norm(p)
        s.append([*p, rng.uniform(.5, 1.)])
    base, rng, out = np.array(s), np.random.default_rng(1), []
    for x, y, z in np.ndindex(3, 3, 3):
        c = base.copy()
        c[:, :3] += np.array([x, y, z]) * 50.0 + rng.normal(0, 1e-3, (c.shape[0], 3))
        out.append(c)
    return np.concatenate(out).astype(np.float32)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("around,lo,hi,steps", [(55, 2.0, 2.4, 6), (60, 2.2, 2.4, 6), (70, 2.0, 2.3, 6), (70, 2.0, 2.3, 1)])
def test_cells_that_outgrow_the_small_slots(around, lo, hi, steps, precision):
    import apo_b200
    from oracle import oracle
    sites = clusters(around, lo, hi)
    assert sites.shape[0] > 4096
    ref = oracle.build(sites, knn_steps=steps)
    assert ref["flags"] == 0 and ref["vertex_nb"].max() > 96
    algo = apo_b200.AlgorithmGPU(sites, knnValidationStep=steps, precision=precision)
    algo.build()
    for name in ("indices", "status", "vertex_nb", "edge_nb", "vertices", "edges"):
        assert np.array_equal(algo.debug_array(name), ref[name]), name
    st = algo.stats()
    assert st["error_flags"] == 0
    algo.close()


@pytest.mark.parametrize("kind", ["cells", "vertices"])
def test_filter_counts_without_the_attempts_that_are_done_again(kind):
    """The FP32 filter's counts of a build that does cells again with the full slots (kNN cells from 4096
    cells on, vertex validation from 400,000) are those of its shards, which are too small for that."""
    import apo_b200
    from apo_b200 import generators
    sites = clusters(70, 2.0, 2.3) if kind == "cells" else generators.lognormal_cloud(410000, 400.0 * (410000 / 5e6) ** (1 / 3), 3)
    counts = []
    for shards in (1, 2):
        total = [0, 0]
        for s in range(shards):
            algo = apo_b200.AlgorithmGPU(sites, knnValidationStep=6 if kind == "cells" else 1, precision="fp32", shard=(s, shards))
            algo.build()
            st = algo.stats()
            total = [total[0] + st["filter_tests"], total[1] + st["filter_escalations"]]
            algo.close()
        counts.append(total)
    assert counts[0] == counts[1] and counts[0][0] > 0
