"""Edge searches on inputs whose cells are not what the arcs between their vertices suggest. The stores are
compared with those of a build that searched the whole ball around the cell's site for every edge (digests
of its stores below, where they were also the same with the bounding sphere in the ball's place):

- sets with a tenth of the sites twice: a cell lacks vertices that a duplicate neighbour took, so the
  arc between two of the others is not all of the edge that is open;
- lattices with a jitter of 1e-4: where four centres lie in a plane but for the rounding of their
  coordinates, the root that their spheres touch comes out at any height over it.
"""
import hashlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def duplicates(n: int, seed: int, lognormal: bool) -> np.ndarray:
    rng = np.random.default_rng(seed)
    x = rng.uniform(0, 6.0 * n ** (1 / 3), (n, 3))
    r = np.clip(rng.lognormal(0, .5, n), .2, 3.) if lognormal else rng.uniform(.5, 2, n)
    q = rng.choice(n, n // 10, replace=False)
    return np.concatenate([np.concatenate([x, x[q]]), np.concatenate([r, r[q]])[:, None]], axis=1).astype(np.float32)


def stores(sites, status_ok, precision):
    import apo_b200
    algo = apo_b200.AlgorithmGPU(sites, precision=precision)
    try:
        algo.build()
        assert status_ok
    except apo_b200.Apo2Error as e:
        # two equal neighbours may leave a cell that no round validates
        assert not status_ok and e.status == apo_b200.APO2_ERR_ITER_LIMIT
    digest = hashlib.md5()
    for name in ("status", "vertex_nb", "edge_nb", "vertices", "edges"):
        digest.update(algo.debug_array(name).tobytes())
    algo.close()
    return digest.hexdigest()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,seed,lognormal,status_ok,digest", [
    (300, 35, True, True, "221f3bd51b5829a7a962bc7929acbd9e"),
    (300, 70, True, True, "2082fd94e41c33c8256c8bdf38f730f2"),
    (300, 78, True, True, "958a163bb1888a665428db0ce3cf6b39"),
    (300, 29, True, False, "b43be4703407b5b7b362290650532576"),
    (800, 4, True, False, "b8b0328e75dae157dabffe1c4e131a9f"),
    (300, 31, False, True, "7bfb29b1fce27b3345bce25da7c7053e"),
    (300, 66, False, True, "5eabca6fc4e525be0e4d7eb31646f479"),
    (300, 20, False, False, "c50df43b5c764ceb05c18bdbf564b455"),
])
def test_duplicate_sites(n, seed, lognormal, status_ok, digest, precision):
    assert stores(duplicates(n, seed, lognormal), status_ok, precision) == digest


def layered(side: int, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    x = np.stack(np.meshgrid(*[np.arange(side) * 3.] * 3, indexing="ij"), -1).reshape(-1, 3) + rng.normal(0, 1e-4, (side ** 3, 3))
    return np.concatenate([x, np.clip(rng.lognormal(0, .5, side ** 3), .2, 3.)[:, None]], axis=1).astype(np.float32)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("side,seed,digest", [
    (7, 0, "128ba5fe2085b587b6989fb2d969ba3d"),
    (7, 40, "2e51dd43199e9486b18b26e70061c732"),
    (8, 0, "9a78d0b7f0eee5fe01194b1661143c72"),
    (8, 18, "022aec58a6350f12d7dee0f2ca564e47"),
    (8, 52, "378b1854427f1ff868cc8f522eddcf01"),
    (8, 55, "b9d92b5d7458a8e79ab8de9a029c1d4e"),
])
def test_coplanar_sites(side, seed, digest, precision):
    assert stores(layered(side, seed), True, precision) == digest
