"""Performance cases of the diagram build: what a user of this library has it do, through its
public entry points, over the range of sizes, clouds, types and forms that it is used with.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs and the handle a program keeps
    run(state)          one pass, and its outputs
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   64-bit values of the outputs, where they exist

Clouds (all seeded, apo_b200/generators.py): "uniform" -- uniform centres and radii, the
reference's benchmark and precision clouds; "protein" -- self-avoiding chains with van der Waals
radii at 0.01 atoms per cubic angstrom; "lognormal" -- uniform centres, log-normal radii, at the
density of the 5M-site evaluation cloud (5e6 sites in a cube of 400); "lattice" -- jittered
cubic lattice of tangent spheres (nearly degenerate everywhere).

Calls:
    "one_call"  computeApolloniusDiagram / computeFullApolloniusDiagram on host sites: everything
                is set up and given back inside the call
    "object"    AlgorithmGPU(sites), build(), toHostFull(): the reference's own usage
    "rebuild"   a handle kept over changing sites (a trajectory): new sites from device memory,
                build and extraction, the outputs left on the device
    "batch"     Batch.build over many small diagrams of uneven size
    "cavity"    occlusion ratios and cavity vertices of a built diagram
    "check"     interval certificate and vertex error of a built diagram's vertices
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import apo_b200
from apo_b200 import generators, proposal

# output vertices per site of each cloud, rounded (for the byte counts; the layout of the output
# is 32 bytes of position and 16 bytes of ids per vertex)
_VERTICES_PER_SITE = {"uniform": 6.4, "protein": 6.7, "lognormal": 4.9, "lattice": 6.0}
# FP64 operations of one tangent-sphere solve and of one conflict test against a neighbour
_SOLVE, _TEST, _NEIGHBOURS = 216, 11, 16


def listed() -> list[dict]:
    return [
        # the smallest call: the reference's 100-site precision cloud (25^3, r 1..3), one call from
        # host doubles to host arrays; latency, allocation and launches are all of it
        {"name": "one_call_100", "call": "one_call", "full": False, "cloud": "uniform", "sites": 100, "side": 25.0,
         "rmin": 1.0, "rmax": 3.0, "dtype": "f64", "form": "plain"},
        # the 1,000-site precision cloud (50^3, overlapping spheres, some buried), vertices and
        # closed edges
        {"name": "one_call_full_1000", "call": "one_call", "full": True, "cloud": "uniform", "sites": 1000, "side": 50.0,
         "rmin": 1.0, "rmax": 3.0, "dtype": "f64", "form": "plain"},
        # the reference's own 10,000-site benchmark cloud (100^3, r 0.5..2), rebuilt in place
        {"name": "rebuild_uniform_10k", "call": "rebuild", "cloud": "uniform", "sites": 10000, "side": 100.0,
         "rmin": 0.5, "rmax": 2.0, "dtype": "f32", "form": "plain"},
        # 100,000 uniform sites at the same density, double input
        {"name": "rebuild_uniform_100k", "call": "rebuild", "cloud": "uniform", "sites": 100000, "side": 215.443469,
         "rmin": 0.5, "rmax": 2.0, "dtype": "f64", "form": "plain"},
        # a mid-sized protein the way the reference's applications build it: object, build, arrays
        # on the host (an odd number of sites)
        {"name": "object_protein_61k", "call": "object", "cloud": "protein", "sites": 61237, "dtype": "f64", "form": "plain"},
        # a capsid-sized packing, the largest protein of the reference's benchmark
        {"name": "rebuild_protein_1m", "call": "rebuild", "cloud": "protein", "sites": 1000000, "dtype": "f32", "form": "plain"},
        # the evaluation cloud's density at 800,000 sites: the heaviest case (a pass takes 0.6 to 1.4 s,
        # as the seed's longest edge search does)
        {"name": "rebuild_lognormal_800k", "call": "rebuild", "cloud": "lognormal", "sites": 800000, "dtype": "f32",
         "form": "plain"},
        # the benchmark's headline form (learned k-proposal and FP32 filter) on the same cloud
        {"name": "rebuild_lognormal_300k_forms", "call": "rebuild", "cloud": "lognormal", "sites": 300001, "dtype": "f32",
         "form": "learned_fp32"},
        # nearly degenerate input: 46^3 tangent spheres
        {"name": "rebuild_lattice_46", "call": "rebuild", "cloud": "lattice", "sites": 46 ** 3, "dtype": "f32", "form": "plain"},
        # many small proteins of uneven size in one call (200 to 50,000 sites, log-uniform)
        {"name": "batch_28", "call": "batch", "cloud": "protein", "sites": 28 * 9000, "diagrams": 28, "largest": 50000,
         "dtype": "f32", "form": "plain"},
        # the cavity application on a 100,000-atom packing
        {"name": "cavity_protein_100k", "call": "cavity", "cloud": "protein", "sites": 100000, "samples": 64, "dtype": "f32",
         "form": "plain"},
        # the checks a user runs on a finished diagram
        {"name": "check_lognormal_200k", "call": "check", "cloud": "lognormal", "sites": 200003, "dtype": "f32", "form": "plain"},
    ]


def _log_size(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    call = rng.choice(["one_call", "one_call", "object", "rebuild", "rebuild", "rebuild", "rebuild", "batch", "cavity", "check"])
    form = "plain"
    if call == "one_call":
        n = _log_size(rng, 50, 4000)
        # the precision clouds' two densities: overlapping spheres, and mixed radii far apart
        dense = rng.random() < 0.6
        return {"call": call, "full": rng.random() < 0.5, "cloud": "uniform", "sites": n,
                "side": (5.4 if dense else 20.0) * n ** (1 / 3), "rmin": 1.0 if dense else 0.1,
                "rmax": 3.0 if dense else 10.0, "dtype": rng.choice(["f32", "f64"]), "form": form}
    if call == "batch":
        d = rng.randint(8, 28)
        return {"call": call, "cloud": "protein", "sites": 9000 * d, "diagrams": d, "largest": _log_size(rng, 5000, 50000),
                "dtype": "f32", "form": rng.choice(["plain", "plain", "learned_fp32"])}
    if call == "cavity":
        return {"call": call, "cloud": "protein", "sites": _log_size(rng, 10000, 200000), "samples": rng.choice([32, 64, 100]),
                "dtype": "f32", "form": form}
    if call == "check":
        return {"call": call, "cloud": rng.choice(["protein", "lognormal"]), "sites": _log_size(rng, 20000, 300000),
                "dtype": "f32", "form": form}
    if call == "object":
        return {"call": call, "cloud": rng.choice(["protein", "lognormal"]), "sites": _log_size(rng, 5000, 150000),
                "dtype": rng.choice(["f32", "f64"]), "form": form}
    cloud = rng.choice(["uniform", "protein", "protein", "lognormal", "lognormal", "lattice"])
    case = {"call": call, "cloud": cloud, "dtype": rng.choice(["f32", "f64"]),
            "form": rng.choice(["plain", "plain", "fp32", "learned", "learned_fp32"])}
    if cloud == "lattice":
        case["sites"] = rng.randint(15, 48) ** 3
    elif cloud == "uniform":
        n = _log_size(rng, 2000, 150000)
        case.update(sites=n, side=round(100.0 * (n / 10000) ** (1 / 3), 6), rmin=0.5, rmax=2.0)
    else:
        case["sites"] = _log_size(rng, 10000, 900000 if cloud == "protein" else 700000)
    return case


def _cloud(case: dict, n: int, seed: int) -> np.ndarray:
    """(n, 4) sites of the case's cloud in its input type."""
    if case["cloud"] == "uniform":
        sites = generators.uniform_random(n, case["side"], case["rmin"], case["rmax"], seed)
    elif case["cloud"] == "protein":
        atoms = 500 if n >= 20000 else 100
        sites = generators.protein_chains(-(-n // atoms), atoms, 0.01, seed=seed + 1)[:n]
    elif case["cloud"] == "lognormal":
        sites = generators.lognormal_cloud(n, 400.0 * (n / 5e6) ** (1 / 3), seed)
    else:
        sites = generators.lattice(round(n ** (1 / 3)), "A", seed)
    if case["dtype"] == "f64":
        # a double input that a float cannot hold exactly
        return generators.joggle_sites(sites, 1e-5)
    return np.ascontiguousarray(sites)


def _batch_sites(case: dict, seed: int) -> list[np.ndarray]:
    """Log-uniform sizes in [200, largest], scaled down together to the case's total of sites."""
    sizes = generators.batch_sizes(case["diagrams"], 200, case["largest"], seed)
    scale = min(1.0, case["sites"] / float(sizes.sum()))
    return [_cloud(case, max(200, int(s * scale)), seed * 1000 + d) for d, s in enumerate(sizes)]


# A program that keeps its results keeps buffers of a fixed size for them, since the counts change
# with the sites: eight vertices per site, as the library's own, and a count.
def _rows(case: dict) -> tuple[int, int]:
    return 8 * case["sites"] + 1024, case["sites"] // 16 + 1024


def _host_frame(case: dict) -> dict:
    vertices, closed = _rows(case)
    return {"counts": np.zeros(2, np.int64), "positions": np.zeros((vertices, 4)), "ids": np.zeros((vertices, 4), np.int32),
            "closed_positions": np.zeros((closed, 4)), "closed_ids": np.zeros((closed, 3), np.int32)}


def _device_frame(case: dict) -> dict:
    return {k: torch.from_numpy(v).cuda() for k, v in _host_frame(case).items() if k != "counts" and k != "closed_ids"} | {
        "closed_ids": torch.zeros((_rows(case)[1], 4), dtype=torch.int32, device="cuda")}


def _store(frame: dict, diagram) -> dict:
    """A host diagram's arrays in the program's buffers (the fourth id of a closed edge is unused)."""
    v = diagram.verticesId.size // 4
    frame["positions"][:v] = diagram.vertices.reshape(-1, 4)
    frame["ids"][:v] = diagram.verticesId.reshape(-1, 4)
    c = 0
    if isinstance(diagram, apo_b200.FullDiagram):
        c = diagram.closedEdgesId.size // 4
        frame["closed_positions"][:c] = diagram.closedEdgesMin.reshape(-1, 4)
        frame["closed_ids"][:c] = diagram.closedEdgesId.reshape(-1, 4)[:, :3]
    frame["counts"][:] = v, c
    return frame


def prepare(case: dict, seed: int) -> dict:
    state = {"case": case}
    precision = "fp32" if "fp32" in case["form"] else "fp64"
    model = proposal.Model.load() if "learned" in case["form"] else None
    if case["call"] == "batch":
        state["diagrams"] = _batch_sites(case, seed)
        state["batch"] = apo_b200.Batch(max(s.shape[0] for s in state["diagrams"]), streams=8, precision=precision,
                                        proposal=model)
        state["frame"] = _host_frame(case)
        return state
    sites = _cloud(case, case["sites"], seed)
    if case["call"] in ("one_call", "object"):
        state["sites"] = sites
        state["frame"] = _host_frame(case)
        return state
    algo = apo_b200.AlgorithmGPU(sites, precision=precision)
    if model is not None:
        proposal.attach(algo, model)
    state["algo"] = algo
    if case["call"] == "rebuild":
        state["sites"] = torch.from_numpy(sites).cuda()
        state["frame"] = _device_frame(case)
    else:
        _build(algo)
        rows = _rows(case)[0]
        if case["call"] == "cavity":
            state["frame"] = {"ratios": np.zeros(rows, np.float32), "cavities": np.zeros((rows, 4), np.float32)}
        else:
            state["frame"] = {"flags": np.zeros(rows, np.uint8), "errors": np.zeros(rows, np.float32)}
    torch.cuda.synchronize()
    return state


def _build(algo) -> int:
    """A build's status; cells left over after the last round leave the diagram as it is."""
    try:
        algo.build()
    except apo_b200.Apo2Error as e:
        if e.status != apo_b200.APO2_ERR_ITER_LIMIT:
            raise
        return e.status
    return apo_b200.APO2_OK


def run(state: dict):
    case, frame = state["case"], state["frame"]
    call = case["call"]
    if call == "one_call":
        compute = apo_b200.computeFullApolloniusDiagram if case["full"] else apo_b200.computeApolloniusDiagram
        try:
            return apo_b200.APO2_OK, _store(frame, compute(state["sites"]))
        except apo_b200.Apo2Error as e:
            if e.status != apo_b200.APO2_ERR_ITER_LIMIT:
                raise
            return e.status, frame
    if call == "object":
        algo = apo_b200.AlgorithmGPU(state["sites"])
        try:
            status = _build(algo)
            return status, _store(frame, algo.toHostFull())
        finally:
            algo.close()
    if call == "batch":
        diagrams, counts, _ = state["batch"].build(state["diagrams"])
        at = 0
        for d, v in zip(diagrams, counts):
            frame["positions"][at:at + v] = d.vertices.reshape(-1, 4)
            frame["ids"][at:at + v] = d.verticesId.reshape(-1, 4)
            at += int(v)
        return counts, frame["positions"], frame["ids"]
    algo = state["algo"]
    if call == "cavity":
        ratios, _ = algo.cavity_hit_ratios(samples=case["samples"])
        cavities = algo.cavity_vertices()
        frame["ratios"][:ratios.size] = ratios
        frame["cavities"][:cavities.shape[0]] = cavities
        return ratios.size, cavities.shape[0], frame
    if call == "check":
        bad, flags = algo.certify()
        largest, above, singular, errors = algo.vertex_error()
        frame["flags"][:flags.size] = flags
        frame["errors"][:errors.size] = errors
        return bad, largest, above, singular, frame
    # rebuild: this step's sites, the build, and the outputs in the program's device buffers
    lib = apo_b200.load_library()
    sites = state["sites"]
    dtype = apo_b200.APO2_F64 if sites.dtype == torch.float64 else apo_b200.APO2_F32
    stream = torch.cuda.current_stream().cuda_stream
    apo_b200._check(lib.apo2_set_sites(algo.handle, sites.data_ptr(), dtype, apo_b200.APO2_DEVICE, ctypes.c_void_p(stream)))
    algo.build_and_extract(stream)
    vertices, closed = ctypes.c_uint64(), ctypes.c_uint64()
    for copy, positions, ids, count in ((lib.apo2_get_vertices, "positions", "ids", vertices),
                                        (lib.apo2_get_closed_edges, "closed_positions", "closed_ids", closed)):
        apo_b200._check(copy(algo.handle, frame[positions].data_ptr(), frame[ids].data_ptr(), frame[ids].shape[0],
                             apo_b200.APO2_DEVICE, ctypes.byref(count)))
    return (vertices.value, closed.value, frame["positions"], frame["ids"], frame["closed_positions"],
            frame["closed_ids"][:, :3])


def work(case: dict) -> dict:
    """Sites read once, outputs written once; the tangent-sphere solve of every vertex in each of
    its four cells and its conflict test against the cell's nearest neighbours."""
    n = case["sites"]
    vertices = _VERTICES_PER_SITE[case["cloud"]] * n
    read = n * (32 if case["dtype"] == "f64" else 16)
    if case["call"] == "cavity":
        # every vertex's rays: at least one sphere test (20 operations) per ray
        return {"bytes": read + 32 * vertices + 4 * vertices, "flops": vertices * case["samples"] * 20}
    if case["call"] == "check":
        # four interval distances and one Newton-refined solve per vertex
        return {"bytes": read + 48 * vertices + 5 * vertices, "flops": vertices * (4 * 2 * _TEST + _SOLVE)}
    return {"bytes": read + 48 * vertices, "flops": 4 * vertices * (_SOLVE + _NEIGHBOURS * _TEST)}


def exact(case: dict, seed: int):
    """None for every case: which vertices a diagram has, and their order, are decided by the
    build's own comparisons (single-precision lengths against 1e-8, ties by sorted position), so
    plain 64-bit arithmetic has no arrays of the same layout; the hit ratios, certificates and
    errors are per vertex of such a diagram."""
    return None
