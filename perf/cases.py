"""What the performance of this package is measured on: neighbor lists as its
users build them, through the public calculators, from a single molecule to
half a million atoms of a crystal or two million of a liquid.

``listed()`` names the cases, ``draw()`` gives more of the same ranges,
``prepare()`` makes what a program holds before the call (positions and box on
the GPU, or on the host where the caller works with numpy; the calculator it
keeps from step to step), ``run()`` is one pass, ``work()`` what a pass cannot
do without, ``tolerance()`` how far two correct passes may be apart.

The pairs of a list come in no particular order unless the caller asks for
one, and their number differs from system to system, so a pass ends as the
programs that ask for lists do, with sums over the neighbours of every point
(of the distances, and for some cases of the vectors). Programs that ask for
rows in order take the rows as they lie: where each one starts, and its sum
from first to last, which for a list in canonical order is one exact number.
"""

import math

import numpy as np
import torch

import vesin_b200

DIAMOND_A = 3.567  # lattice constant of the crystals, 8 atoms per cubic cell
DIAMOND_DENSITY = 8.0 / DIAMOND_A**3
LIQUID_DENSITY = 0.0334  # molecules of a liquid per cubic Angstrom
CELL_DENSITY = 0.1  # atoms of a small cell
MOLECULE_RADIUS = 6.0


def listed():
    return [
        # One molecule at a time: a conformer search or a geometry optimisation. No box, all latency.
        dict(name="molecule", kind="list", system="molecule", n=48, cutoff=5.0, full=False, dtype="float64", order="any", periodic="FFF", quantities="ijdD", sums="dD", copy=True, skin=0.0),
        # A unit cell with a cutoff longer than the cell (periodic images of every atom): training sets, phonons.
        dict(name="unit_cell", kind="list", system="cell", n=64, cutoff=9.0, full=True, dtype="float64", order="any", periodic="TTT", quantities="ijSdD", sums="dD", copy=True, skin=0.0),
        # The ordinary system of atomistic simulations with learned potentials.
        dict(name="crystal_1k", kind="list", system="crystal", nx=5, ny=5, nz=5, cutoff=5.0, full=True, dtype="float64", order="any", periodic="TTT", quantities="ijSdD", sums="d", copy=True, skin=0.0),
        # Molecular dynamics of a small liquid with a Verlet skin: four steps in which no atom leaves the skin.
        dict(name="liquid_12k_skin", kind="steps", system="liquid", n=12000, cutoff=6.0, full=False, dtype="float64", order="any", periodic="TTT", quantities="ijdD", sums="dD", copy=False, skin=1.0, steps=4),
        # A surface (periodic in two directions) for code that walks the rows of every atom.
        dict(name="surface_27k_sorted", kind="list", system="crystal", nx=15, ny=15, nz=15, cutoff=5.0, full=True, dtype="float64", order="sorted", periodic="TTF", quantities="ijSd", sums="d", copy=True, skin=0.0),
        # Single precision, as learned potentials run.
        dict(name="crystal_110k_f32", kind="list", system="crystal", nx=24, ny=24, nz=24, cutoff=5.0, full=True, dtype="float32", order="any", periodic="TTT", quantities="ijSdD", sums="d", copy=True, skin=0.0),
        # The benchmark system of this package.
        dict(name="crystal_512k", kind="list", system="crystal", nx=40, ny=40, nz=40, cutoff=5.0, full=True, dtype="float64", order="any", periodic="TTT", quantities="ijSdD", sums="d", copy=True, skin=0.0),
        # A large liquid, half list, used in place before the next step: few pairs per atom.
        dict(name="liquid_2m_half", kind="list", system="liquid", n=1 << 21, cutoff=6.0, full=False, dtype="float64", order="any", periodic="TTT", quantities="ijSdD", sums="d", copy=False, skin=0.0),
        # The list in its one canonical order, for comparison and reproducible sums.
        dict(name="crystal_216k_canonical", kind="list", system="crystal", nx=30, ny=30, nz=30, cutoff=5.0, full=True, dtype="float64", order="canonical", periodic="TTT", quantities="ijSdD", sums="d", copy=True, skin=0.0),
        # numpy arrays in and out: analysis scripts.
        dict(name="host_liquid_20k", kind="host", system="liquid", n=20000, cutoff=6.0, full=True, dtype="float64", order="any", periodic="TTT", quantities="ijSd", sums="d", copy=True, skin=0.0),
        # A batch of molecules in one call: training and screening.
        dict(name="molecules_16k_f32", kind="batch", system="molecule", n_systems=16384, n_min=16, n_max=64, cutoff=4.0, full=True, dtype="float32", quantities="ijSdD", sums="d", copy=True),
        # A batch of periodic cells of very different sizes: a training set of crystals.
        dict(name="cells_512", kind="batch", system="cell", n_systems=512, n_min=4, n_max=200, cutoff=5.0, full=True, dtype="float64", quantities="ijSD", sums="D", copy=True),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """Another case: the kinds of the listed ones, sizes over their whole range."""
    kind = rng.choice(["molecule", "cell", "crystal", "crystal", "surface", "liquid", "liquid", "steps", "host", "molecules", "cells"])
    full = rng.random() < 0.6
    common = dict(full=full, dtype=rng.choice(["float64", "float64", "float32"]), copy=rng.random() < 0.7)
    if kind == "molecules":
        low = rng.randint(4, 24)
        return dict(
            kind="batch", system="molecule", n_systems=_log_uniform(rng, 100, 16000), n_min=low, n_max=rng.randint(low, 80),
            cutoff=round(rng.uniform(3.5, 5.5), 2), quantities=rng.choice(["ijSdD", "ijdD"]), sums="d", **common,
        )
    if kind == "cells":
        low = rng.randint(2, 20)
        return dict(
            kind="batch", system="cell", n_systems=_log_uniform(rng, 20, 600), n_min=low, n_max=rng.randint(low, 200),
            cutoff=round(rng.uniform(4.0, 6.0), 2), quantities=rng.choice(["ijSD", "ijSdD"]), sums="D", **common,
        )
    single = dict(kind="list", periodic="TTT", skin=0.0, cutoff=round(rng.uniform(4.0, 6.5), 2), **common)
    order = rng.choice(["any", "any", "any", "sorted", "canonical"])
    quantities = rng.choice(["ijSdD", "ijSdD", "ijdD", "ijSd", "ijd"])
    if kind == "molecule":
        return dict(single, system="molecule", n=rng.randint(4, 120), order="any", periodic="FFF", quantities="ijdD", sums="dD")
    if kind == "cell":
        return dict(single, system="cell", n=rng.randint(2, 200), order="any", quantities="ijSdD", sums="dD", cutoff=round(rng.uniform(5.0, 9.0), 2))
    if kind == "steps":
        return dict(
            single, kind="steps", system="liquid", n=_log_uniform(rng, 500, 40000), order="any", quantities="ijdD", sums="dD",
            skin=round(rng.uniform(0.5, 1.5), 2), steps=4,
        )
    if kind == "host":
        return dict(single, kind="host", system="liquid", n=_log_uniform(rng, 50, 60000), order=order, quantities="ijSd", sums="d", copy=True)
    if kind == "liquid":
        n = _log_uniform(rng, 300, 1900000)
        return dict(single, system="liquid", n=n, order=order, quantities=quantities, sums="d")
    # crystals and surfaces: blocks of any shape, at most 400 000 atoms (of 5 A cutoff) in all
    shape = [_log_uniform(rng, 3, 60) for _ in range(3)]
    cutoff = single["cutoff"]
    while 8 * shape[0] * shape[1] * shape[2] * (cutoff / 5.0) ** 3 > 400000:
        shape[shape.index(max(shape))] = max(shape) - 1
    return dict(
        single, system="crystal", nx=shape[0], ny=shape[1], nz=shape[2], order=order, periodic="TTF" if kind == "surface" else "TTT",
        quantities=quantities, sums="d",
    )


# ---- inputs ----


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _crystal(case, generator):
    axes = [torch.arange(case[k], dtype=torch.float64, device="cuda") for k in ("nx", "ny", "nz")]
    cells = torch.stack(torch.meshgrid(*axes, indexing="ij"), dim=-1).reshape(-1, 1, 3)
    basis = torch.tensor(
        [[0, 0, 0], [0, 2, 2], [2, 0, 2], [2, 2, 0], [1, 1, 1], [1, 3, 3], [3, 1, 3], [3, 3, 1]], dtype=torch.float64, device="cuda"
    )
    points = ((cells + basis / 4.0) * DIAMOND_A).reshape(-1, 3)
    points += 0.05 * torch.randn(points.shape, dtype=torch.float64, device="cuda", generator=generator)
    box = torch.diag(torch.tensor([case["nx"], case["ny"], case["nz"]], dtype=torch.float64, device="cuda") * DIAMOND_A)
    return points, box


def _liquid(case, generator):
    length = (case["n"] / LIQUID_DENSITY) ** (1.0 / 3.0)
    points = length * torch.rand((case["n"], 3), dtype=torch.float64, device="cuda", generator=generator)
    return points, length * torch.eye(3, dtype=torch.float64, device="cuda")


def _molecules(counts, generator):
    """Molecules of `counts` atoms: places of a grid of 1.5 A inside a sphere,
    each moved by up to a quarter of an Angstrom, back to back."""
    ticks = torch.arange(-4, 5, dtype=torch.float64, device="cuda") * 1.5
    grid = torch.stack(torch.meshgrid(ticks, ticks, ticks, indexing="ij"), dim=-1).reshape(-1, 3)
    grid = grid[(grid * grid).sum(dim=1) <= MOLECULE_RADIUS**2]
    counts = torch.as_tensor(counts, device="cuda")
    chosen = torch.rand((len(counts), len(grid)), device="cuda", generator=generator).argsort(dim=1)[:, : int(counts.max())]
    taken = torch.arange(chosen.shape[1], device="cuda") < counts[:, None]
    points = grid[chosen[taken]]
    return points + 0.5 * torch.rand(points.shape, dtype=torch.float64, device="cuda", generator=generator) - 0.25


def _cells(counts, generator):
    """Triclinic cells of `counts` atoms at one density, lengths within 30 % of
    each other and sheared by up to half a length, atoms anywhere inside."""
    n = len(counts)
    counts = torch.as_tensor(counts, device="cuda")
    draws = torch.rand((n, 6), dtype=torch.float64, device="cuda", generator=generator)
    boxes = torch.zeros((n, 3, 3), dtype=torch.float64, device="cuda")
    for k in range(3):
        boxes[:, k, k] = 1.0 + 0.3 * draws[:, k]
    boxes[:, 1, 0] = draws[:, 3] - 0.5
    boxes[:, 2, 0] = draws[:, 4] - 0.5
    boxes[:, 2, 1] = draws[:, 5] - 0.5
    volume = boxes[:, 0, 0] * boxes[:, 1, 1] * boxes[:, 2, 2]
    boxes *= (counts / CELL_DENSITY / volume).pow(1.0 / 3.0)[:, None, None]
    system = torch.repeat_interleave(torch.arange(n, device="cuda"), counts)
    inside = torch.rand((len(system), 3), dtype=torch.float64, device="cuda", generator=generator)
    return torch.bmm(inside[:, None, :], boxes[system])[:, 0, :].contiguous(), boxes


def _counts(case):
    """Sizes of the systems of a batch: part of the case, as a training set is."""
    return np.random.default_rng(case["n_systems"]).integers(case["n_min"], case["n_max"] + 1, case["n_systems"])


def prepare(case, seed):
    dtype = getattr(torch, case["dtype"])
    generator = _generator(seed)
    state = dict(case=case)
    if case["kind"] == "batch":
        counts = _counts(case)
        state["offsets"] = np.concatenate([[0], np.cumsum(counts)])
        if case["system"] == "molecule":
            points, boxes, periodic = _molecules(counts, generator), None, None
        else:
            points, boxes = _cells(counts, generator)
            boxes = boxes.to(dtype)
            periodic = torch.ones((len(counts), 3), dtype=torch.bool, device="cuda")
        state.update(points=points.to(dtype), boxes=boxes, periodic=periodic)
        state["list"] = vesin_b200.BatchNeighborList(case["cutoff"], case["full"])
        return state

    if case["system"] == "crystal":
        points, box = _crystal(case, generator)
    elif case["system"] == "liquid":
        points, box = _liquid(case, generator)
    elif case["system"] == "molecule":
        points, box = _molecules([case["n"]], generator), torch.zeros((3, 3), dtype=torch.float64, device="cuda")
    else:
        points, boxes = _cells([case["n"]], generator)
        box = boxes[0]
    state["periodic"] = True if case["periodic"] == "TTT" else [letter == "T" for letter in case["periodic"]]
    if case["kind"] == "host":
        state.update(points=points.to(dtype).cpu().numpy(), box=box.to(dtype).cpu().numpy())
    else:
        state.update(points=points.to(dtype), box=box.to(dtype).contiguous())
    if case["kind"] == "steps":
        frames = [points]
        for _ in range(case["steps"] - 1):
            frames.append(frames[-1] + 0.02 * torch.randn(points.shape, dtype=torch.float64, device="cuda", generator=generator))
        state["frames"] = [frame.to(dtype) for frame in frames]
    state["list"] = vesin_b200.NeighborList(
        case["cutoff"], case["full"], sorted=case["order"] == "sorted", skin=case["skin"], canonical=case["order"] == "canonical"
    )
    return state


# ---- one pass ----


def _sums(case, n_points, outputs, sums):
    """Per point, what a pair potential adds up over its neighbours."""
    i = outputs["i"].view(torch.int64)
    j = outputs["j"].view(torch.int64)
    result = {"pairs": i.shape[0]}
    if "d" in sums:
        d = outputs["d"]
        total = torch.zeros(n_points, dtype=d.dtype, device=d.device).scatter_add_(0, i, d)
        result["d"] = total if case["full"] else total.scatter_add_(0, j, d)
    if "D" in sums:
        D = outputs["D"]
        total = torch.zeros((n_points, 3), dtype=D.dtype, device=D.device).index_add_(0, j, D)
        result["D"] = total if case["full"] else total.index_add_(0, i, D, alpha=-1)
    return result


def _row_sums(n_points, outputs):
    """The rows of a list in order: where they start, and the sum of each."""
    i = outputs["i"].view(torch.int64)
    row_start = torch.searchsorted(i, torch.arange(n_points + 1, device=i.device))
    return {"row_start": row_start, "d": torch.segment_reduce(outputs["d"], "sum", offsets=row_start, initial=0.0)}


def _host_sums(case, n_points, outputs):
    i = outputs["i"].view(np.int64)
    total = np.bincount(i, weights=outputs["d"], minlength=n_points)
    if not case["full"]:
        total += np.bincount(outputs["j"].view(np.int64), weights=outputs["d"], minlength=n_points)
    return {"pairs": len(i), "d": total}


def run(state):
    case = state["case"]
    calculator = state["list"]
    quantities = case["quantities"]
    if case["kind"] == "batch":
        points = state["points"]
        values, pair_offsets = calculator.compute(
            points, state["offsets"], state["boxes"], state["periodic"], quantities, global_indices=True, copy=case["copy"]
        )
        result = _sums(case, points.shape[0], dict(zip(quantities, values)), case["sums"])
        result["pair_offsets"] = pair_offsets
        return result
    if case["kind"] == "steps":
        results = []
        for points in state["frames"]:
            values = calculator.compute(points, state["box"], state["periodic"], quantities, copy=case["copy"])
            results.append(_sums(case, points.shape[0], dict(zip(quantities, values)), case["sums"]))
        return results

    points = state["points"]
    values = calculator.compute(points, state["box"], state["periodic"], quantities, copy=case["copy"])
    outputs = dict(zip(quantities, values))
    if case["kind"] == "host":
        return _host_sums(case, points.shape[0], outputs)
    if case["order"] != "any":
        return _row_sums(points.shape[0], outputs)
    return _sums(case, points.shape[0], outputs, case["sums"])


# ---- what a pass cannot do without, and how exact it is ----


def _points_and_pairs(case):
    """Points and (from the density, boundaries left out) pairs of one list."""
    sphere = 4.0 / 3.0 * math.pi * case["cutoff"] ** 3
    half = 1.0 if case["full"] else 0.5
    if case["kind"] == "batch":
        points = case["n_systems"] * 0.5 * (case["n_min"] + case["n_max"])
        in_system = 0.5 * (case["n_min"] + case["n_max"])
    elif case["system"] == "crystal":
        points = 8.0 * case["nx"] * case["ny"] * case["nz"]
        in_system = points
    else:
        points = in_system = float(case["n"])
    if case["system"] == "molecule":
        # two points of one ball of radius R are within c of each other with this probability
        t = min(case["cutoff"] / MOLECULE_RADIUS, 2.0)
        close = t**3 * (1.0 - 9.0 * t / 16.0 + t**3 / 32.0)
        return points, half * points * max(in_system - 1.0, 0.0) * close
    density = {"crystal": DIAMOND_DENSITY, "liquid": LIQUID_DENSITY, "cell": CELL_DENSITY}[case["system"]]
    return points, half * points * sphere * density


def work(case):
    """Positions read once, the list of pairs written once (indices of 8 bytes,
    shifts of 12), sums written once; a vector, its square and a root per pair."""
    value = 4 if case["dtype"] == "float32" else 8
    per_pair = {"i": 8, "j": 8, "S": 12, "d": value, "D": 3 * value}
    points, pairs = _points_and_pairs(case)
    size = points * 3 * value + pairs * sum(per_pair[q] for q in case["quantities"])
    size += points * value * sum({"d": 1, "D": 3}[q] for q in case["sums"])
    steps = case.get("steps", 1)
    return {"bytes": steps * size, "flops": steps * 10.0 * pairs}


def tolerance(case):
    """Distances and vectors are correctly rounded results of one fixed sequence
    of operations; what differs between two correct passes is the order in which
    they are added up. Measured on passes over the same inputs: up to 3.4e-15
    (largest 2.4e-14) in double precision, where the vectors around an atom of a
    crystal nearly cancel, and the same in units of the last place of float32."""
    if case.get("order") == "canonical":
        return "exact"
    return {"rel": 5e-6, "max": 4e-5} if case["dtype"] == "float32" else {"rel": 1.4e-14, "max": 1e-13}
