"""Performance cases of the framework: the calls a user's program makes, over their real range.

Transport cases run scenes of ``monki.scenes`` through ``CUDA`` (``run_batches``,
``accumulate``), ``simulate``, ``importance.pilot`` and ``batched.run_batched``; network cases
train, differentiate and evaluate ``importance.ImportanceModel``. A case is a dict of plain
values; ``prepare`` makes what the program holds before the call (scene, session, network,
rows), ``run`` is one call, ``exact`` its result in 64 bits where it has one (the network;
a Monte Carlo run has none).
"""

from __future__ import annotations

import math
import shutil
import sys
import tempfile
from pathlib import Path

import numpy as np

_ROOT = Path(__file__).resolve().parents[1]
if str(_ROOT / "monki-gpu_gb300") not in sys.path:
    sys.path.insert(0, str(_ROOT / "monki-gpu_gb300"))

from monki import Guided, importance, scenes, simulate  # noqa: E402
from monki.batched import run_batched  # noqa: E402
from monki.execution import CUDA, BatchControls  # noqa: E402

# Scatters per photon of each kind of scene, counted by the kernels on the listed sizes
# (they set ``work`` only).
_SCATTERS = {"clear": 6.0, "box": 13.1, "layered": 51.5, "backward": 20.0, "batched": 20.0}
_GUIDED_SCATTERS = 9.6
# Arithmetic one scatter cannot do without: free path and direction sampling with the Stokes
# rotation, and per view a phase matrix, a rotation and an optical depth.
_FLOPS_SCATTER, _FLOPS_VIEW = 300, 150


def listed():
    return [
        # A quick look at a scene: few photons, so latency and launches count.
        _transport("clear-quick", "clear", 30, 20, 100, 1),
        # The clear-sky workload as a whole product run: 2,000 photons per column x 32 rounds.
        _transport("clear-simulate", "clear", 30, 20, 2000, 32, call="simulate"),
        # One statistical round of a precision run on the box cloud.
        _transport("box-round", "box", 30, 20, 1000, 1),
        # The group of rounds before the first check of a precision run, folded on the device.
        _transport("box-check", "box", 30, 20, 1000, 32, call="accumulate"),
        # The same group with the guided method's default weight window.
        _transport("box-guided", "box", 30, 20, 1000, 32, call="accumulate", guided=True),
        # The box-cloud workload's own round: 50,000 photons per column.
        _transport("box-large", "box", 30, 20, 50000, 1),
        # Polarized layered cloud with layer air-mass factors, two rounds of the adaptive run.
        _transport("layered-amf", "layered", 30, 20, 2000, 2, call="accumulate"),
        # Backward transport (photons from the sensor) on an odd grid.
        _transport("backward-odd", "backward", 23, 17, 2000, 2),
        # Uneven scenes in one launch sequence, sessions included.
        {"name": "batched-scenes", "kind": "batched", "scenes": 16, "scale": 0.02, "first": 0},
        # A pilot run that tallies the detector importance for the network's training rows.
        _transport("pilot", "box", 30, 20, 300, 2, call="pilot"),
        # Training of the importance network at its default batch.
        {"name": "fit", "kind": "network", "call": "fit", "rows": 105000, "batch": 65536, "steps": 300},
        # The trained network's map of one scene (30 x 20 x 35 cells).
        {"name": "predict", "kind": "network", "call": "predict", "rows": 21000, "batch": 65536},
    ]


def _transport(name, scene, nx, ny, photons, rounds, *, call="batches", guided=False):
    case = {"kind": "transport", "scene": scene, "nx": nx, "ny": ny, "photons": photons, "rounds": rounds,
            "call": call, "guided": guided}
    return {"name": name, **case} if name else case


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    pick = rng.random()

    if pick < 0.12:
        return {"kind": "network", "call": "fit", "rows": _log_uniform(rng, 20000, 105000),
                "batch": _log_uniform(rng, 1000, 65536), "steps": rng.randint(50, 300)}
    if pick < 0.18:
        return {"kind": "network", "call": "predict", "rows": _log_uniform(rng, 1000, 150000), "batch": 65536}
    if pick < 0.24:
        return {"kind": "network", "call": "gradients", "rows": _log_uniform(rng, 100, 65536), "batch": 65536}
    if pick < 0.32:
        return {"kind": "batched", "scenes": rng.randint(4, 16), "scale": 0.01 * rng.uniform(0.5, 2.0),
                "first": rng.randint(16, 48)}

    scene = rng.choice(["clear", "box", "box", "layered", "backward"])
    guided = scene == "box" and rng.random() < 0.4
    nx, ny = rng.randint(12, 64), rng.randint(10, 48)
    call = "pilot" if scene == "box" and not guided and rng.random() < 0.2 else rng.choice(
        ["batches", "accumulate", "simulate"])
    rounds = {"batches": rng.randint(1, 4), "accumulate": rng.randint(2, 32), "simulate": rng.randint(31, 40),
              "pilot": 2}[call]
    # Scatters from a quick look to a third of the largest listed run.
    scatters = math.exp(rng.uniform(math.log(1e6), math.log(1.2e8)))
    photons = max(4, int(scatters / (_scatters(scene, guided) * nx * ny * rounds)))
    return _transport(None, scene, nx, ny, photons, rounds, call=call, guided=guided)


def _scatters(scene, guided):
    return _GUIDED_SCATTERS if guided else _SCATTERS[scene]


def _scene(case, seed):
    """The case's scene; the seed places the box (the other scenes are uniform, and differ
    from seed to seed in their random streams)."""

    kind, nx, ny, photons, rounds = (case[k] for k in ("scene", "nx", "ny", "photons", "rounds"))
    if kind == "clear":
        return scenes.clear_sky(photons, rounds, nx=nx, ny=ny)
    if kind == "layered":
        return scenes.layered_cloud(photons, rounds, nx=nx, ny=ny)
    rng = np.random.default_rng(seed)
    width, depth = max(2, nx // 3), max(2, (3 * ny) // 10)
    x0, y0 = int(rng.integers(0, nx - width + 1)), int(rng.integers(0, ny - depth + 1))
    if kind == "box":
        return scenes.box_cloud(photons, rounds, nx=nx, ny=ny, box_x=(x0, x0 + width), box_y=(y0, y0 + depth))
    return _backward_scene(nx, ny, photons, rounds, x0, y0, width, depth)


def _backward_scene(nx, ny, photons, rounds, x0, y0, width, depth):
    levels = scenes.layer_levels_km()
    layers = len(levels) - 1
    profile = scenes.layer_fraction(levels, 1.0, 2.0) * np.diff(levels)
    cloud = np.zeros((nx, ny, layers))
    cloud[x0 : x0 + width, y0 : y0 + depth] = 8.0 * profile / profile.sum()
    depths = np.stack([scenes.aerosol_depth(levels, nx, ny), cloud])
    view = {"nx": nx, "ny": ny, "nmat": 3, "solar_zenith": 40.0, "solar_azimuth": 0.0,
            "view_zeniths": [0.0, 30.0, 60.0], "view_azimuths": [0.0, 90.0, 180.0], "albedo": 0.1,
            "save_path": False, "gas_scattering": scenes.rayleigh_layers(levels),
            "gas_absorption": scenes.ozone_layers(levels), "particle_optical_depth": depths}
    tables = scenes.build_tables(levels_km=levels, particles=[scenes.AEROSOL, scenes.CLOUD], backward=True, **view)
    metadata = scenes.scene_metadata("backward", levels, **view)
    return scenes.TransportScene("backward", tables, metadata, photons, rounds, True)


class _Held:
    """What a program keeps between calls; its native handle is closed with it."""

    def __init__(self, case):
        self.case = case
        self.owned = None
        self.directory = None
        self.calls = 0

    def __del__(self):
        if self.owned is not None:
            self.owned.close()
        if self.directory is not None:
            shutil.rmtree(self.directory, ignore_errors=True)


def _rows(case, seed):
    """Feature rows of the network: cells of randomly placed box clouds, a smooth log
    importance of their optical depths with noise, and the weights of well sampled cells."""

    rng = np.random.default_rng(seed)
    parts, rows = [], 0
    while rows < case["rows"]:
        parts.append(importance.cell_features(scenes.box_cloud_variant(int(rng.integers(1 << 30)), 300, 2).tables))
        rows += len(parts[-1])
    x = np.concatenate(parts)[: case["rows"]]
    target = -0.8 * x[:, 8] - 0.3 * x[:, 10] + 0.5 * np.sin(3.0 * x[:, 0]) - 1.5 + rng.normal(0.0, 0.1, len(x))
    weight = np.minimum(1.0, rng.gamma(2.0, 0.6, len(x)))
    return x, target.astype(np.float32), weight.astype(np.float32)


def prepare(case, seed):
    held = _Held(case)

    if case["kind"] == "network":
        held.rows = _rows(case, seed)
        held.params = importance.initial_params(seed % 1000)
        held.owned = importance.ImportanceModel(rows=case["batch"], params=held.params)
        x = held.rows[0]
        held.owned.mean = x.mean(axis=0).astype(np.float32)
        spread = x.std(axis=0)
        held.owned.scale = np.where(spread > 1e-6, 1.0 / np.maximum(spread, 1e-6), 1.0).astype(np.float32)
        return held

    held.seed = seed % (1 << 31)
    if case["kind"] == "batched":
        first = case["first"]
        held.scenes = [scenes.batched_scene(s, photons_scale=case["scale"]) for s in range(first, first + case["scenes"])]
        return held

    held.scene = _scene(case, seed)
    held.guided = Guided(0.0, 0.25, 0.0, 2.0) if case["guided"] else None
    if case["call"] in ("batches", "accumulate"):
        held.owned = CUDA(seed=held.seed, guided=held.guided)
        held.owned.prepare(held.scene)
    elif case["call"] == "simulate":
        held.directory = Path(tempfile.mkdtemp(prefix="monki_"))
    return held


def _next_rounds(held):
    first = held.calls * held.case["rounds"] + 1
    held.calls += 1
    return [BatchControls(i, held.case["photons"]) for i in range(first, first + held.case["rounds"])]


def _tallies(batches):
    out = {"stokes": np.stack([b.stokes for b in batches])}
    if batches[0].weighted_paths is not None:
        out["paths"] = np.stack([b.weighted_paths for b in batches])
        out["weights"] = np.stack([b.weights for b in batches])
    return out


def run(held):
    case = held.case

    if case["kind"] == "network":
        model, (x, target, weight) = held.owned, held.rows
        if case["call"] == "predict":
            return model.predict(x)
        if case["call"] == "gradients":
            loss, gradient = model.gradients(x, target, weight)
            return {"loss": np.float32(loss), "gradient": gradient}
        # Training from the initial parameters (setting them also clears Adam's moments).
        model.params = held.params
        losses = model.fit(x, target, weight, steps=case["steps"], batch=case["batch"])
        return {"losses": losses, "params": model.params}

    if case["kind"] == "batched":
        results, _ = run_batched(held.scenes, seed=held.seed)
        return [np.stack([b.stokes for b in batches]) for batches, _ in results]

    if case["call"] == "batches":
        return _tallies(held.owned.run_batches(_next_rounds(held)))

    if case["call"] == "accumulate":
        held.owned.reset_statistics()
        history = held.owned.accumulate(_next_rounds(held))
        statistics = held.owned.statistics()
        return {"history": history, **{k: v for k, v in statistics.items() if k != "rounds"}}

    if case["call"] == "pilot":
        tally, batches = importance.pilot(held.scene, rounds=case["rounds"], photons_per_column=case["photons"],
                                          seed=held.seed)
        return {"tally": tally, **_tallies(batches)}

    held.calls += 1
    result = simulate(held.scene, CUDA(seed=held.seed, guided=held.guided), held.directory / f"{held.calls}.nc")
    names = ("radiance", "std_radiance", "DOP", "radiance_convergence", "AMF_layer")
    return {name: result.values[name] for name in names if name in result.values}


def _network_work(case):
    weights = 64 * 256 + 2 * 256 * 256 + 256
    if case["call"] == "predict":
        return {"bytes": case["rows"] * (48 + 1) * 4 + 4 * weights, "flops": 2.0 * case["rows"] * weights}
    # Forward and weight gradients of every layer, input gradients of all but the first.
    per_row = 2 * (3 * weights - 64 * 256)
    rows = case["rows"] if case["call"] == "gradients" else case["steps"] * case["batch"]
    steps = 1 if case["call"] == "gradients" else case["steps"]
    return {"bytes": rows * (48 + 2) * 4 + steps * weights * 4 * 7, "flops": float(rows * per_row)}


def work(case):
    if case["kind"] == "network":
        return _network_work(case)

    if case["kind"] == "batched":
        data = flops = 0.0
        for s in range(case["first"], case["first"] + case["scenes"]):
            scene = scenes.batched_scene(s, photons_scale=case["scale"])
            nmat, nx, ny, _, views = scene.shape
            data += scene.tables.size * 4 + nmat * nx * ny * views * 8
            flops += scene.photons_per_column * nx * ny * _SCATTERS["batched"] * (_FLOPS_SCATTER + views * _FLOPS_VIEW)
        return {"bytes": data, "flops": flops}

    columns, layers, views = case["nx"] * case["ny"], 35, 3
    nmat = 1 if case["scene"] == "clear" else 3
    pixel = columns * views * (nmat + (layers + 1 if case["scene"] == "layered" else 0))
    outputs = pixel * (3 if case["call"] in ("accumulate", "simulate") else case["rounds"])
    tables = columns * layers * 4 + 8 * 3601 * (1 if case["scene"] == "clear" else 2)
    events = columns * case["photons"] * case["rounds"] * _scatters(case["scene"], case["guided"])
    return {"bytes": 4.0 * tables + 8.0 * outputs, "flops": events * (_FLOPS_SCATTER + views * _FLOPS_VIEW)}


def exact(case, seed):
    """The network in 64 bits from the same rows and parameters; a Monte Carlo run and a
    training run (hundreds of dependent steps) have no such value."""

    if case["kind"] != "network" or case["call"] == "fit":
        return None

    from scipy.special import erf

    x, target, weight = _rows(case, seed)
    params = importance.initial_params(seed % 1000).astype(np.float64)
    mean = x.mean(axis=0).astype(np.float32)
    spread = x.std(axis=0)
    scale = np.where(spread > 1e-6, 1.0 / np.maximum(spread, 1e-6), 1.0).astype(np.float32)
    h = np.zeros((len(x), 64))
    h[:, :48] = ((x - mean) * scale).astype(np.float32)
    shapes = ((256, 64), (256,), (256, 256), (256,), (256, 256), (256,), (256,), (1,))
    parts, at = [], 0
    for shape in shapes:
        size = math.prod(shape)
        parts.append(params[at : at + size].reshape(shape))
        at += size
    inputs, slopes = [h], []
    for layer in range(3):
        z = inputs[-1] @ parts[2 * layer].T + parts[2 * layer + 1]
        cdf = 0.5 * (1.0 + erf(z / math.sqrt(2.0)))
        slopes.append(cdf + z * np.exp(-0.5 * z * z) / math.sqrt(2.0 * math.pi))
        inputs.append(z * cdf)
    y = inputs[3] @ parts[6] + parts[7][0]
    if case["call"] == "predict":
        return y
    t, w = target.astype(np.float64), weight.astype(np.float64)
    d = (y - t) / w.sum()
    dy = 2.0 * w * d
    gradients = [np.array([dy.sum()]), inputs[3].T @ dy]
    g = np.outer(dy, parts[6])
    for layer in (2, 1, 0):
        g = g * slopes[layer]
        gradients += [g.sum(axis=0), (g.T @ inputs[layer]).ravel()]
        g = g @ parts[2 * layer]
    return {"loss": float((w * d * (y - t)).sum()), "gradient": np.concatenate(gradients[::-1])}
