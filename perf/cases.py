"""What the engine's speed is measured on: the calls that a search over
walking creatures makes, through the package's public entry points.

A case is a dict of plain values. `call` names the entry point:

* ``record``: Engine.record, every frame of a few creatures, as a viewer or
  a replay file needs them.
* ``evaluate``: Engine.run, a packed generation from host memory to results
  in host memory (the drop-in boundary of a scheduler).
* ``resident``: Engine.advance_device_cells, the kernel entry on device
  arrays with the niche cells in the same launch.
* ``gradient``: Engine.forward and Tape.backward.
* ``ascent``: one launch of an Ascent graph (forward, backward, gene
  gradients, clipped step and repacking per step), its fitness and genes.
* ``emitters``: one search generation, CmaEmitters.ask, packing, evaluation
  and CmaEmitters.tell.
* ``epilogue``: metrics rows and niche cells, dump rows and the rung audit
  of a generation's results on the device.

Bodies are drawn by the package's generator with the repository's own
workload specs (`spec` is a key of configs.WORKLOADS). An evaluated
generation has other bodies each seed; where the outputs' sizes follow from
the bodies (frames, gradients, genes, emitters) the body plans stay and the
seed draws their genes. With `evolved`, muscles get what mutation gives
them: anchors moved along their bones, tendons and touch sensors on some.
"""
import ctypes
import dataclasses
import functools

import numpy as np
import torch

import evolution_simulator_gpu_b200 as ce
from evolution_simulator_gpu_b200 import api
from evolution_simulator_gpu_b200.cma import CmaEmitters
from evolution_simulator_gpu_b200.configs import QUAKE, WORKLOADS, effects_world_kw

# Worlds: the calm ground; the effects world of the repository's workload;
# the same with pebbles and tremors; every effect at once; and a world that
# has no kernel of its own (mud on a slope), which reads its switches at run
# time.
WORLDS = {
    "calm": {},
    "effects": effects_world_kw(),
    "tremors": dict(effects_world_kw(), terrain=1, quake=QUAKE[1]),
    "every": dict(terrain=2, gravity=14.7, air_retention=0.985, ground_friction=1.0, slope=0.03, wind=-1.0, mud=0.05,
                  brambles=3.0, water=0.12, patches=0.5, gaps=0.35, hurdles=0.08, quake=0.05),
    "mud": dict(mud=0.05, slope=0.03),
}
# Mean nodes and muscles of a spec's bodies, and the part of a trial that its
# creatures run before a fall ends it (calm, with effects), for work().
MEANS = {"small": (4.5, 4.0), "game": (6.5, 13.0), "effects": (7.0, 6.5), "gradients": (8.0, 12.0),
         "refine": (9.5, 9.0)}
RUNS = {"calm": 0.64, "mud": 0.4}


def listed():
    return [
        # One creature's replay, as a viewer asks for it: the smallest call.
        dict(name="record_one", call="record", spec="game", world="calm", count=1, seconds=20.0, evolved=True),
        # The replay frames of a small population's first 16 creatures.
        dict(name="record_16", call="record", spec="small", world="calm", count=16, seconds=20.0, evolved=False),
        # A small population on the CPU-sized workload, whole trials.
        dict(name="evaluate_4096", call="evaluate", spec="small", world="calm", count=4096, seconds=20.0, rate=60,
             screen=False, evolved=False),
        # One wave (CE_WAVE) of the game workload, whole trials.
        dict(name="evaluate_wave", call="evaluate", spec="game", world="calm", count=262_144, seconds=20.0, rate=60,
             screen=False, evolved=False),
        # An evolved population on rough ground, an odd count, whole trials.
        dict(name="evaluate_effects", call="evaluate", spec="effects", world="effects", count=200_003, seconds=20.0,
             rate=60, screen=False, evolved=True),
        # An island's round at 120 steps a second, with the 5 s screen.
        dict(name="evaluate_island", call="evaluate", spec="gradients", world="calm", count=20_011, seconds=8.0,
             rate=120, screen=True, evolved=True),
        # A big generation resident on the device, short trials, with cells.
        dict(name="resident_million", call="resident", spec="game", world="calm", count=1_000_003, seconds=4.0,
             evolved=False),
        # Gradients of an elite set in the calm, grippy world.
        dict(name="gradient_calm", call="gradient", spec="gradients", world="calm", count=16_381, seconds=4.0),
        # Gradients of a few elites over longer trials with tremors.
        dict(name="gradient_tremors", call="gradient", spec="refine", world="tremors", count=1_021, seconds=10.0),
        # Gradient ascent of a thousand elites as one graph.
        dict(name="ascent", call="ascent", spec="refine", world="tremors", count=1_024, seconds=4.0, steps=2),
        # A search generation: 16 samples of each of 512 CMA-ES emitters.
        dict(name="emitters", call="emitters", spec="refine", world="effects", count=512, samples=16, seconds=10.0),
        # What follows a generation's results: metrics, cells, dump and audit.
        dict(name="epilogue", call="epilogue", spec="game", world="calm", count=300_007, seconds=20.0),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    call = rng.choice(["record", "evaluate", "evaluate", "resident", "gradient", "ascent", "emitters", "epilogue"])
    seconds = round(rng.uniform(2.0, 20.0), 1)
    spec = rng.choice(["small", "game", "effects", "refine"])
    world = rng.choice(["calm", "effects", "tremors"])
    evolved = rng.random() < 0.5
    if call == "record":
        return dict(call=call, spec=spec, world=world, count=_log(rng, 1, 64), seconds=seconds, evolved=evolved)
    if call == "evaluate":
        world = rng.choice(["calm", "calm", "effects", "tremors", "every", "mud"])
        return dict(call=call, spec=spec, world=world, seconds=seconds,
                    count=_log(rng, 200, min(250_000, int((5e6 if spec in ("small", "game") else 2e6) / seconds))),
                    rate=rng.choice([60, 60, 120]) if seconds < 10 else 60, screen=rng.random() < 0.5, evolved=evolved)
    if call == "resident":
        return dict(call=call, spec=spec, world=world, seconds=round(seconds / 2, 1), evolved=evolved,
                    count=_log(rng, 1_000, int((4e6 if spec in ("small", "game") else 1e6) / seconds)))
    if call == "gradient":
        return dict(call=call, spec=rng.choice(["gradients", "refine"]), world=world, count=_log(rng, 64, 16_000),
                    seconds=round(rng.uniform(1.0, 4.0), 1))
    if call == "ascent":
        steps = rng.randint(1, 3)
        return dict(call=call, spec=rng.choice(["gradients", "refine"]), world=world, count=_log(rng, 64, 4_000),
                    seconds=round(rng.uniform(1.0, min(4.0, 7.0 / steps)), 1), steps=steps)
    if call == "emitters":
        return dict(call=call, spec="refine", world=world, count=_log(rng, 16, 1_000), samples=rng.randint(4, 40),
                    seconds=seconds)
    return dict(call="epilogue", spec=spec, world=world, count=_log(rng, 1_000, 600_000), seconds=20.0)


@functools.lru_cache(maxsize=1)
def _engine():
    """The engine handle that a program opens once and keeps."""
    return ce.Engine(0)


def _world(case):
    kw = dict(WORLDS[case["world"]], duration=case["seconds"], rate=case.get("rate", 60))
    if case["spec"] == "gradients" and case["world"] == "calm":
        kw["ground_friction"] = 3.0
    if case.get("screen"):
        kw["screen"] = (min(5.0, 0.6 * case["seconds"]), 0.3, 0.1, 0.2)
    return ce.make_world(**kw)


def _population(case, seed):
    spec = WORKLOADS[case["spec"]].spec
    plans_stay = case["call"] in ("record", "gradient", "ascent", "emitters")
    pop = ce.generate(spec if plans_stay else dataclasses.replace(spec, seed=spec.seed + 16 * (seed + 1)),
                      min(case["count"], 20_000) if case["call"] == "epilogue" else case["count"])
    rng = np.random.default_rng(seed)
    m, n = pop.muscles, len(pop.muscles)
    if plans_stay:
        pop.nodes["friction"] = rng.uniform(spec.friction_lo, spec.friction_hi, len(pop.nodes))
        pop.bones["rest_length"] *= rng.uniform(0.95, 1.05, len(pop.bones)).astype(np.float32)
        scale = rng.uniform(0.95, 1.05, n).astype(np.float32)
        m["short"] *= scale
        m["long"] *= scale
        m["phase"] = rng.random(n, np.float32)
        m["duty"] = rng.uniform(0.05, 0.95, n)
        pop.strength[:] = rng.uniform(0.5, 1.5, n)
    if case.get("evolved"):
        for end in ("anchor_a", "anchor_b"):
            m[end] = np.clip(m[end] + rng.normal(0.0, 0.3, n), 0.0, 1.0)
        m["tendon"] = np.where(rng.random(n) < 0.2, rng.random(n), 0.0)
        m["sensor"] = np.where(rng.random(n) < 0.1, rng.integers(0, 4, n), api.NO_SENSOR)
        m["reset"] = rng.random(n)
    return pop


def _up(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).cuda()


def _synthetic_results(count, seed):
    """Results of a generation without running it: trials that end at any
    step, random trace words (half floats, finite), as their fields range."""
    rng = np.random.default_rng(seed)
    words = rng.integers(0, 1 << 32, size=(count, 7), dtype=np.uint64).astype(np.uint32) & np.uint32(0x7bff7bff)
    steps = rng.integers(1, 1201, count).astype(np.uint32)
    words[:, 2] = (words[:, 2] & 0xffff) | (steps << 16)
    res = np.zeros(count, ce.RESULT_DTYPE)
    for k, f in enumerate(("contact_hi", "lift_hi", "ground_hi", "previous_center_y", "vertical_extremum",
                           "vertical_trend", "gait_turns")):
        res[f] = words[:, k].view(np.float32)
    early = (steps < 1200) & (rng.random(count) < 0.9)
    end = (steps / np.float32(60.0)).astype(np.float32)
    cut = early & (rng.random(count) < 0.3)
    res["fall_time"] = np.where(early & ~cut, end, 0.0)
    res["screened"] = np.where(cut, end, 0.0)
    res["fitness"] = rng.normal(2.0, 1.5, count)
    res["screen_x"] = rng.normal(2.0, 1.5, count)
    res["ground_contact"] = rng.integers(0, 4000, count)
    res["height_sum"] = rng.random(count) * steps
    res["vertical_oscillation"] = rng.random(count) * 0.5
    res["gait_frequency"] = rng.random(count) * 6.0
    res["lift_lo"] = rng.integers(0, 64, count).astype(np.uint32).view(np.float32)
    return res, rng


def prepare(case, seed):
    call, world = case["call"], _world(case)
    s = dict(call=call, world=world, engine=_engine())
    if call == "epilogue":
        return _prepare_epilogue(case, seed, s)
    pop = _population(case, seed)
    if call in ("record", "evaluate", "gradient"):
        s["wave"] = ce.pack(pop, world)
    elif call == "resident":
        wave = ce.pack(pop, world)
        n, rows, mm = len(wave), wave.max_nodes, wave.max_muscles
        s.update(n=n, rows=rows, mm=mm, params=ce.make_params(world, 0, n),
                 lanes=_up(wave.lanes), muscles=_up(wave.muscles), heads=_up(wave.heads),
                 shapes=_up(ce.shape_classes(pop, wave)),
                 results=torch.zeros((n, 19), dtype=torch.int32, device="cuda"),
                 cells=torch.zeros(n, dtype=torch.int64, device="cuda"),
                 metrics=torch.zeros((n, 9), dtype=torch.int32, device="cuda"),
                 counter=torch.zeros(64, dtype=torch.int32, device="cuda"),
                 scratch=torch.empty(_engine().scratch_bytes(ce.world_flags(world), world.rate, rows, mm, n),
                                     dtype=torch.uint8, device="cuda"))
    elif call == "ascent":
        s.update(ascent=api.Ascent(_engine(), pop, world, case["steps"], 1e-2), steps=case["steps"])
    elif call == "emitters":
        s.update(emitters=CmaEmitters(pop), samples=case["count"] * case["samples"], seed=seed)
    return s


def _prepare_epilogue(case, seed, s):
    n = case["count"]
    pop = _population(case, seed)
    which = np.arange(n) % len(pop)
    res, rng = _synthetic_results(n, seed)
    genomes = pop.genomes[which].copy()
    genomes["flags"] = (rng.random(n) < 1 / 128).astype(np.uint32)
    heads = np.zeros((n, 8), np.uint32)
    heads[:, 0] = genomes["node_count"]
    heads[:, 1] = genomes["muscle_count"]
    dump = np.zeros(n, ce.DUMP_HEAD_DTYPE)
    dump["parent"] = rng.integers(0, 2 ** 63, n, dtype=np.uint64)
    dump["slot"] = np.arange(n, dtype=np.uint32)
    dump["kind"] = rng.integers(0, 16, n)
    dump["nodes"], dump["muscles"] = genomes["node_count"], genomes["muscle_count"]
    scratch = int(api.lib().ce_audit_scratch_bytes(n))
    s.update(n=n, results=_up(res), heads=_up(heads), dump=_up(dump), genomes=_up(genomes), genes=_up(pop.muscles),
             bars=_up(rng.normal(2.0, 0.5, n).astype(np.float32)),
             shapes=_up(rng.integers(0, 4, n).astype(np.uint8)),
             metrics=torch.zeros((n, 9), dtype=torch.int32, device="cuda"),
             cells=torch.zeros(n, dtype=torch.int64, device="cuda"),
             rows=torch.zeros((n, 64), dtype=torch.uint8, device="cuda"),
             scratch=torch.empty(scratch, dtype=torch.uint8, device="cuda"),
             audit=torch.zeros(ctypes.sizeof(api.AuditC), dtype=torch.uint8, device="cuda"),
             words=torch.zeros(2 * 65_536 * 6, dtype=torch.int16, device="cuda"))
    return s


# Fields of a result that hold numbers; the others hold bits (contact and
# lift sets, the half-precision trace and the end code).
NUMBERS = ["fitness", "ground_contact", "vertical_oscillation", "gait_frequency", "height_sum", "fall_time",
           "head_shake", "screen_x", "screened"]


def _results(res):
    return dict(words=res.view(np.uint32).reshape(len(res), 19), **{f: res[f] for f in NUMBERS})


def run(s):
    call = s["call"]
    if call == "record":
        frames, res = s["engine"].record(s["wave"], s["world"])
        return dict(frames=frames, results=_results(res))
    if call == "evaluate":
        res, _ = s["engine"].run(s["wave"], s["world"])
        return _results(res)
    if call == "resident":
        stream = torch.cuda.current_stream().cuda_stream
        s["engine"].advance_device_cells(
            s["lanes"].data_ptr(), s["muscles"].data_ptr(), s["heads"].data_ptr(), s["results"].data_ptr(),
            s["counter"].data_ptr(), s["scratch"].data_ptr(), s["params"], s["world"], s["rows"], s["mm"],
            s["shapes"].data_ptr(), s["cells"].data_ptr(), s["metrics"].data_ptr(), stream)
        return dict(results=s["results"], cells=s["cells"], metrics=s["metrics"])
    if call == "gradient":
        with s["engine"].forward(s["wave"], s["world"]) as tape:
            return dict(gradients=tape.backward(), results=_results(tape.results))
    if call == "ascent":
        s["ascent"].launch()
        pop = s["ascent"].population()
        return dict(fitness=[s["ascent"].fitness(k) for k in range(s["steps"] + 1)],
                    nodes=pop.nodes.view(np.float32), muscles=pop.muscles.view(np.uint32),
                    lengths=[pop.muscles["short"], pop.muscles["long"]], strength=pop.strength)
    if call == "emitters":
        e = s["emitters"]
        pop = e.ask(s["samples"], seed=s["seed"])
        res = ce.evaluate(s["engine"], pop, s["world"])
        e.tell(pop, res["fitness"])
        return dict(results=_results(res), mean=e.mean, covariance=e.covariance, path_c=e.path_c,
                    path_sigma=e.path_sigma, sigma=e.sigma)
    return _run_epilogue(s)


def _run_epilogue(s):
    n, world = s["n"], s["world"]
    stream = torch.cuda.current_stream().cuda_stream
    ce.metrics_device(s["results"].data_ptr(), s["heads"].data_ptr(), s["shapes"].data_ptr(), n, world,
                      s["metrics"].data_ptr(), s["cells"].data_ptr(), stream)
    ce.dump_rows_device(s["results"].data_ptr(), s["heads"].data_ptr(), s["dump"].data_ptr(), 0, n, world,
                        s["rows"].data_ptr(), stream)
    api._check(api.lib().ce_audit_device(
        s["results"].data_ptr(), s["genomes"].data_ptr(), s["genes"].data_ptr(), s["bars"].data_ptr(), n,
        s["scratch"].data_ptr(), s["scratch"].numel(), s["audit"].data_ptr(), s["words"].data_ptr(), 65_536, stream),
        "ce_audit_device")
    return dict(metrics=s["metrics"], values=s["metrics"].view(torch.float32)[:, :7], cells=s["cells"],
                rows=s["rows"], audit=s["audit"], words=s["words"])


def work(case):
    """Bytes: packed records, results, frames, gradients and genes once.
    Operations: those of a substep of the mean body (75 a muscle, 40 a bone,
    36 a node, 110 a joint; twice that with the effects' ground, water and
    wind) times the substeps that the trials run, six times that for a
    gradient (the rerun and the reverse)."""
    n, m = MEANS[case["spec"]]
    call, count = case["call"], case["count"]
    if call == "epilogue":
        # Results, heads and genomes in; metrics, cells and dump rows out.
        return dict(bytes=count * (76 + 32 + 40 + 32 + 4 + 1 + 36 + 8 + 64), flops=count * 40)
    steps = case["seconds"] * case.get("rate", 60)
    if call == "emitters":
        count *= case["samples"]
    substeps = count * steps * 16 * (1.0 if call == "record" else RUNS.get(case["world"], 0.1))
    ops = 75 * m + 40 * (n - 1) + 36 * n + 110 * (n - 2)
    if case["world"] != "calm":
        ops *= 2
    body = 24 * n + 24 * (n - 1) + 80 * m + 32
    per = body + 76
    if call == "record":
        per += (steps + 101) * (32 + 2 * m + n) * 8
    elif call == "resident":
        per += 36 + 8
    elif call in ("gradient", "ascent"):
        per += (9 * m + 4 * n) * 4
    flops = substeps * ops * (6.0 if call in ("gradient", "ascent") else 1.0)
    if call == "ascent":
        flops, per = flops * case["steps"], per * case["steps"]
    if call == "emitters":
        per += 2 * (4 * n + 5 * (n - 1) + 1 + 8 * m) * 4
    return dict(bytes=count * per, flops=flops)


def exact(case, seed):
    """The epilogue's metrics in 64 bits. The other calls return what 1,200
    or more steps of a chaotic 32-bit recurrence give (contacts, stick or
    slip and joint limits flip on a rounding), which no other arithmetic
    reproduces: their outputs have no value in 64 bits."""
    if case["call"] != "epilogue":
        return None
    res, _ = _synthetic_results(case["count"], seed)
    nodes = _population(case, seed).genomes["node_count"]
    nodes = nodes[np.arange(case["count"]) % len(nodes)].astype(np.float64)
    d = {f: res[f].astype(np.float64) for f in NUMBERS}
    total = int(np.round(case["seconds"] * 60))
    ended = np.where(d["fall_time"] > 0, d["fall_time"], d["screened"])
    steps = np.where(ended > 0, np.clip(np.round(ended * 60), 1, total), total)
    lifted = res["lift_lo"].view(np.uint32)
    feet = sum(((lifted >> k) & 1) for k in range(32)).astype(np.float64)
    values = np.stack([d["fitness"], np.clip(d["ground_contact"] / (steps * nodes), 0, 1),
                       np.maximum(d["vertical_oscillation"], 0), np.maximum(d["gait_frequency"], 0),
                       np.maximum(d["height_sum"] / steps, 0), feet, d["screen_x"]], axis=1)
    return dict(metrics=None, values=values, cells=None, rows=None, audit=None, words=None)
