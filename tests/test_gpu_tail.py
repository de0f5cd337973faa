"""Large launches hand their last trials to teams of lanes: against an engine
that keeps every creature on its lane, all fields to the bit. A handed-over
creature carries its positions, velocities, energy stores, touchdown offsets,
result words and step, so the bodies here have touch sensors, tendons and
moved anchors, and the trials a screen and falls before and after it. The
lane kernels of the gradients' runs are compared with teams too."""
import numpy as np
import pytest

import evolution_simulator_gpu_b200 as ce
from evolution_simulator_gpu_b200.configs import WORKLOADS, effects_world_kw

pytestmark = pytest.mark.gpu

EVERY = dict(terrain=2, gravity=14.7, air_retention=0.985, ground_friction=1.0, slope=0.03, wind=-1.0, mud=0.05,
             brambles=3.0, water=0.12, patches=0.5, gaps=0.35, hurdles=0.08, quake=0.05)
TREMORS = dict(effects_world_kw(), terrain=1, quake=0.05)
WORLDS = {"calm": {}, "effects": effects_world_kw(), "tremors": TREMORS, "every": EVERY,
          "mud": dict(mud=0.05, slope=0.03)}
# Bodies of 3 to 24 nodes in equal numbers: large ones enough for a launch of
# their own on lanes.
EVEN = ce.GenSpecPy(seed=5, min_nodes=3, max_nodes=24, muscle_rule=0, max_extra=3, joint_lo_deg=30.0,
                    joint_hi_deg=150.0)


@pytest.fixture(scope="module")
def lanes():
    pytest.importorskip("torch")
    with ce.Engine(0, teams=2) as e:
        yield e


def evolved(pop, seed=1):
    rng = np.random.default_rng(seed)
    m, n = pop.muscles, len(pop.muscles)
    for end in ("anchor_a", "anchor_b"):
        m[end] = np.clip(m[end] + rng.normal(0.0, 0.3, n), 0.0, 1.0)
    m["tendon"] = np.where(rng.random(n) < 0.2, rng.random(n), 0.0)
    m["sensor"] = np.where(rng.random(n) < 0.3, rng.integers(0, 4, n), 255)
    m["reset"] = rng.random(n)
    return pop


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32).reshape(len(a), -1)


@pytest.fixture(scope="module")
def populations():
    cache = {}

    def get(name, count):
        if (name, count) not in cache:
            cache[name, count] = evolved(ce.generate(EVEN if name == "even" else WORKLOADS[name].spec, count))
        return cache[name, count]

    return get


@pytest.mark.parametrize("rate", [60, 120])
@pytest.mark.parametrize("world", sorted(WORLDS))
@pytest.mark.parametrize("name,count", [("effects", 24_576), ("effects", 24_577), ("game", 60_000), ("even", 60_000)])
def test_results_match(engine, lanes, populations, name, count, world, rate):
    """One launch on teams, one that just misses it, one class with a tail (a
    second on teams beside it where there is one), two classes with tails."""
    w = ce.make_world(duration=1.5, rate=rate, screen=(0.8, 0.1), **WORLDS[world])
    wave = ce.pack(populations(name, count), w)
    a, b = engine.run(wave, w)[0], lanes.run(wave, w)[0]
    assert (bits(a) == bits(b)).all()
    assert ((a["screened"] > 0).any() and (a["fall_time"] > 1.0).any()) or world == "calm"


@pytest.mark.parametrize("count", [9_000, 40_000])
@pytest.mark.parametrize("world", ["effects", "mud"])
def test_device_entry_matches(engine, lanes, populations, world, count):
    """Results, metrics and cells of the kernel entry on device arrays."""
    import torch
    w = ce.make_world(duration=1.5, **WORLDS[world])
    pop = populations("effects", count)
    wave = ce.pack(pop, w)

    def up(a):
        return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).cuda()

    ins = [up(a) for a in (wave.lanes, wave.muscles, wave.heads)]
    shapes = up(ce.shape_classes(pop, wave))
    out = []
    for e in (engine, lanes):
        results = torch.zeros((count, 19), dtype=torch.int32, device="cuda")
        cells = torch.zeros(count, dtype=torch.int64, device="cuda")
        metrics = torch.zeros((count, 9), dtype=torch.int32, device="cuda")
        counter = torch.zeros(64, dtype=torch.int32, device="cuda")
        scratch = torch.empty(e.scratch_bytes(ce.world_flags(w), w.rate, wave.max_nodes, wave.max_muscles, count),
                              dtype=torch.uint8, device="cuda")
        e.advance_device_cells(*(a.data_ptr() for a in ins), results.data_ptr(), counter.data_ptr(),
                               scratch.data_ptr(), ce.make_params(w, 0, count), w, wave.max_nodes, wave.max_muscles,
                               shapes.data_ptr(), cells.data_ptr(), metrics.data_ptr(),
                               torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        out.append([a.cpu() for a in (results, cells, metrics)])
    assert all(torch.equal(a, b) for a, b in zip(*out))


def test_generations_with_every_kind_of_launch(engine, lanes, populations):
    """A graph whose generations share one scratch: two classes on lanes with
    tails, all on teams, a class on teams beside one on lanes."""
    w = ce.make_world(duration=1.0, **WORLDS["effects"])
    waves = [ce.pack(populations(*k), w) for k in (("even", 60_000), ("effects", 3_000), ("effects", 60_000))]
    with ce.GenerationGraph(engine, waves, w) as g:
        for _ in range(2):
            g.launch()
            for k, wave in enumerate(waves):
                assert (bits(g.results(k)) == bits(lanes.run(wave, w)[0])).all()


@pytest.mark.parametrize("rate", [60, 120])
@pytest.mark.parametrize("world", sorted(WORLDS))
def test_recordings_match(engine, lanes, populations, world, rate):
    w = ce.make_world(duration=1.0, rate=rate, **WORLDS[world])
    wave = ce.pack(populations("even", 33), w)
    fa, ra = engine.record(wave, w)
    fb, rb = lanes.record(wave, w)
    assert (fa.view(np.uint32) == fb.view(np.uint32)).all()
    assert (bits(ra) == bits(rb)).all()


@pytest.mark.parametrize("name,count,seconds", [("gradients", 1024, 2.0), ("refine", 1024, 2.0), ("effects", 1024, 2.0),
                                                ("gradients", 256, 20.0)])
def test_reruns_on_lanes_reproduce_the_forward_run(engine, lanes, name, count, seconds):
    """On lanes a backward run reruns each segment from its checkpoint and each
    substep from the segment's tape: both land on the forward run's states
    (mismatch bits 0 and 1), and the gradients are those of teams, which rerun
    a segment once and check it against the checkpoints."""
    w = WORKLOADS[name].world(duration=seconds)
    wave = ce.pack(ce.generate(WORKLOADS[name].spec, count), w)
    with engine.forward(wave, w) as a, lanes.forward(wave, w) as b:
        ga, bad_a = a.backward(check=True)
        gb, bad_b = b.backward(check=True)
        plain = b.backward()
    assert not bad_a.any() and not bad_b.any()
    assert (bits(ga) == bits(gb)).all() and (bits(gb) == bits(plain)).all()


@pytest.mark.parametrize("world", ["calm", "effects", "tremors"])
@pytest.mark.parametrize("rate", [60, 120])
def test_gradients_beyond_teams(engine, lanes, world, rate):
    """34,000 creatures are more than backward runs take to teams; the first
    creatures of the batch, alone, go on them."""
    w = ce.make_world(duration=0.6, rate=rate, **WORLDS[world])
    pop = ce.generate(WORKLOADS["gradients"].spec, 34_000)
    wave = ce.pack(pop, w)
    some = np.arange(0, 34_000, 70)
    with engine.forward(wave, w) as t:
        g, bad = t.backward(check=True)
        rows, mm = t.shape
    assert not bad.any()
    with engine.forward(wave.take(some), w) as t:
        h = t.backward()
        assert t.shape == (rows, mm)
    assert (bits(g[some]) == bits(h)).all()
