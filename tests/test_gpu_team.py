"""Trials on teams of lanes equal those of one creature a lane, to the bit.

Both kernels keep the reference's order of operations. An engine that is
given a number of blocks an SM runs one creature a lane whatever the count,
so it is the oracle here: every field of every result, frame and gradient
must match, at the edges of the team sizes (8, 16 and 32 nodes), in compiled
worlds and in worlds whose switches are read at run time.
"""
import numpy as np
import pytest

import evolution_simulator_gpu_b200 as ce
from evolution_simulator_gpu_b200.configs import WORKLOADS, effects_world_kw

pytestmark = pytest.mark.gpu

EVERY = dict(terrain=2, gravity=14.7, air_retention=0.985, ground_friction=1.0, slope=0.03, wind=-1.0, mud=0.05,
             brambles=3.0, water=0.12, patches=0.5, gaps=0.35, hurdles=0.08, quake=0.05)
WORLDS = {
    "calm": {}, "effects": effects_world_kw(), "tremors": dict(effects_world_kw(), terrain=1, quake=0.05),
    "every": EVERY, "mud": dict(mud=0.05, slope=0.03), "rough": dict(terrain=2), "sea": dict(water=0.35, slope=0.15),
    "gaps": dict(gaps=0.35, air_retention=0.985), "brambles": dict(brambles=3.0, hurdles=0.2, wind=-1.0),
    "space": dict(ground=0, wind=-1.0),
}


@pytest.fixture(scope="module")
def lanes():
    pytest.importorskip("torch")
    e = ce.Engine(0, ctas_per_sm=2)
    yield e
    e.close()


def evolved(pop, seed=1):
    """Anchors along the bones, tendons and touch sensors on some muscles."""
    rng = np.random.default_rng(seed)
    m, n = pop.muscles, len(pop.muscles)
    for end in ("anchor_a", "anchor_b"):
        m[end] = np.clip(m[end] + rng.normal(0.0, 0.3, n), 0.0, 1.0)
    m["tendon"] = np.where(rng.random(n) < 0.2, rng.random(n), 0.0)
    m["sensor"] = np.where(rng.random(n) < 0.2, rng.integers(0, 4, n), 255)
    m["reset"] = rng.random(n)
    return pop


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32).reshape(len(a), -1)


def bodies(nodes, muscles, count):
    """Bodies of exactly `nodes` nodes and about `muscles` muscles."""
    return ce.generate(ce.GenSpecPy(seed=9, min_nodes=nodes, max_nodes=nodes, muscle_rule=1, min_muscles=muscles,
                                    max_muscles=muscles, joint_lo_deg=30.0, joint_hi_deg=150.0), count)


@pytest.mark.parametrize("world", sorted(WORLDS))
@pytest.mark.parametrize("rate", [60, 120])
def test_results_match(engine, lanes, world, rate):
    w = ce.make_world(duration=3.0, rate=rate, screen=(1.5, 0.1), **WORLDS[world])
    wave = ce.pack(evolved(ce.generate(WORKLOADS["effects"].spec, 2111)), w)
    a, b = engine.run(wave, w)[0], lanes.run(wave, w)[0]
    assert (bits(a) == bits(b)).all()


@pytest.mark.parametrize("nodes,muscles,count", [(3, 1, 1), (3, 2, 33), (8, 24, 130), (9, 7, 65), (16, 40, 37),
                                                 (17, 96, 9), (32, 96, 5), (32, 1, 70)])
def test_team_sizes_match(engine, lanes, nodes, muscles, count):
    w = ce.make_world(duration=2.0, **effects_world_kw())
    wave = ce.pack(evolved(bodies(nodes, muscles, count)), w)
    assert (bits(engine.run(wave, w)[0]) == bits(lanes.run(wave, w)[0])).all()


def test_two_node_bodies_and_mixed_sizes_match(engine, lanes):
    w = ce.make_world(duration=2.0)
    for n in (2, 3, 5):
        pop = ce.generate(WORKLOADS["refine"].spec, 40)
        wave = ce.pack(pop, w)
        some = wave.take(np.argsort(wave.heads[:, 0] & 255)[[0, -1] * n])
        assert (bits(engine.run(some, w)[0]) == bits(lanes.run(some, w)[0])).all()


def test_trials_that_blow_up_match(engine, lanes):
    """Infinite forces: the weights of zero that the sums leave out count."""
    w = ce.make_world(duration=1.0, **effects_world_kw())
    pop = ce.generate(WORKLOADS["game"].spec, 500)
    wave = ce.pack(pop, w)
    wave.muscles[1::20] *= 1.0
    wave.muscles[4::20] = np.float32(3e38)  # the force cap
    wave.muscles[8::20] = np.float32(1e30)  # the stroke
    a, b = engine.run(wave, w)[0], lanes.run(wave, w)[0]
    assert (a["fitness"] < -1e19).any()
    same = (bits(a) == bits(b)) | (np.isnan(a.view(np.float32).reshape(len(a), -1))
                                   & np.isnan(b.view(np.float32).reshape(len(b), -1)))
    assert same.all()


def test_a_pivot_after_its_bones_end_matches(engine, lanes):
    """Records whose bones are not in parent-first order run bone by bone."""
    w = ce.make_world(duration=2.0)
    wave = ce.pack(bodies(5, 3, 64), w)
    for c in range(0, 64, 3):
        r0 = int(wave.heads[c, 3]) + 5 * 6
        wave.lanes[r0] = 2  # bone 0 (to node 1) hangs from node 2
    assert (bits(engine.run(wave, w)[0]) == bits(lanes.run(wave, w)[0])).all()


@pytest.mark.parametrize("spec,world", [("game", "calm"), ("effects", "effects"), ("refine", "mud")])
@pytest.mark.parametrize("count", [1, 37])
def test_recordings_match(engine, lanes, spec, world, count):
    w = ce.make_world(duration=3.0, **WORLDS[world])
    wave = ce.pack(evolved(ce.generate(WORKLOADS[spec].spec, count)), w)
    fa, ra = engine.record(wave, w)
    fb, rb = lanes.record(wave, w)
    assert (fa.view(np.uint32) == fb.view(np.uint32)).all()
    assert (bits(ra) == bits(rb)).all()


@pytest.mark.parametrize("world", ["calm", "effects", "tremors"])
def test_checkpoints_match(engine, lanes, world):
    w = ce.make_world(duration=1.5, **WORLDS[world])
    wave = ce.pack(ce.generate(WORKLOADS["refine"].spec, 257), w)
    with engine.forward(wave, w) as a, lanes.forward(wave, w) as b:
        steps = ce.trial_steps(w)
        assert (bits(a.results) == bits(b.results)).all()
        ended = np.where(a.results["fall_time"] > 0, np.round(a.results["fall_time"] * 60), steps).astype(int)
        ca, cb = a.checkpoints(steps).view(np.uint32), b.checkpoints(steps).view(np.uint32)
        for c in range(len(wave)):
            n, m = int(wave.heads[c, 0] & 255), int(wave.heads[c, 1])
            rows = a.shape[0]
            cols = np.concatenate([np.arange(2 * n), 2 * rows + np.arange(2 * n), 4 * rows + np.arange(m)])
            k = (ended[c] + 15) // 16
            assert (ca[c, :k, cols] == cb[c, :k, cols]).all()
        assert (a.backward().view(np.uint32) == b.backward().view(np.uint32)).all()


@pytest.mark.parametrize("world", ["calm", "effects", "tremors"])
@pytest.mark.parametrize("nodes,muscles,count", [(2, 1, 3), (3, 2, 33), (8, 24, 9), (9, 7, 13), (16, 40, 5),
                                                 (17, 60, 3), (32, 24, 2)])
def test_gradients_match(engine, lanes, world, nodes, muscles, count):
    """Anchors and tendons, weighted, at 120 substeps a second; the rerun of
    every segment must reproduce the forward run."""
    w = ce.make_world(duration=1.5, rate=120, **WORLDS[world])
    pop = evolved(bodies(nodes, muscles, count) if nodes > 2 else ce.generate(WORKLOADS["refine"].spec, count))
    pop.muscles["sensor"] = 255
    wave = ce.pack(pop, w)
    weights = np.linspace(-2.0, 3.0, len(wave)).astype(np.float32)
    with engine.forward(wave, w) as a, lanes.forward(wave, w) as b:
        ga, bad = a.backward(weights, check=True)
        gb, _ = b.backward(weights, check=True)
    assert not bad.any()
    assert np.isfinite(ga).all() and (ga != 0).any()
    assert (ga.view(np.uint32) == gb.view(np.uint32)).all()
