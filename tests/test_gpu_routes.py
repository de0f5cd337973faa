"""A launch goes on teams of lanes only where that is the faster: against an
engine that keeps one creature a lane, on bodies of one size at counts where
their number alone would put them on teams. Teams take 1.5 to 2.5 times as
long there."""
import time

import numpy as np
import pytest

import evolution_simulator_gpu_b200 as ce
from evolution_simulator_gpu_b200.configs import WORKLOADS

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lanes():
    pytest.importorskip("torch")
    with ce.Engine(0, teams=2) as e:
        yield e


def bodies(nodes, muscles, count):
    return ce.generate(ce.GenSpecPy(seed=9, min_nodes=nodes, max_nodes=nodes, muscle_rule=1, min_muscles=muscles,
                                    max_muscles=muscles, joint_lo_deg=30.0, joint_hi_deg=150.0), count)


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.parametrize("nodes,muscles,count", [(3, 1, 24_576), (3, 1, 28_000), (9, 1, 24_576), (17, 8, 24_576),
                                                 (17, 8, 28_000), (24, 1, 24_576)])
def test_trials(engine, lanes, nodes, muscles, count):
    w = ce.make_world(duration=1.5)
    wave = ce.pack(bodies(nodes, muscles, count), w)
    a, b = engine.run(wave, w)[0], lanes.run(wave, w)[0]
    assert (bits(a) == bits(b)).all()
    mine, theirs = (min(e.run(wave, w)[1] for _ in range(3)) for e in (engine, lanes))
    assert mine < 1.15 * theirs


@pytest.mark.parametrize("nodes,muscles,count", [(3, 1, 16_384), (9, 8, 32_768), (17, 8, 32_768)])
def test_backward_runs(engine, lanes, nodes, muscles, count):
    w = ce.make_world(duration=0.5)
    wave = ce.pack(bodies(nodes, muscles, count), w)
    took, grads = [], []
    for e in (engine, lanes):
        with e.forward(wave, w) as tape:
            grads.append(tape.backward())
            seconds = []
            for _ in range(2):
                tape.backward()
                seconds.append(tape.seconds[1])
            took.append(min(seconds))
    assert (bits(grads[0]) == bits(grads[1])).all()
    assert took[0] < 1.15 * took[1]


def test_a_stream_of_batches(engine, lanes):
    """Four submissions in flight share the schedulers: each as if it were
    alone on teams takes 1.4 times as long as on lanes."""
    w = ce.make_world(duration=4.0)
    spec = WORKLOADS["small"].spec
    waves = [ce.pack(ce.generate(spec, 16_384, first=16_384 * k), w) for k in range(4)]

    def stream(e):
        out, sent = [], 0
        start = time.perf_counter()
        while len(out) < 8:
            while sent < 8 and e.free_slots():
                e.submit(waves[sent % 4], w)
                sent += 1
            out.append(e.poll(60.0)[1])
        return time.perf_counter() - start, out

    took, results = [], []
    for e in (engine, lanes):
        stream(e)
        runs = [stream(e) for _ in range(3)]
        took.append(min(r[0] for r in runs))
        results.append(runs[0][1])
    assert all((bits(a) == bits(b)).all() for a, b in zip(*results))
    assert took[0] < 1.15 * took[1]


def test_a_backward_run_holds_tapes_for_its_teams_only(engine):
    """1,000 bodies of up to 8 nodes, 4 to a warp, and one of more than 16: 251
    warps of 1.2 MB, not one for every body because the largest fills one."""
    import torch
    w = ce.make_world(duration=0.5)
    pop = ce.generate(WORKLOADS["effects"].spec, 3000)
    nodes = pop.genomes["node_count"]
    wave = ce.pack(pop.subset(np.concatenate([np.where(nodes <= 8)[0][:1000], np.where(nodes > 16)[0][:1]])), w)
    assert len(wave) == 1001
    with engine.forward(wave, w) as tape:
        tape.backward()  # kernels and their local memory are loaded
    free = torch.cuda.mem_get_info()[0]
    with engine.forward(wave, w) as tape:
        tape.backward()
        assert free - torch.cuda.mem_get_info()[0] < 0.6e9


@pytest.mark.parametrize("max_nodes,count", [(24, 40_000), (16, 60_000)])
def test_two_classes(engine, lanes, max_nodes, count):
    """Bodies of 3 to `max_nodes` nodes, of which the large ones alone would
    pay for teams: beside the small ones' lanes they took 1.2 to 1.5 times as
    long as both on lanes."""
    w = ce.make_world(duration=0.5)
    spec = ce.GenSpecPy(seed=5, min_nodes=3, max_nodes=max_nodes, muscle_rule=0, max_extra=3, joint_lo_deg=30.0,
                        joint_hi_deg=150.0)
    wave = ce.pack(ce.generate(spec, count), w)
    a, b = engine.run(wave, w)[0], lanes.run(wave, w)[0]
    assert (bits(a) == bits(b)).all()
    mine, theirs = (min(e.run(wave, w)[1] for _ in range(4)) for e in (engine, lanes))
    assert mine < 1.1 * theirs
