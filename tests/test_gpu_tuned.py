"""What ce_autotune leaves alone: the choice of teams of lanes, which is made
when an engine is opened, and the size of the device entry's scratch, which a
caller may have allocated before."""
import pytest

import evolution_simulator_gpu_b200 as ce
from evolution_simulator_gpu_b200.configs import WORKLOADS, effects_world_kw

pytestmark = pytest.mark.gpu

SIZES = [(3, 1), (6, 8), (10, 24), (17, 40), (32, 96)]


def scratch(engine, world, count):
    return [engine.scratch_bytes(ce.world_flags(world), world.rate, n, m, count) for n, m in SIZES]


def test_a_small_sample_times_the_lane_settings(engine):
    """The settings shape launches of one creature a lane: a sample that small
    launches would run on teams (here five times as fast) is timed on lanes,
    and the engine goes on running such launches on teams."""
    world = ce.make_world(duration=2.0, **effects_world_kw())
    sample = ce.pack(ce.generate(WORKLOADS["effects"].spec, 2048), world)
    engine.run(sample, world)
    team = min(engine.run(sample, world)[1] for _ in range(3))
    with ce.Engine(0) as tuned:
        best, secs = tuned.autotune(sample, world)
        after = min(tuned.run(sample, world)[1] for _ in range(3))
    assert secs > 2.0 * team
    assert best["teams"] == 1
    assert after < 0.5 * secs
    with ce.Engine(0, **best) as again:
        assert min(again.run(sample, world)[1] for _ in range(3)) < 0.5 * secs


@pytest.mark.parametrize("opts,teams", [(dict(), True), (dict(ctas_per_sm=3), False), (dict(ctas_per_sm=3, teams=1), True),
                                        (dict(teams=2), False)])
def test_teams_are_chosen_when_an_engine_is_opened(opts, teams):
    """Seen from outside by the scratch of a large launch, of which the
    creatures that it hands over to teams are a part."""
    world = ce.make_world(duration=1.0)
    small = ce.pack(ce.generate(WORKLOADS["small"].spec, 500), world)
    with ce.Engine(0, **opts) as e, ce.Engine(0, **dict(opts, teams=2)) as lanes:
        large = scratch(e, world, 300_000)
        best, _ = e.autotune(small, world)
        assert best["teams"] == (1 if teams else 2)
        assert all((a > b) == teams for a, b in zip(large, scratch(lanes, world, 300_000)))


@pytest.mark.parametrize("count", [1, 1000, 300_000])
def test_scratch_does_not_depend_on_what_the_tuner_changes(count):
    """The autotuner sets 0 or 3 blocks an SM on any engine: scratch sized
    before has to hold the largest grid it may choose. Nothing is launched
    into the scratch here."""
    world = ce.make_world(duration=1.0)
    small = ce.pack(ce.generate(WORKLOADS["small"].spec, 300), world)
    with ce.Engine(0) as plain:
        want = scratch(plain, world, count)
    for ctas in (1, 2, 3):
        with ce.Engine(0, ctas_per_sm=ctas, teams=1) as e:
            assert scratch(e, world, count) == want
            e.autotune(small, world)
            assert scratch(e, world, count) == want
