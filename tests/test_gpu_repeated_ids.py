"""An id given more than once in a call is one simulation: stepped, run and finished once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["PLAIN", "BATCHED"])
@pytest.mark.parametrize("sides", [[4, 5], [22, 21]], ids=["small", "threaded"])
def test_repeated_ids_are_one_simulation(mode, sides):
    """The same poses and results, bit for bit, and the same count of voxel steps, as from ids given
    once; sizes below and above the one from which results are finished by several threads.  (Every
    voxel position is kept for the report, so a result finished twice would write its list twice.)"""
    import gpuvoxels_gb300 as g
    from gpuvoxels_gb300 import synth
    docs = [synth.random_creature(70 + k, (s, s, s), 0.9, stop_time=1.0).vxa.replace(
        "<Simulator>", "<Simulator><SavePositionOfAllVoxels>1</SavePositionOfAllVoxels>", 1)
        for k, s in enumerate(sides)]
    got = []
    for pick in ([0, 1], [0, 1, 0, 0, 1]):
        with g.Context(0, 1 << 30) as ctx:
            ids = ctx.load_many(docs)
            ctx.step([ids[k] for k in pick], 7, getattr(g, mode))
            work = [ctx.timing()["voxel_steps"]]
            ctx.run([ids[k] for k in pick], getattr(g, mode), 16)
            work.append(ctx.timing()["voxel_steps"])
            rs = [ctx.result(i) for i in ids]
            pos, q, fl, off = ctx.get_states(ids)
            got.append((work, [(r.steps, r.status, r.current_time, r.fitness_score, tuple(r.current_center_of_mass),
                                r.total_distance_of_all_voxels) for r in rs], pos, q, fl))
    a, b = got
    assert a[0] == b[0] and a[1] == b[1] and all(r[0] == 23 for r in a[1])
    assert all(np.array_equal(x, y) for x, y in zip(a[2:], b[2:]))


@pytest.mark.parametrize("order", ["SERVE_FCFS", "SERVE_LEAST_WORK", "SERVE_LONG_LANE"])
def test_an_id_submitted_again_waits_for_its_turn(order):
    """A request whose simulation is running waits until it is done and then runs it afresh: each
    submission gives one result, all of a simulation's the same, and others are not held up."""
    import gpuvoxels_gb300 as g
    from gpuvoxels_gb300 import synth
    with g.Context(0, 256 << 20) as ctx:
        ctx.set_serving(getattr(g, order))
        ids = ctx.load_many([synth.random_creature(80 + k, (4 + k, 4, 4), 0.9, stop_time=100.0).vxa for k in range(3)])
        for i in (ids[0], ids[1], ids[0], ids[2], ids[0]):
            ctx.submit(i, 100)
        got, polls = [], 0
        while ctx.pending() and polls < 100:
            got += ctx.poll(32)
            polls += 1
        assert ctx.pending() == 0
        assert sorted(r.id for r in got) == sorted([ids[0]] * 3 + [ids[1], ids[2]])
        assert [r.steps for r in got] == [100] * 5
        first = [(r.current_time, tuple(r.current_center_of_mass), r.total_distance_of_all_voxels) for r in got if r.id == ids[0]]
        assert first[0] == first[1] == first[2]
        assert {r.id for r in got[:3]} == set(ids)
