"""Results and poses of many simulations taken together equal those taken one by one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _docs(sides):
    from gpuvoxels_gb300 import synth
    return [synth.random_creature(40 + i, (s, s + 1, max(1, s - 1)), 0.8, stop_time=1.0).vxa for i, s in enumerate(sides)]


@pytest.mark.parametrize("sides", [[3], [1, 4], [2, 5, 7, 3, 6], [16, 20, 18, 5]], ids=["one", "two", "five", "threaded"])
def test_results_together_and_alone(sides):
    """The same steps, times, centres of mass, fitness and travelled distance, bit for bit, whether
    the engine finishes the simulations together (sizes below and above its threads' threshold) or
    one at a time; and the same poses."""
    import gpuvoxels_gb300 as g
    docs = _docs(sides)

    def fields(r):
        return (r.steps, r.status, r.num_voxel, r.current_time, r.fitness_score, tuple(r.initial_center_of_mass),
                tuple(r.current_center_of_mass), r.total_distance_of_all_voxels)

    with g.Context(0, 512 << 20) as ctx:
        ids = ctx.load_many(docs)
        ctx.run(ids, g.BATCHED, 30)
        together = [fields(ctx.result(i)) for i in ids]
        pos, q, fl, off = ctx.get_states(ids)
    alone = []
    with g.Context(0, 512 << 20) as ctx:
        for k, d in enumerate(docs):
            i = ctx.load_vxa(d)
            ctx.run(i, g.BATCHED, 30)
            alone.append(fields(ctx.result(i)))
            p, w, f = ctx.get_state(i)
            assert np.array_equal(p, pos[off[k]:off[k + 1]]) and np.array_equal(w, q[off[k]:off[k + 1]])
    assert together == alone
    assert all(t[0] == 30 for t in together)


@pytest.mark.parametrize("slots", [16, 1])
def test_contacts_alone_and_in_a_large_batch(slots):
    """A self-colliding creature's poses are the same bits whether its contact lists are walked by
    eight lanes a voxel (alone) or by one (beside 60,000 other surface voxels); with one contact
    slot a voxel every further contact goes through the spill pool."""
    import gpuvoxels_gb300 as g
    from gpuvoxels_gb300 import synth
    mats = [dict(E=1e5, rho=1000.0, nu=0.35, cte=0.01, mus=1.0, muk=0.5), dict(E=1e6, rho=1000.0, nu=0.35, cte=0.0, mus=1.0, muk=0.5)]
    small = [synth.random_creature(k, (12, 12, 12), 0.5, mats, collision=True, expansion=False).vxa for k in (3, 4)]
    big = [synth.random_creature(k, (40, 40, 40), 0.5, mats, collision=True, expansion=False).vxa for k in (5, 6)]
    poses = []
    for docs in (small, small + big):
        with g.Context(0, 2 << 30) as ctx:
            ctx.set_contact_slots(slots)
            ids = ctx.load_many(docs)
            ctx.step(ids, 700)
            pos, q, fl, off = ctx.get_states(ids)
            n = off[2]
            poses.append((pos[:n], q[:n], fl[:n]))
    assert all(np.array_equal(a, b) for a, b in zip(*poses))


@pytest.mark.parametrize("side", [34, 68], ids=["every_warp_busy", "many_chunks_a_warp"])
def test_a_creature_beside_a_large_body(side):
    """A creature's poses are the same bits alone (few warps an SM) and beside a solid body that gives
    every resident warp a chunk of links, or many: the builds of the step kernels for those."""
    import gpuvoxels_gb300 as g
    from gpuvoxels_gb300 import synth
    docs = [synth.config0_creature(6).vxa, synth.slab(side, side, side, seed=2).vxa]
    poses = []
    for d in (docs[:1], docs):
        with g.Context(0, 2 << 30) as ctx:
            ids = ctx.load_many(d)
            ctx.step(ids, 40)
            pos, q, fl, off = ctx.get_states(ids)
            n = off[1]
            poses.append((pos[:n], q[:n], fl[:n]))
    assert all(np.array_equal(a, b) for a, b in zip(*poses))
