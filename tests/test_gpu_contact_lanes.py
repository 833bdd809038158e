"""Eight lanes or one walk a voxel's watch list by the surface voxels and the work items of the batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bodies", [60, 300, 1100], ids=["few_items", "many_items", "too_many_items"])
def test_small_colliding_bodies_together_and_alone(bodies):
    """Each of many small self-colliding bodies moves as it does alone, bit for bit: 60 and 300 of them hold
    so few surface voxels that eight lanes walk a list, 1,100 so many work items that one does."""
    import gpuvoxels_gb300 as g
    from gpuvoxels_gb300 import synth
    mats = [dict(E=1e5, rho=1000.0, nu=0.35, cte=0.02, mus=1.0, muk=0.5), dict(E=1e6, rho=1000.0, nu=0.35, cte=0.0, mus=1.0, muk=0.5)]
    docs = [synth.random_creature(k, (5, 5, 5), 0.5, mats, collision=True, expansion=False).vxa for k in range(12)]
    alone = []
    for d in docs:
        with g.Context(0, 64 << 20) as ctx:
            i = ctx.load_vxa(d)
            ctx.step(i, 300)
            alone.append(ctx.get_state(i))
    with g.Context(0, 4 << 30) as ctx:
        ids = ctx.load_many([docs[k % len(docs)] for k in range(bodies)])
        ctx.step(ids, 300)
        for k in (0, 1, 5, 11, bodies // 2, bodies - 1):
            for x, y in zip(ctx.get_state(ids[k]), alone[k % len(docs)]):
                assert np.array_equal(x, y), k
