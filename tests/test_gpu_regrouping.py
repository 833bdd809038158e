"""GVX_LINK_BIN_EVERY sets the steps between two regroupings of a large batch's links."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("every,groupings", [("1", 16), ("3", 6), ("8", 2), ("64", 1), (None, 8)])
def test_regrouping_period(monkeypatch, every, groupings):
    """Of 16 steps of a body above the size from which links are regrouped during a call (200,000
    links), launched one by one: three kernels a step, and three for each grouping.  Unset: every
    fourth step, and launches that may leave it out between them."""
    import gpuvoxels_gb300 as g
    from gpuvoxels_gb300 import synth
    if every is None:
        monkeypatch.delenv("GVX_LINK_BIN_EVERY", raising=False)
    else:
        monkeypatch.setenv("GVX_LINK_BIN_EVERY", every)
    with g.Context(0, 1 << 30) as ctx:
        sim = ctx.load_vxa(synth.slab(42, 42, 42).vxa)
        assert ctx.info(sim).num_link >= 200000
        ctx.step(sim, 16)
        assert ctx.timing()["launches"] == 3 * 16 + 3 * groupings


def test_launch_count_with_contacts():
    """A self-colliding body's step is five kernels (links, watch lists, contacts, voxels, control), and the
    grouping three more: the count a call reports is that of the kernels it launched."""
    import gpuvoxels_gb300 as g
    from gpuvoxels_gb300 import synth
    mats = [dict(E=1e5, rho=1000.0, nu=0.35, cte=0.01, mus=1.0, muk=0.5)]
    with g.Context(0, 256 << 20) as ctx:
        sim = ctx.load_vxa(synth.random_creature(2, (6, 6, 6), 0.6, mats, collision=True, expansion=False).vxa)
        ctx.step(sim, 40)
        ctx.step(sim, 10)
        assert ctx.timing()["launches"] == 5 * 10 + 3
