"""The integer-pipe forms of the link and voxel updates store the bits of the plain forms: whole bodies
stepped by the library and by one whose exact kernels are compiled with the plain forms alone
(GVX_PLAIN_FORMS), and by the library in calls that group its elements at other steps, so that they take
either form at other times."""
import json
import os
import subprocess
import sys
import zlib

import numpy as np
import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
MAT = dict(E=1e6, rho=1000.0, nu=0.35, cte=0.01, mus=1.0, muk=0.5)
SOFT = dict(MAT, E=1e5, cte=0.02)
STEPS = (1, 5, 20, 400)


def _block(side, mats, phase=None, **kw):
    from gpuvoxels_gb300 import synth
    X, Y, Z = side
    rng = np.random.default_rng(X * 100 + Y * 10 + Z)
    grid = rng.integers(1, len(mats) + 1, size=(Z, Y, X)).astype(np.int32)
    ph = rng.random((Z, Y, X)) if phase is None else np.full((Z, Y, X), float(phase))
    return synth.vxa_document(grid, ph, mats, **kw)


def _bodies():
    """name -> (document, voxels of the plane x = 0 fixed): bodies that hardly ever take the plain form,
    whose exact zeros last (equal phases, no actuation, no damping, fixed voxels), that slide, lie
    still or fall, with small and large angles."""
    from gpuvoxels_gb300 import synth
    plastic = dict(MAT, mech="<MatModel>2</MatModel><Plastic_Mod>2e5</Plastic_Mod><Yield_Stress>2e3</Yield_Stress><Fail_Stress>6e3</Fail_Stress>")
    cilia = _block((5, 5, 4), [dict(MAT, mech="<Cilia>1</Cilia>")]).replace("<Simulator>", "<Simulator><EnableCilia>1</EnableCilia>", 1)
    cilia = cilia.replace("</Data>", "</Data><BaseCiliaForce>" + 4 * ("<Layer><![CDATA[" + ",".join(["0.001,0,0.001"] * 25) + "]]></Layer>") +
                          "</BaseCiliaForce>", 1)
    return {
        "creature": (synth.config0_creature(5).vxa, False),
        "two_stiffnesses": (_block((9, 8, 7), [MAT, dict(MAT, E=2e5, cte=0.0)]), False),
        "large_angles": (_block((12, 3, 3), [SOFT], temp_period=0.02), False),
        "sliding": (_block((6, 6, 2), [dict(MAT, mus=0.3, muk=0.2)], temp_period=0.004), False),
        "frictionless": (_block((5, 5, 2), [dict(MAT, mus=0.0, muk=0.0)], temp_period=0.004), False),
        "undamped_bonds": (_block((5, 4, 4), [MAT], damping=(0.0, 0.8, 0.01)), False),
        "undamped_voxels": (_block((5, 4, 4), [MAT], damping=(1.0, 0.0, 0.0)), False),
        "no_poisson": (_block((4, 5, 6), [dict(MAT, nu=0.0)]), False),
        "equal_phases": (_block((8, 8, 8), [MAT], 0.1), False),
        "equal_phases_odd": (_block((7, 5, 9), [SOFT], 0.3), False),
        "still": (_block((4, 4, 5), [MAT], 0.0, vary_temp=False), False),
        "falling": (_block((4, 4, 4), [MAT], 0.0, vary_temp=False, floor=False), False),
        "beam": (_block((1, 1, 9), [MAT], 0.0), False),
        "cantilever": (_block((10, 4, 3), [SOFT], floor=False), True),
        "cantilever_equal": (_block((9, 3, 3), [MAT], 0.2), True),
        "expansion_off": (_block((5, 5, 5), [MAT], expansion=False), False),
        "plastic": (_block((5, 4, 4), [plastic]), False),
        "cilia": (cilia, False),
        "collide": (synth.random_creature(9, (9, 9, 9), 0.5, [SOFT, dict(MAT, cte=0.0)], collision=True, expansion=False).vxa, False),
    }


def _state(ctx, sim):
    """A checksum of each field of the voxels' and the links' state."""
    out = {}
    for kind, st in (("voxel", ctx.voxel_state(sim)), ("link", ctx.link_state(sim))):
        for f, a in st.items():
            out[f"{kind}.{f}"] = zlib.crc32(np.ascontiguousarray(a).tobytes())
    return out


def _load(ctx, g, doc, fixed):
    sim = ctx.load_vxa(doc)
    if fixed:
        for v in np.flatnonzero(g.inspect_vxa(doc)["voxels"][:, 0] == 0):
            ctx.set_external(sim, int(v), 0x3F)
    return sim


def _alone(schedule):
    """State checksums of every body after each of STEPS, each body alone: `schedule` is 'chunks' (one call
    from each of STEPS to the next), 'single' (calls of one step: elements grouped in every step) or
    'plain' (PLAIN mode)."""
    import gpuvoxels_gb300 as g
    got = {}
    for name, (doc, fixed) in _bodies().items():
        with g.Context(0, 256 << 20) as ctx:
            sim = _load(ctx, g, doc, fixed)
            at = 0
            for n in STEPS:
                if schedule == "single":
                    for _ in range(n - at):
                        ctx.step(sim, 1)
                else:
                    ctx.step(sim, n - at, g.PLAIN if schedule == "plain" else g.BATCHED)
                at = n
                got[f"{name}@{n}"] = _state(ctx, sim)
    return got


def _together(side):
    """State checksums of every body after 20 and 400 steps beside a solid body: with `side` 34 every
    resident warp has work, with 68 much of it (then after 20 steps only)."""
    import gpuvoxels_gb300 as g
    from gpuvoxels_gb300 import synth
    got = {}
    with g.Context(0, 3 << 30) as ctx:
        ids = {name: _load(ctx, g, doc, fixed) for name, (doc, fixed) in _bodies().items()}
        big = ctx.load_vxa(synth.slab(side, side, side, seed=2).vxa)
        at = 0
        for n in (20, 400) if side < 60 else (20,):
            ctx.step(list(ids.values()) + [big], n - at)
            at = n
            for name, sim in ids.items():
                got[f"{name}@{n}"] = _state(ctx, sim)
            got[f"solid@{n}"] = _state(ctx, big)
    return got


RUNS = {"chunks": lambda: _alone("chunks"), "single": lambda: _alone("single"), "plain": lambda: _alone("plain"),
        "beside_34": lambda: _together(34), "beside_68": lambda: _together(68)}


def main(lib, out, which):
    from gpuvoxels_gb300 import build
    import gpuvoxels_gb300 as g
    if lib:
        build.LIB = lib
    g.library(build_if_missing=False)
    with open(out, "w") as f:
        json.dump({w: RUNS[w]() for w in which.split(",")}, f)


def _run(tmp, tag, lib, which):
    out = str(tmp / f"{tag}.json")
    r = subprocess.run([sys.executable, os.path.abspath(__file__), lib, out, which], cwd=ROOT, capture_output=True, text=True, timeout=900,
                       env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0, r.stdout + r.stderr
    with open(out) as f:
        return json.load(f)


@pytest.fixture(scope="module")
def states(tmp_path_factory):
    """The library's states, and those of its exact kernels compiled with the plain forms alone."""
    from gpuvoxels_gb300 import build
    tmp = tmp_path_factory.mktemp("forms")
    build.build()
    exe, src = build.nvcc(), "kernels_exact.cu"
    obj, lib = str(tmp / "plain.o"), str(tmp / "plain.so")
    subprocess.run([exe, "-c", os.path.join(build.CSRC, src), "-o", obj, "-DGVX_PLAIN_FORMS"] + build._flags(src), check=True, capture_output=True)
    rest = [os.path.join(build.OUT_DIR, s + ".o") for s in build.SOURCES if s != src]
    subprocess.run([exe, "-shared", "-o", lib, obj] + rest + build.ARCH + ["-cudart", "static"], check=True, capture_output=True)
    plain = _run(tmp, "plain", lib, "chunks,beside_34,beside_68")
    return plain, _run(tmp, "forms", "", ",".join(RUNS))


@pytest.mark.gpu
@pytest.mark.parametrize("run", list(RUNS))
def test_whole_bodies_have_the_bits_of_the_plain_forms(states, run):
    """Every field of every voxel's and link's state, flags among them, after 1, 5, 20 and 400 steps."""
    plain, forms = states
    want = plain[run if run.startswith("beside") else "chunks"]
    got = forms[run]
    assert set(got) == set(want) and len(got) >= 19
    bad = [f"{k} {f}" for k in got for f in got[k] if got[k][f] != want[k][f]]
    assert not bad, bad[:20]


@pytest.mark.gpu
def test_bodies_beside_others_as_alone(states):
    """What a body does does not depend on those it is batched with."""
    _, forms = states
    alone = forms["chunks"]
    for run in ("beside_34", "beside_68"):
        bad = [k for k, st in forms[run].items() if not k.startswith("solid") and st != alone[k]]
        assert not bad, (run, bad)


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [1, 20, 200])
def test_angle_modes_against_the_oracle(steps):
    """Each link's angle mode is the oracle's."""
    import gpuvoxels_gb300 as g
    from oracle.oracle import OracleSim, desc_from_vxa
    bodies = _bodies()
    seen = set()
    for name in ("creature", "two_stiffnesses", "large_angles", "equal_phases_odd", "sliding"):
        doc = bodies[name][0]
        with g.Context(0, 256 << 20) as ctx:
            sim = ctx.load_vxa(doc)
            ctx.step(sim, steps)
            small = ctx.link_state(sim)["flags"] & 1
        o = OracleSim(desc_from_vxa(doc))
        o.step(steps)
        assert np.array_equal(small, o.link_state()["smallAngle"]), name
        seen |= set(small.tolist())
    assert steps == 1 or seen == {0, 1}


if __name__ == "__main__":
    main(*sys.argv[1:])
