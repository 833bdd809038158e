"""The integer-pipe forms of the link and voxel updates: their exact operations against IEEE arithmetic (host and
device), and whole bodies on it and on the plain form it falls back to against the CPU oracle."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _check(tmp_path, cmd, cases):
    exe = str(tmp_path / "fp64_band_check")
    subprocess.run(cmd + ["-o", exe, os.path.join(HERE, "fp64_band_check.cpp")], check=True)
    r = subprocess.run([exe, str(cases)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_band_operations_match_ieee_on_the_host(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host compiler")
    _check(tmp_path, [cxx, "-O2", "-std=c++17", "-ffp-contract=off"], 3000000)


@pytest.mark.gpu
def test_band_operations_match_the_fp64_instructions(tmp_path):
    from gpuvoxels_gb300 import build
    _check(tmp_path, [build.nvcc(), "-x", "cu", "-O3", "-std=c++17", "-fmad=false"] + build.ARCH, 200000000)


MAT = dict(E=1e6, rho=1000.0, nu=0.35, cte=0.01, mus=1.0, muk=0.5)
# (name, lattice x, y, z, materials, phases equal, world options): bodies that keep to the plain form
# by exact zeros (a straight beam, no actuation, equal phases; no bond damping), that leave it after
# some steps, and that hardly ever take it
BODIES = [("beam_1x1x9", (1, 1, 9), [MAT], True, {}), ("one_link", (2, 1, 1), [MAT], False, {}),
          ("still_block", (3, 3, 3), [MAT], False, dict(vary_temp=False)), ("plate_5x5x1", (5, 5, 1), [MAT], False, {}),
          ("undamped", (4, 4, 4), [MAT], False, dict(damping=(0.0, 0.8, 0.01))),
          ("no_poisson", (4, 3, 5), [dict(MAT, nu=0.0)], False, {}),
          ("two_stiffnesses", (7, 6, 5), [MAT, dict(MAT, E=2e5, cte=0.0)], False, {}),
          ("no_floor", (4, 4, 3), [MAT], False, dict(floor=False)),
          ("sliding", (6, 6, 2), [dict(MAT, mus=0.3, muk=0.2)], False, dict(temp_period=0.004)),
          ("frictionless", (5, 5, 2), [dict(MAT, mus=0.0, muk=0.0)], False, dict(temp_period=0.004)),
          ("undamped_voxels", (4, 4, 4), [MAT], False, dict(damping=(1.0, 0.0, 0.0))),
          ("large_angles", (9, 3, 3), [dict(MAT, E=1e5, cte=0.02)], False, dict(temp_period=0.02))]


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [1, 3, 5, 70, 400])
@pytest.mark.parametrize("name,side,mats,same,kw", BODIES, ids=[b[0] for b in BODIES])
def test_links_against_the_oracle(name, side, mats, same, kw, steps):
    """Positions within 1e-6 voxel sizes (the parity bound of whole bodies), flags equal, and link
    flags without the engine's own bit.  The steps lie on both sides of the plain form's retries."""
    import gpuvoxels_gb300 as g
    from gpuvoxels_gb300 import synth
    from oracle.oracle import OracleSim, desc_from_vxa
    rng = np.random.default_rng(11)
    X, Y, Z = side
    grid = rng.integers(1, len(mats) + 1, size=(Z, Y, X)).astype(np.int32)
    phase = np.zeros((Z, Y, X)) if same else rng.random((Z, Y, X))
    vxa = synth.vxa_document(grid, phase, mats, **kw)
    with g.Context(0, 256 << 20) as ctx:
        sim = ctx.load_vxa(vxa)
        ctx.step(sim, steps)
        v, l = ctx.voxel_state(sim), ctx.link_state(sim)
    o = OracleSim(desc_from_vxa(vxa))
    o.step(steps)
    w = o.voxel_state()
    assert np.abs(v["pos"] - w["pos"]).max() <= 1e-6 * 0.01
    assert np.abs(v["orient"] - w["orient"]).max() <= 1e-6
    static = (v["flags"] >> 6) & 1
    assert np.array_equal(static, (w["flags"] & 8) >> 3) and v["flags"].max() < 1 << 15
    assert l["flags"].max() < 128 and np.isfinite(l["pos2"]).all()
