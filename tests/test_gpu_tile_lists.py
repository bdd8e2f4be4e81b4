"""The fused step visits only the tiles its previous step's lists name, at tile
heights chosen from the lists' lengths.  A caller that declares its state
changed before every step (gb300_state_changed) gets the same step over the
whole mesh, so both must agree bit for bit, step after step: state, velocities,
timestep and totals.  The fields put moving cells where the lists have their
edges: in corners (ghost images), crossing 127- and 128-column tiles and 16-row
bands, apart from one another, reaching a wall, and along a whole row and
column; meshes of one tile column, of ragged and of power-of-two sides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "e", "u", "v", "rho_u", "rho_v")


def boxes(w, h, *cells):
    """Blasts of 4x4 cells at the given cells on a w x h mesh at rest."""
    return [(1.0, 1e-5, 0.0, 0.0, 1.0, 1.0)] + [
        (1.0, 1e3, (x + 0.25) / w - 0.5 / w, (y + 0.25) / h - 0.5 / h, 4 / w, 4 / h)
        for x, y in cells]


def problems_with_lists():
    from flow_gb300 import problems
    P = problems.Problem
    return {
        "corners_513x257": P(513, 257).boxes(boxes(513, 257, (0, 0), (509, 253))).with_cfl_dt(),
        "apart_1024x256": P(1024, 256).boxes(boxes(1024, 256, (125, 14), (900, 200))).with_cfl_dt(),
        "narrow_100x900": P(100, 900).boxes(boxes(100, 900, (60, 450))).with_cfl_dt(),
        "wall_260x530": P(260, 530).boxes(boxes(260, 530, (250, 30))).with_cfl_dt(),
        "row_front_400x300": P(400, 300).boxes(
            [(0.125, 2.0, 0.0, 0.0, 1.0, 1.0), (1.0, 2.5, 0.0, 0.0, 1.0, 0.4)]).with_cfl_dt(),
        "column_front_777x211": problems.sod(777, 211),
    }


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("name", ["corners_513x257", "apart_1024x256", "narrow_100x900",
                                  "wall_260x530", "row_front_400x300", "column_front_777x211"])
def test_listed_steps_equal_whole_steps(name, form):
    import flow_gb300 as fg
    fg.set_mode(fg.MODE_FUSED)
    p = problems_with_lists()[name]
    runs = [fg.MixedSim(p) if form == "mixed" else fg.DeviceSim(p) for _ in range(2)]
    got = [[], []]
    for which, sim in enumerate(runs):
        if form == "fp64":
            sim.initial_timestep()
        for tt in range(48):
            if which:
                fg.lib().gb300_state_changed()
            sim.step()
            got[which].append((sim.mesh.dt, sim.mesh.dt_h) + sim.conservation())
    assert got[0] == got[1], next(k for k, (a, b) in enumerate(zip(*got)) if a != b)
    for k in FIELDS:
        a, b = runs[0].interior(k), runs[1].interior(k)
        assert np.array_equal(a, b), (k, int(np.count_nonzero(a != b)))
