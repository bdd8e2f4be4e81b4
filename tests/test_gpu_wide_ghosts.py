"""The fused step's tile lists on a mesh with very wide ghost layers, where the
cells a tile depends on reach over more columns of skip marks than on an
ordinary one.  A blast starts at rest in one column of marks and moves into the
tiles beside it; a run that declares its state changed before every step takes
every step over the whole mesh, and both must agree bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAD, NX, NY = 130, 700, 150


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("x", [129, 256, 384, 385, 508])
def test_lists_reach_over_every_mark_column(form, x, monkeypatch):
    import flow_gb300 as fg
    from flow_gb300 import problems, sim as sim_module
    monkeypatch.setattr(problems, "PAD", PAD)
    monkeypatch.setattr(sim_module, "PAD", PAD)
    fg.set_mode(fg.MODE_FUSED)
    p = problems.Problem(NX, NY).boxes(
        [(1.0, 1e-5, 0.0, 0.0, 1.0, 1.0),
         (1.0, 1e3, (x - 0.25) / NX, 70.0 / NY, 4 / NX, 4 / NY)]).with_cfl_dt()
    runs = [fg.MixedSim(p) if form == "mixed" else fg.DeviceSim(p) for _ in range(2)]
    got = [[], []]
    for which, sim in enumerate(runs):
        if form == "fp64":
            sim.initial_timestep()
        for _ in range(40):
            if which:
                fg.lib().gb300_state_changed()
            sim.step()
            got[which].append((sim.mesh.dt, sim.mesh.dt_h))
    for k in ("rho", "e", "u", "v", "rho_u", "rho_v"):
        a, b = runs[0].interior(k), runs[1].interior(k)
        assert np.array_equal(a, b), (k, int(np.count_nonzero(a != b)))
    assert got[0] == got[1]
