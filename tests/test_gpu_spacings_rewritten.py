"""A caller may write new spacings into the mesh arrays between two steps: the
next step takes them, whether the mesh was uniform, of powers of two or neither
before and after.  The field moves everywhere (no tile is at rest); a run that
declares the change (gb300_state_changed) must give the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def set_spacings(sim, scale, kind):
    import torch
    for axis, n in (("x", sim.nx), ("y", sim.ny)):
        h = scale / 64
        cell = np.full(n + 1, h)
        if kind == "stretched":
            cell = h * (1.0 + 0.3 * np.sin(np.linspace(0.0, 4.0, n + 1)))
        elif kind == "halves":
            cell[n // 2:] = 2.0 * h
        edge = np.concatenate([cell[:1], 0.5 * (cell[1:] + cell[:-1])]) if kind != "uniform" else cell
        sim.mesh_arrays["celld" + axis].copy_(torch.from_numpy(cell))
        sim.mesh_arrays["edged" + axis].copy_(torch.from_numpy(edge))


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("before,after", [
    ((1.0, "uniform"), (1.25, "uniform")), ((1.1, "uniform"), (1.25, "uniform")),
    ((1.0, "uniform"), (2.0, "uniform")), ((1.1, "uniform"), (1.1, "stretched")),
    ((1.0, "halves"), (1.25, "halves")), ((1.1, "stretched"), (2.0, "uniform"))])
def test_new_spacings_are_taken(form, before, after):
    import flow_gb300 as fg
    from flow_gb300 import problems
    fg.set_mode(fg.MODE_FUSED)
    p = problems.smooth_random(200, np.random.default_rng(11))
    p.dt_param *= 0.2
    runs = [fg.MixedSim(p) if form == "mixed" else fg.DeviceSim(p) for _ in range(2)]
    got = [[], []]
    for which, sim in enumerate(runs):
        set_spacings(sim, *before)
        if form == "fp64":
            sim.initial_timestep()
        for tt in range(10):
            if tt in (4, 7):
                set_spacings(sim, *(after if tt == 4 else before))
                if which:
                    fg.lib().gb300_state_changed()
            sim.step()
            got[which].append((sim.mesh.dt, sim.mesh.dt_h))
    assert got[0] == got[1]
    for k in ("rho", "e", "u", "v", "rho_u", "rho_v"):
        assert np.array_equal(runs[0].interior(k), runs[1].interior(k)), k
