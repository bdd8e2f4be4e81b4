"""The bit-exact timestep minimum where the FP32 ranks that leave most cells
out do not hold: densities and energies so small that a viscous stress which
sets the timestep is below the smallest normal FP32 number.  The timestep must
be the oracle's, from one call on given fields and over whole steps.

A cell of negative energy has a NaN candidate, and the reference's minimum over
NaNs depends on the order it is taken in: only a step with such a candidate
(from the energies and stresses the minimum is taken over) may differ, and ends
its run.
"""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

GAM = 1.4


@pytest.fixture
def fg():
    import flow_gb300
    flow_gb300.set_mode(flow_gb300.MODE_EXACT)
    yield flow_gb300
    flow_gb300.set_mode(flow_gb300.MODE_FUSED)


# Density, energy, the largest stress, and the width of the mesh.  The first two
# have stresses below 2^-126 (1.2e-38) that set the timestep; in the next the
# ranks themselves, or the square of the reciprocal spacing, leave FP32's normal
# range; the last are ordinary.
@pytest.mark.parametrize("rho,e,q,width", [
    (1e-25, 3e-15, 1e-39, 1.0), (1e-29, 1e-10, 9e-39, 1e-4), (1e-29, 1e-45, 2e-70, 1e-17),
    (1.0, 1e-50, 1e-50, 1e-18), (1e-3, 1e-3, 1e-6, 1e21), (1e29, 1e-2, 1e27, 1.0),
    (1.0, 1.0, 1e-39, 1.0), (1.0, 1.0, 1.0, 1.0)])
@pytest.mark.parametrize("stressed", [1, 40])
def test_minimum_of_small_fields(fg, rho, e, q, width, stressed):
    import torch
    from flow_gb300 import problems
    nx, ny = 64, 48
    p = problems.Problem(nx, ny, width=width, height=width, max_dt=1e300)
    hm = O.HostMesh(nx, ny, width=width, height=width, dt=p.dt_param, max_dt=1e300)
    st = O.HostState(hm)
    rng = np.random.default_rng(stressed)
    shape = (p.ny, p.nx)
    fields = {"rho": rho * rng.uniform(0.9, 1.1, shape), "e": e * rng.uniform(0.5, 1.0, shape),
              "Qxx": np.zeros(shape), "Qyy": np.zeros(shape)}
    for k in ("Qxx", "Qyy"):
        at = rng.integers(2, 2 + ny, stressed), rng.integers(2, 2 + nx, stressed)
        fields[k][at] = q * rng.uniform(0.5, 1.0, stressed)
    sim = fg.DeviceSim(p)
    for k, a in fields.items():
        sim.a[k].copy_(torch.from_numpy(a.reshape(-1)))
        np.asarray(st[k]).reshape(-1)[: a.size] = a.reshape(-1)
    sim.mesh.dt_h = hm.mesh.dt_h = 1e299  # (the rule's growth limit is out of the way)
    sim.initial_timestep()
    O.initial_timestep(hm, st)
    assert hm.mesh.dt_h < 1e290
    assert (sim.mesh.dt, sim.mesh.dt_h) == (hm.mesh.dt, hm.mesh.dt_h)


def nan_candidate(hm, st):
    """Whether a candidate of the step from this state is a NaN: the step's
    stages up to set_timestep on a copy, then sqrt(c_s^2 + 2 Q / rho)."""
    s, L = st.copy(), O.lib()
    m, mp, nx, ny = hm.mesh, ctypes.byref(hm.mesh), hm.nx, hm.ny
    a = {k: O.ptr(s[k]) for k in O.FIELDS}
    L.equation_of_state(nx, ny, a["P"], a["rho"], a["e"])
    L.pressure_acceleration(nx, ny, mp, m.dt, a["rho_u"], a["rho_v"], a["u"], a["v"], a["P"],
                            a["rho"], m.edgedx, m.edgedy, m.celldx, m.celldy)
    L.artificial_viscosity(nx, ny, mp, m.dt, a["Qxx"], a["Qyy"], a["u"], a["v"], a["rho_u"],
                           a["rho_v"], a["rho"], m.edgedx, m.edgedy, m.celldx, m.celldy)
    L.shock_heating_and_work(nx, ny, mp, m.dt_h, a["e"], a["P"], a["u"], a["v"], a["rho"],
                             a["Qxx"], a["Qyy"], m.celldx, m.celldy)
    r, e = s.interior("rho"), s.interior("e")
    with np.errstate(all="ignore"):
        sound = np.sqrt(GAM * (GAM - 1.0) * e)
        return any(np.isnan(np.sqrt(sound * sound + 2.0 * s.interior(k) / r)).any()
                   for k in ("Qxx", "Qyy"))


@pytest.mark.parametrize("width", [1.0, 3e-7, 1e9])
@pytest.mark.parametrize("rho,e", [(1.0, 1.0), (1e-25, 1e-15), (1e-29, 1e-10), (1e-28, 1e-20),
                                   (1e-160, 1e-160), (1e250, 1e-3), (1.0, 1e280), (3e-39, 7e35)])
def test_timesteps_of_whole_steps(fg, rho, e, width):
    from flow_gb300 import problems
    nx, ny = 45, 32
    p = problems.Problem(nx, ny, width=width, height=width, max_dt=1e300).boxes(
        [(0.125 * rho, 2.0 * e, 0.0, 0.0, width, width),
         (rho, 2.5 * e, 0.3 * width, 0.2 * width, 0.4 * width, 0.5 * width)]).with_cfl_dt()
    sim = fg.DeviceSim(p)
    hm = O.HostMesh(nx, ny, width=width, height=width, dt=p.dt_param, max_dt=1e300)
    st = O.HostState(hm)
    O.fill_fields(hm, st, p.interior(p.rho), p.interior(p.e))
    sim.initial_timestep()
    O.initial_timestep(hm, st)
    for tt in range(8):
        assert (sim.mesh.dt, sim.mesh.dt_h) == (hm.mesh.dt, hm.mesh.dt_h), tt
        last = nan_candidate(hm, st)
        sim.step()
        O.step(hm, st, tt)
        if last:
            break
        for k in ("rho", "e", "u", "v"):
            assert np.array_equal(sim.interior(k), st.interior(k), equal_nan=True), (tt, k)
    else:
        assert (sim.mesh.dt, sim.mesh.dt_h) == (hm.mesh.dt, hm.mesh.dt_h)
