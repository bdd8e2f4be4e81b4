"""The bit-exact mode divides with a seeded quotient whose residual proves it,
multiplies by power-of-two spacings as exponent adds, and takes the IEEE
operations where a value nears the ends of the exponent range.  Here its steps
must give the oracle's bits on states from one end of the range to the other
(densities and energies whose products, quotients and squares cross into the
guarded exponents, overflow or become subnormal), on meshes of power-of-two and
other spacings, wide and narrow."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "e", "u", "v", "rho_u", "rho_v", "P", "Qxx", "Qyy", "F_x", "F_y")


def min_over_nans(st):
    """Whether a cell's timestep candidate (from the energy after shock heating,
    which this step's advection has moved on since) may have been a NaN."""
    e = st.interior("e")
    with np.errstate(all="ignore"):
        return not np.all(np.isfinite(e * e)) or e.min() < 0.0


@pytest.mark.parametrize("width", [1.0, 3e-7, 1e9])
@pytest.mark.parametrize("rho,e", [(1.0, 1.0), (1e-270, 1.0), (1e250, 1e-3), (1.0, 1e-280),
                                   (1.0, 1e280), (1e-160, 1e-160), (3e-39, 7e35)])
@pytest.mark.parametrize("nx,ny", [(64, 32), (45, 23)])
def test_exact_steps_over_the_range(rho, e, width, nx, ny):
    import flow_gb300 as fg
    from flow_gb300 import problems
    fg.set_mode(fg.MODE_EXACT)
    try:
        p = problems.Problem(nx, ny, width=width, height=width, max_dt=1e300).boxes(
            [(0.125 * rho, 2.0 * e, 0.0, 0.0, width, width),
             (rho, 2.5 * e, 0.3 * width, 0.2 * width, 0.4 * width, 0.5 * width)]).with_cfl_dt()
        sim = fg.DeviceSim(p)
        hm = O.HostMesh(nx, ny, width=width, height=width, dt=p.dt_param, max_dt=1e300)
        st = O.HostState(hm)
        O.fill_fields(hm, st, p.interior(p.rho), p.interior(p.e))
        sim.initial_timestep()
        O.initial_timestep(hm, st)
        with np.errstate(all="ignore"):
            for tt in range(8):
                sim.step()
                O.step(hm, st, tt)
                for k in FIELDS:
                    a, b = sim.interior(k), st.interior(k)
                    assert np.array_equal(a, b, equal_nan=True), (tt, k)
                got, want = (sim.mesh.dt, sim.mesh.dt_h), (hm.mesh.dt, hm.mesh.dt_h)
                if got != want:
                    # A cell whose energy went negative has a NaN candidate,
                    # and the reference's minimum over NaNs depends on the
                    # order it is taken in; both go on with one timestep.
                    assert min_over_nans(st), (tt, got, want)
                    hm.mesh.dt, hm.mesh.dt_h = got
    finally:
        fg.set_mode(fg.MODE_FUSED)


@pytest.mark.parametrize("stress", ["none", "some", "all", "one_axis"])
@pytest.mark.parametrize("nx,ny", [(31, 5), (700, 640), (1024, 512)])
def test_timestep_minimum_by_ranks(stress, nx, ny):
    """The CFL minimum evaluates only the cells that FP32 ranks leave in
    question; the mesh sizes give a thread no cell, one, and several."""
    import torch

    import flow_gb300 as fg
    from flow_gb300 import problems
    p = problems.sod(nx, ny)
    rng = np.random.default_rng(nx + len(stress))
    sim = fg.DeviceSim(p)
    hm = O.HostMesh(nx, ny, dt=p.dt_param)
    st = O.HostState(hm)
    shape = (p.ny, p.nx)
    e = np.round(rng.uniform(0.5, 2.5, shape), 2)  # (many equal energies)
    keep = {"none": 0.0, "some": 0.3, "all": 1.0, "one_axis": 0.5}[stress]
    q = [rng.uniform(0.0, 3.0, shape) * (rng.random(shape) < keep) for _ in range(2)]
    if stress == "one_axis":
        q[1][:] = 0.0
    fields = {"rho": rng.uniform(0.1, 2.0, shape), "e": e, "Qxx": q[0], "Qyy": q[1]}
    for k, a in fields.items():
        sim.a[k].copy_(torch.from_numpy(np.ascontiguousarray(a).reshape(-1)))
        np.asarray(st[k]).reshape(-1)[: a.size] = a.reshape(-1)
    sim.initial_timestep()
    O.initial_timestep(hm, st)
    assert (sim.mesh.dt, sim.mesh.dt_h) == (hm.mesh.dt, hm.mesh.dt_h)
