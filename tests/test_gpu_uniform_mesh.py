"""The FP64 tiles fold a uniform mesh's spacings into the timestep; any other
mesh takes the general tiles, which read the spacing arrays.  Both against the
oracle: stretched meshes (spacings varying by up to 40 %, x and y apart, no two
axes alike), and meshes that are uniform but for one ghost spacing that no
interior cell reads, where the general tiles must agree with the oracle of the
uniform mesh too.  Tolerances are those of the FP64 fixtures: density and
energy 1e-12 per cell (floor 1e-3 of the field's maximum), the signed fields
the larger of that and twice the difference between the oracle's own two
builds (strict IEEE, and with FMA contraction), which on a smooth field, whose
momenta are sums of small pressure differences, is about 2e-11."""
import numpy as np
import pytest

from oracle import oracle as O
from tolerance import FP64_TOL, cell_rel_err

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "e", "u", "v", "rho_u", "rho_v")


def spacings(p, kind, rng):
    dx, dy = p.width / p.gnx, p.height / p.gny
    out = {}
    for n, h, c, e in ((p.nx, dx, "celldx", "edgedx"), (p.ny, dy, "celldy", "edgedy")):
        if kind == "stretched":
            cell = h * (1.0 + 0.4 * np.sin(np.linspace(0.0, 5.0, n + 1)) * rng.uniform(0.5, 1.0))
            edge = np.concatenate([cell[:1], 0.5 * (cell[1:] + cell[:-1])])
        else:
            cell, edge = np.full(n + 1, h), np.full(n + 1, h)
            cell[0] = 2.0 * h
        out[c], out[e] = cell, edge
    return out


def oracle_run(p, arrays, build):
    hm = O.HostMesh(p.gnx, p.gny, dt=p.dt_param)
    for k, a in arrays.items():
        getattr(hm, k)[:] = a
    st = O.HostState(hm)
    O.fill_fields(hm, st, p.interior(p.rho), p.interior(p.e))
    O.initial_timestep(hm, st, build)
    O.run(hm, st, 60, build)
    return hm, st


@pytest.mark.parametrize("kind", ["stretched", "one_ghost"])
@pytest.mark.parametrize("field,nx,ny", [("smooth", 96, 96), ("box", 130, 70), ("box", 64, 128)])
def test_general_tiles_match_oracle(kind, field, nx, ny):
    import flow_gb300 as fg
    import torch
    from flow_gb300 import problems
    fg.set_mode(fg.MODE_FUSED)
    rng = np.random.default_rng(7)
    if field == "smooth":
        p = problems.smooth_random(nx, rng)
    else:
        p = problems.Problem(nx, ny).boxes([(0.125, 2.0, 0.0, 0.0, 1.0, 1.0),
                                            (1.0, 2.5, 0.3, 0.2, 0.4, 0.5)]).with_cfl_dt()
    p.dt_param *= 0.5
    arrays = spacings(p, kind, rng)
    sim = fg.DeviceSim(p)
    for k, a in arrays.items():
        sim.mesh_arrays[k].copy_(torch.from_numpy(a))
    sim.initial_timestep()
    sim.run(60)
    hm, st = oracle_run(p, arrays, "port")
    _, other = oracle_run(p, arrays, "fast")
    assert abs(sim.mesh.dt - hm.mesh.dt) <= FP64_TOL * hm.mesh.dt
    for k in FIELDS:
        tol = FP64_TOL
        if k not in ("rho", "e"):
            tol = max(tol, 2.0 * cell_rel_err(other.interior(k), st.interior(k)))
        err = cell_rel_err(sim.interior(k), st.interior(k))
        assert err <= tol, (k, err, tol)
