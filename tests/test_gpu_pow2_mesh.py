"""The FP64 tiles whose spacings are all powers of two on a mesh that is not
uniform: the general tiles' numbers, with products and quotients by a spacing
as exponent adds.  On a mesh one tile wide a ghost cell's width, which no
interior cell reads, decides which of the two run (twice the others' is a power
of two, three times is not), so both must give the same bits; meshes of halves
and quarters of different widths, whose tiles take both kinds, are held to the
oracle by the rule of the FP64 fixtures (density and energy 1e-12 per cell, the
signed fields that or twice what the oracle's own two builds differ by)."""
import numpy as np
import pytest

from oracle import oracle as O
from tolerance import FP64_TOL, cell_rel_err

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "e", "u", "v", "rho_u", "rho_v")


def problem(field, nx, ny):
    from flow_gb300 import problems
    if field == "smooth":
        rng = np.random.default_rng(nx)
        p = problems.smooth_random(max(nx, ny), rng)
        rho, e = p.interior(p.rho)[:ny, :nx], p.interior(p.e)[:ny, :nx]
        p = problems.Problem(nx, ny).fields(rho, e).with_cfl_dt()
    else:
        p = problems.Problem(nx, ny).boxes([(0.125, 2.0, 0.0, 0.0, 1.0, 1.0),
                                            (1.0, 2.5, 0.3, 0.2, 0.4, 0.5)]).with_cfl_dt()
    p.dt_param *= 0.5
    return p


def device_run(p, arrays, steps):
    import flow_gb300 as fg
    import torch
    fg.set_mode(fg.MODE_FUSED)
    sim = fg.DeviceSim(p)
    for k, a in arrays.items():
        sim.mesh_arrays[k].copy_(torch.from_numpy(a))
    sim.initial_timestep()
    sim.run(steps)
    return sim


# (The last is large enough for the tiles to test their own spacings; there only
# the first column of tiles holds the odd ghost cell.)
@pytest.mark.parametrize("field", ["smooth", "box"])
@pytest.mark.parametrize("nx,ny", [(5, 3), (64, 32), (100, 77), (124, 200), (2048, 1024)])
def test_same_bits_as_general_tiles(field, nx, ny):
    p = problem(field, nx, ny)
    got = []
    for ghost in (2.0, 3.0):
        arrays = {}
        for n, h, c, e in ((p.nx, 2.0 ** -7, "celldx", "edgedx"), (p.ny, 2.0 ** -6, "celldy", "edgedy")):
            arrays[c], arrays[e] = np.full(n + 1, h), np.full(n + 1, h)
        arrays["celldx"][0] *= ghost
        got.append(device_run(p, arrays, 12))
    a, b = got
    assert np.array_equal([a.mesh.dt, a.mesh.dt_h], [b.mesh.dt, b.mesh.dt_h], equal_nan=True)
    for k in FIELDS:
        assert np.array_equal(a.interior(k), b.interior(k), equal_nan=True), k


@pytest.mark.parametrize("field", ["smooth", "box"])
@pytest.mark.parametrize("nx,ny", [(300, 150), (512, 64)])
def test_graded_meshes_match_oracle(field, nx, ny):
    p = problem(field, nx, ny)
    arrays = {}
    for n, c, e in ((p.nx, "celldx", "edgedx"), (p.ny, "celldy", "edgedy")):
        cell = np.full(n + 1, 2.0 ** -9)
        cell[n // 2:] *= 2.0
        cell[3 * n // 4:] *= 2.0
        arrays[c], arrays[e] = cell, np.concatenate([cell[:1], 0.5 * (cell[1:] + cell[:-1])])
    sim = device_run(p, arrays, 40)
    runs = []
    for build in ("port", "fast"):
        hm = O.HostMesh(nx, ny, dt=p.dt_param)
        for k, a in arrays.items():
            getattr(hm, k)[:] = a
        st = O.HostState(hm)
        O.fill_fields(hm, st, p.interior(p.rho), p.interior(p.e))
        O.initial_timestep(hm, st, build)
        O.run(hm, st, 40, build)
        runs.append((hm, st))
    (hm, st), (_, other) = runs
    assert abs(sim.mesh.dt - hm.mesh.dt) <= FP64_TOL * hm.mesh.dt
    for k in FIELDS:
        tol = FP64_TOL
        if k not in ("rho", "e"):
            tol = max(tol, 2.0 * cell_rel_err(other.interior(k), st.interior(k)))
        err = cell_rel_err(sim.interior(k), st.interior(k))
        assert err <= tol, (k, err, tol)
