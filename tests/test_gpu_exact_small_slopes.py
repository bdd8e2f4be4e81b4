"""Limited slopes of the bit-exact mode at the ends of the exponent range: the
reference scales each difference (0.5 / h, 2 / h) before it selects one, so
where half a difference is not a number of its own (a subnormal one), or twice
it or 2 / h overflows, the selection has to be made on the scaled products.
Every advection stage's outputs against the oracle, bit for bit, on velocities,
energies and densities whose neighbours differ by a few units of the last
subnormal place, by about the smallest normal number, and by about the largest.
"""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

OUT = ("F_x", "F_y", "uF_x", "uF_y", "vF_x", "vF_y", "rho", "e", "u", "v", "rho_u", "rho_v")


def random_values(rng, kind, n):
    if kind == "last_place":
        return rng.integers(-9, 10, n) * 2.0 ** -1074
    if kind == "smallest_normal":
        return rng.integers(-99, 100, n) * 2.0 ** -1028 + rng.integers(-1, 2, n) * 2.0 ** -1074
    if kind == "largest":
        return rng.integers(-3, 4, n) * 2.0 ** 1021
    if kind == "mixed":
        return rng.uniform(-1, 1, n) * 2.0 ** rng.integers(-1074, -990, n).astype(float)
    return rng.uniform(-1, 1, n)


def spacings(rng, n, h):
    """Cell widths and edge spacings of an irregular mesh."""
    return h * rng.uniform(0.5, 2.0, n + 1), h * rng.uniform(0.5, 2.0, n + 1)


@pytest.mark.parametrize("tt", [0, 1])
@pytest.mark.parametrize("width", [1.0, 2.0 ** -900, 2.0 ** 1010])
@pytest.mark.parametrize("vel,energy", [
    ("ordinary", "last_place"), ("ordinary", "smallest_normal"), ("ordinary", "mixed"),
    ("ordinary", "largest"), ("last_place", "ordinary"), ("smallest_normal", "ordinary"),
    ("mixed", "ordinary"), ("largest", "ordinary")])
def test_advection_stages_bit_exact(vel, energy, width, tt):
    import flow_gb300 as fg
    import torch
    from flow_gb300 import problems
    fg.set_mode(fg.MODE_EXACT)
    try:
        gnx, gny = 37, 29
        sim = fg.DeviceSim(problems.Problem(gnx, gny, width=width, height=width).fields(
            np.ones((gny, gnx)), np.ones((gny, gnx))))
        hm = O.HostMesh(gnx, gny, width=width, height=width)
        st = O.HostState(hm)
        rng = np.random.default_rng(tt + len(vel) + 16 * len(energy))
        for axis, n in (("x", hm.nx), ("y", hm.ny)):
            for k, a in zip(("celld" + axis, "edged" + axis), spacings(rng, n, width / 37)):
                getattr(hm, k)[:] = a
                sim.mesh_arrays[k].copy_(torch.from_numpy(a))

        def fill(k, a):
            st[k][:] = a
            sim.a[k].copy_(torch.from_numpy(a))

        for k in O.FIELDS:
            if k == "reduce":
                continue
            n = st[k].size
            fill(k, rng.uniform(0.5, 2.0, n) if k in ("rho", "rho_old") else
                 random_values(rng, energy, n) if k == "e" else
                 random_values(rng, vel, n) if k in ("u", "v") else rng.uniform(-1.0, 1.0, n))
        nx, ny = hm.nx, hm.ny
        dt, dt_h = 0.012 * width, 0.01 * width

        def mass_and_energy(X, a, mp, m):
            X.advect_mass_and_energy(nx, ny, mp, tt, dt, dt_h, a["rho"], a["e"], a["rho_old"],
                                     a["F_x"], a["F_y"], a["uF_x"], a["uF_y"], a["u"], a["v"],
                                     m.edgedx, m.edgedy, m.celldx, m.celldy)

        def momentum(X, a, mp, m):
            X.advect_momentum(nx, ny, tt, mp, dt_h, dt, a["u"], a["v"], a["uF_x"], a["uF_y"],
                              a["vF_x"], a["vF_y"], a["rho_u"], a["rho_v"], a["rho"], a["F_x"],
                              a["F_y"], m.edgedx, m.edgedy, m.celldx, m.celldy)

        for fn in (mass_and_energy, momentum):
            if fn is momentum:  # (ordinary mass fluxes, whatever the sweeps made of theirs)
                for k in ("F_x", "F_y", "rho"):
                    fill(k, rng.uniform(0.5, 2.0, st[k].size))
            fn(fg.lib(), {k: fg.dptr(sim.a[k]) for k in O.FIELDS}, ctypes.byref(sim.mesh), sim.mesh)
            fg.check()
            fn(O.lib("port"), {k: O.ptr(st[k]) for k in O.FIELDS}, ctypes.byref(hm.mesh), hm.mesh)
            for k in OUT:
                assert np.array_equal(sim.host(k), st[k], equal_nan=True), (fn.__name__, k)
    finally:
        fg.set_mode(fg.MODE_FUSED)
