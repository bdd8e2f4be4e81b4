"""The mixed form's flux differences (precision.cuh f32_diff) over the exponent
range: the scheme is linear in the density, so a density scaled by a power of
two gives the scaled density and momenta and the same energy and velocities, bit
for bit, as long as no FP32 intermediate leaves the normal range (the smallest
here, a flux correction of 2^-40 of the density, stays above 2^-110).  With
2^-66 and 2^-56 the differences lie below 2^-67, where the FP64 instruction forms
them; with 1 and 2^40 they are formed from FP32 differences.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(n, shift, steps=4):
    import flow_gb300
    from flow_gb300 import problems
    prob = problems.smooth_random(n, np.random.default_rng(5))
    prob.rho = prob.rho * 2.0 ** shift
    sim = flow_gb300.MixedSim(prob)
    for _ in range(steps):
        sim.step()
    out = {k: np.array(sim.interior(k), dtype=np.float64) for k in ("rho", "e", "u", "v", "rho_u")}
    for k in ("rho", "rho_u"):
        out[k] = out[k] * 2.0 ** -shift
    return out, sim.mesh.dt


@pytest.mark.parametrize("n", [64, 100])
@pytest.mark.parametrize("shift", [-66, -56, 40])
def test_scaled_density_same_bits(n, shift):
    want, dt_want = run(n, 0)
    got, dt_got = run(n, shift)
    assert dt_got == dt_want
    assert float(np.abs(want["u"]).max()) > 0.0
    for k in want:
        assert np.array_equal(got[k], want[k]), k
