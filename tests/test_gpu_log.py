"""The FP64 log model's logarithm, read back to the last bit through the public entry points.

A uniform field c = k / 2^17 on power-of-two sides passes the transforms without rounding (sums of
equal values double exactly), c^3 has at most 51 bits, and with g = -c the polynomial part of
N(c) = g c^2 + c^3 + log(c) is exactly zero: nonlin_mu of the stepped state is the logarithm as
the step kernel computes it. CUDA's library function is documented within 1 ulp and measured at
0.552 ulp over four million arguments in (0.05, 2) against 80-bit values; the bound here is 0.6 ulp. The
arguments are those in (0.3, 1) at which a short series with a plain final sum is furthest off
(0.75 ulp and more)."""
import numpy as np
import pytest

from pfc_models_b200 import logpfc

pytestmark = pytest.mark.gpu

ARGS = [92184, 91677, 91981, 82990, 49173, 49839, 48687, 82608, 82623, 50382, 92586, 92441, 92218, 48968, 92023, 81415,
        82406, 49447, 80581, 79903, 80627, 49375, 83006, 48743]


@pytest.mark.parametrize("nx,ny,kernels", [(128, 64, "auto"), (64, 64, "auto"), (64, 32, "generic")])
def test_fp64_logarithm_to_the_last_bit(nx, ny, kernels):
    for k in ARGS:
        c = k / 2.0 ** 17
        prm = logpfc.BuildLogPFCModelParameters(Gamma=1.0, beta=0.5, q0=1.0, epsilon=-0.9, g=-c, dt=0.1)
        sim = logpfc.BuildB200_Simulation(prm, logpfc.Build2DGeometry(nx, ny, nx * 0.8, ny * 0.8), kernels=kernels,
                                          one_cta=False)
        sim.State.phi[...] = np.full((ny, nx), c)
        assert np.array_equal(sim.plan.get_state().cpu().numpy(), np.full((ny, nx), c))
        sim.TimeStep()
        got = sim.State.nonlin_mu.get()
        sim.plan.close()
        want = np.log(np.longdouble(c))
        ulp = np.ldexp(1.0, int(np.frexp(float(want))[1]) - 53)
        assert float(np.max(np.abs(got.astype(np.longdouble) - want))) <= 0.6 * ulp, k
