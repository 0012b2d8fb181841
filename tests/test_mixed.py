"""The run-time mixed-radix kernels (pfc_mixed.cuh) at the edges of their sequences: sides of a
single pass (the fused middle pass alone), every radix as first, middle and last pass, the
packed column's CTA with one and with several columns, rows that do not fill a tile. The
state, mu, the coarse-grained field and the reductions against the oracle. FP64: the
transforms' rounding is a few ulp a pass, 1e-12 relative L2 after 5 steps leaves three
orders; FP32-mixed: the deviation carries FP32 rounding, 1e-5 of the deviation's norm (about
160 ulp) covers 5 steps of at most 4 passes each way, on top of the FP64 bound (the oracle and
the mean are FP64; the deviation of a grid of a few sites decays below their rounding)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(4, 2), (4, 3), (8, 5), (10, 7), (14, 11), (22, 13), (26, 4), (64, 9), (18, 16), (36, 32), (128, 26),
         (144, 121), (286, 49), (100, 169), (392, 33), (66, 784)]


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("model", ["std", "log"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_runtime_kernels_at_sequence_edges(nx, ny, model, precision):
    from oracle import pfc_oracle as orc
    from pfc_models_b200 import logpfc, stdpfc
    kw = dict(Gamma=1.0, beta=0.5, q0=1.0, epsilon=-0.9, g=-2.0, dt=0.05) if model == "log" else \
        dict(Gamma=1.0, beta=1.0, q0=1.0, epsilon=-0.25, g=0.1, dt=0.3)
    mean = 0.6 if model == "log" else -0.27
    go = orc.build_geometry(nx, ny, nx * 0.9, ny * 0.8)
    f0 = mean + 0.05 * np.random.default_rng(100 * nx + ny).uniform(-1, 1, (ny, nx))
    o = orc.OracleSim(model, orc.Params(**kw), go)
    o.set_field(f0)
    mod = logpfc if model == "log" else stdpfc
    build = logpfc.BuildLogPFCModelParameters if model == "log" else stdpfc.BuildStdPFCModelParameters
    sim = mod.BuildB200_Simulation(build(**kw), mod.Build2DGeometry(nx, ny, nx * 0.9, ny * 0.8), precision=precision,
                                   kernels="generic", one_cta=False)
    assert sim.plan.path() == "mixed_radix"
    (sim.State.phi if model == "log" else sim.State.n)[...] = f0
    for _ in range(4):
        o.step()
    mu, local = o.mu(), o.local_field()
    o.step()
    sim.TimeSteps(5)
    tol = 1e-12 if precision == "fp64" else 1e-5
    norm = np.linalg.norm(o.n)
    dev = np.linalg.norm(o.n - o.n.mean()) + 1e-7 * norm if precision == "fp32" else norm
    got = (sim.State.phi if model == "log" else sim.State.n).get()
    assert np.linalg.norm(got - o.n) <= tol * dev
    # mu's linear part scales the rounding by up to |L_mu| at the grid's highest wavenumber
    lmu = float(np.max(np.abs(o.lin_mu)))
    assert np.linalg.norm(sim.mu.get() - mu) <= tol * (np.linalg.norm(mu) + lmu * dev)
    assert np.linalg.norm(sim.State.local_mu.get() - o._irfft2(o.gauss * o._rfft2(mu), mu.shape)) <= \
        tol * (np.linalg.norm(mu) + lmu * dev)
    got_local = sim.Get_local_phi() if model == "log" else sim.Get_local_n()
    assert np.linalg.norm(got_local - local) <= tol * np.linalg.norm(local)
    F, mean_mu, mean_n = sim.Reduce()
    ftol = 1e-12 if precision == "fp64" else 1e-6
    assert F == pytest.approx(o.free_energy(), rel=ftol, abs=ftol)
    assert mean_mu == pytest.approx(o.mu_per_site(), rel=ftol, abs=ftol)
    assert mean_n == pytest.approx(float(o.n.mean()), rel=1e-12)
    sim.plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,ny", [(4, 2), (8, 30), (16, 75), (32, 392), (26, 33), (990, 5)])
def test_upload_of_narrow_fields(nx, ny, precision):
    """Tiles of up to 32 rows, the last one partly filled: a field comes back as it was uploaded,
    within the rounding of a forward and an inverse transform."""
    from pfc_models_b200 import stdpfc
    prm = stdpfc.BuildStdPFCModelParameters(Gamma=1.0, beta=1.0, q0=1.0, epsilon=-0.25, g=0.0, dt=0.5)
    sim = stdpfc.BuildB200_Simulation(prm, stdpfc.Build2DGeometry(nx, ny, 0.78 * nx, 0.78 * ny), precision=precision)
    f = np.random.default_rng(nx * ny).uniform(-1, 1, (ny, nx))
    sim.State.n[...] = f
    eps = np.finfo(np.float64 if precision == "fp64" else np.float32).eps
    assert np.abs(sim.State.n.get() - f).max() <= 4 * eps * np.log2(nx * ny)
    sim.plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(32, 16), (32, 45), (90, 16)])
@pytest.mark.parametrize("model", ["std", "log"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_sixteen_point_transforms(nx, ny, model, precision):
    """Rows and columns of 16 points (two passes of radix 4) against the oracle, as above."""
    test_runtime_kernels_at_sequence_edges(nx, ny, model, precision)
