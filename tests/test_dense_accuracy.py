"""Accuracy of the one-CTA step with dense transforms (pfc_dense.cu) against 80-bit values: its
error, pooled over sizes at both ends of its range, is no larger than that of the two-kernel
step's FFT passes on the same fields."""
import math

import numpy as np
import pytest

L = np.longdouble
PI = L("3.14159265358979323846264338327950288")
SIZES = [(28, 24), (14, 24), (6, 30), (20, 36), (48, 20), (30, 22), (36, 40)]
LX, LY = 14.5, 25.1
PRM = {"std": dict(Gamma=1.0, beta=1.0, q0=1.0, epsilon=-0.25, g=0.0, dt=0.5),
       "log": dict(Gamma=1.0, beta=0.5, q0=1.0, epsilon=-0.9, g=-2.0, dt=0.1)}


def _field(model, nx, ny, seed):
    r = np.random.default_rng(1000 * seed + nx * ny)
    x, y = 2 * np.pi * np.arange(nx)[None] / nx, 2 * np.pi * np.arange(ny)[:, None] / ny
    w = np.cos(x) * np.cos(y) + 0.3 * np.cos(2 * y)
    noise = r.standard_normal((ny, nx))
    return 0.55 * (1 + 0.3 * w) * (1 + 1e-3 * noise) if model == "log" else -0.28 + 0.3 * w + 0.01 * noise


def _exact(model, f, steps):
    """The ETD1 step in 80 bits, transforms as matrix products."""
    p = {k: L(v) for k, v in PRM[model].items()}
    ny, nx = f.shape

    def dft(n):
        return np.exp(-2j * PI * (np.outer(np.arange(n), np.arange(n)) % n).astype(L) / L(n)).astype(np.clongdouble)

    def k2(n, length):
        i = np.arange(n)
        return (2 * PI * np.where(i <= (n - 1) // 2, i, i - n).astype(L) / L(length)) ** 2
    fx, fy = dft(nx), dft(ny)
    lap = -(k2(nx, LX)[None] + k2(ny, LY)[:, None])
    z = p["Gamma"] * lap * (p["beta"] * (p["q0"] ** 2 + lap) ** 2 + p["epsilon"]) * p["dt"]
    a1 = np.expm1(z)
    b = np.where(z == 0, L(1), a1 / np.where(z == 0, L(1), z)) * p["dt"] * p["Gamma"] * lap
    n = f.astype(L)
    h, out = fy @ n @ fx, {}
    for s in range(1, max(steps) + 1):
        nl = p["g"] * n * n + n ** 3 + (np.log(n) if model == "log" else 0)
        h = h + a1 * h + b * (fy @ nl @ fx)
        n = ((np.conj(fy) @ h @ np.conj(fx)) / (nx * ny)).real
        out[s] = n
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("model", ["std", "log"])
def test_dense_step_is_as_accurate_as_the_fft_passes(model):
    """Root mean square errors after 1 and 10 steps, as a geometric mean over sizes and fields,
    dense over FFT: at most 1, with 5 % for the 42 samples (their ratios scatter by a fifth)."""
    from pfc_models_b200 import logpfc, stdpfc
    mod = logpfc if model == "log" else stdpfc
    build = mod.BuildLogPFCModelParameters if model == "log" else mod.BuildStdPFCModelParameters
    ratios = []
    for nx, ny in SIZES:
        for seed in range(3):
            f = _field(model, nx, ny, seed)
            exact = _exact(model, f, (1, 10))
            err = {}
            for one_cta in (True, False):
                sim = mod.BuildB200_Simulation(build(**PRM[model]), mod.Build2DGeometry(nx, ny, LX, LY), precision="fp64",
                                               one_cta=one_cta)
                state = sim.State.phi if model == "log" else sim.State.n
                state[...] = f
                assert sim.plan.path() == ("one_cta" if one_cta else "mixed_radix")
                for n, more in ((1, 1), (10, 9)):
                    sim.TimeSteps(more)
                    d = state.get().astype(L) - exact[n]
                    err.setdefault(n, []).append(math.sqrt(float((d * d).mean())))
                sim.plan.close()
            ratios += [math.log(a / b) for a, b in err.values()]
    assert math.exp(np.mean(ratios)) <= 1.05, math.exp(np.mean(ratios))
