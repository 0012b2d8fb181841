"""Which kernels a plan that chooses them itself runs, on both sides of each line of the rule."""
import pytest

pytestmark = pytest.mark.gpu

RUN_TIME = 0
# precision, nx, ny, (row, column) values per thread: 0 the run-time kernel, else the
# register-resident one's
CASES = [
    # odd-factor columns by their number
    ("fp32", 8192, 192, (32, RUN_TIME)), ("fp32", 4096, 384, (32, RUN_TIME)), ("fp32", 8192, 384, (32, 24)),
    ("fp32", 1024, 640, (32, RUN_TIME)), ("fp32", 1280, 640, (20, 20)), ("fp32", 2048, 896, (32, RUN_TIME)),
    ("fp32", 4096, 896, (32, 28)), ("fp32", 512, 768, (32, 24)),
    ("fp64", 1024, 384, (16, RUN_TIME)), ("fp64", 1280, 384, (20, 12)), ("fp64", 1024, 640, (16, RUN_TIME)),
    ("fp64", 1280, 640, (20, 20)), ("fp64", 512, 1280, (16, RUN_TIME)), ("fp64", 1024, 1280, (16, 20)),
    ("fp64", 4096, 896, (16, RUN_TIME)), ("fp64", 512, 3584, (16, 28)),
    # FP64 rows with the factor 7 by their number
    ("fp64", 448, 2048, (RUN_TIME, 16)), ("fp64", 448, 4096, (28, 16)), ("fp64", 896, 2048, (RUN_TIME, 16)),
    ("fp64", 896, 4096, (28, 16)), ("fp64", 1792, 1024, (RUN_TIME, 16)), ("fp64", 3584, 256, (RUN_TIME, 8)),
    ("fp64", 3584, 512, (28, 8)), ("fp64", 7168, 64, (RUN_TIME, 8)), ("fp64", 7168, 256, (28, 8)),
    # a side without a register-resident kernel beside a power-of-two one
    ("fp64", 512, 220, (16, RUN_TIME)), ("fp32", 512, 88, (32, RUN_TIME)), ("fp64", 198, 256, (RUN_TIME, 8)),
    ("fp32", 198, 128, (RUN_TIME, RUN_TIME)),
]


@pytest.mark.parametrize("precision,nx,ny,want", CASES)
def test_plan_mixes_kernels_by_pass(precision, nx, ny, want):
    """The passes' kernels; power-of-two rows are the paired kernel's."""
    from pfc_models_b200 import stdpfc
    prm = stdpfc.BuildStdPFCModelParameters(Gamma=1.0, beta=1.0, q0=1.0, epsilon=-0.25, g=0.0, dt=0.5)
    sim = stdpfc.BuildB200_Simulation(prm, stdpfc.Build2DGeometry(nx, ny, 0.78 * nx, 0.78 * ny), precision=precision)
    v = sim.plan.variant()
    sim.plan.close()
    assert (v["ee_row"], v["ee_col"]) == want
    assert bool(v["row_tile"] & 16) == (nx & (nx - 1) == 0)
