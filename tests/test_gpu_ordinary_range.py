"""The FP64 step's shared-reciprocal divisions against the oracle at the edges
of their operand range: cells, momenta and pressures on both sides of each
bound (where a face or a cell takes the general code instead), signed zeros,
and gas at rest.  Everything is compared bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (density scale, momentum scale, internal-energy scale)
SCALES = [
    (1.0, 1.0, 1.0),
    (1.0, 0.0, 1.0),                 # at rest: zero momenta of both signs
    (1.0, 2.0 ** -440, 1.0),         # 0.5 m^2 about the bound 2^-900
    (1.0, 2.0 ** -460, 1.0),
    (1.0, 2.0 ** -899, 1.0),         # m about 2^-900
    (1.0, 2.0 ** -1040, 1.0),        # denormal momenta
    (1.0, 1e-120, 1e-200),           # pressures about 2^-600
    (1.0, 1e-150, 1e-275),           # ... and below it
    (2.0 ** 115, 2.0 ** 115, 2.0 ** 115),   # cells about the bound 2^116
    (2.0 ** 120, 2.0 ** 121, 2.0 ** 122),
    (1e-28, 1e-28, 1e-28),           # densities near the 1e-30 guard
    (1e-31, 1e-31, 1e-31),
]


@pytest.mark.parametrize("scales", SCALES)
@pytest.mark.parametrize("bc", ["outflow", "periodic"])
def test_f64_step_at_the_ordinary_range(scales, bc):
    import torch
    import bsn
    import oracle as orc
    sr, sm, se = scales
    nx, ny, nz = 13, 9, 11
    rng = np.random.default_rng(5)
    U = orc.state(nx, ny, nz)
    shape = U.shape[1:]
    U[0] = sr * rng.uniform(0.5, 2.0, shape)
    for q in (1, 2, 3):
        U[q] = sm * rng.uniform(-1.0, 1.0, shape)
    if sm == 0.0:
        U[1:4] = np.where(rng.random((3,) + shape) < 0.5, -0.0, 0.0)
    U[4] = se * rng.uniform(0.5, 2.0, shape) + 0.5 * (U[1] ** 2 + U[2] ** 2 + U[3] ** 2) / U[0]
    # a stretch of cells with momenta across many decades beside ordinary ones
    U[1, 5:9] *= 10.0 ** rng.uniform(-320, 0, shape)[5:9]
    g, dx = 5.0 / 3.0, 0.1
    dt = orc.cfl_dt_3d(U, dx, dx, dx, g, 0.3)
    D = torch.from_numpy(U.copy(order="F")).cuda()
    assert bsn.cfl_dt_3d(D, nx, ny, nz, dx, dx, dx, g, 0.3) == dt
    for _ in range(2):
        orc.euler3d_step(U, dx, dx, dx, dt, g, bc=bc, rho_floor=0.0, P_floor=0.0)
        bsn.euler3d_step(D, nx, ny, nz, dx, dx, dx, dt, g, bc=bc, rho_floor=0.0, P_floor=0.0)
    got = D.cpu().numpy()
    assert np.array_equal(got, U, equal_nan=True)
    fin = np.isfinite(U)
    assert np.array_equal(np.signbit(got[fin]), np.signbit(U[fin]))
