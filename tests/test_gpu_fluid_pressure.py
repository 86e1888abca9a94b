"""The fluid's pressure bulk (J^-gamma - 1) on the device, against float64, near J = 1
(where the power minus one would cancel) and under strong compression (where an
exponent rounded to 32 bits would lose several digits of the power).

Particles at rest on grid nodes, too far apart to share one, with F = diag(J, 1, 1):
weights, offsets, volume and the factors of dt and cell width are powers of two or
short binary fractions and det F is J itself, so the momentum of the next node along x is
9/128 V0 h bulk (J^-gamma - 1) J up to the rounding of the pressure and of two
products."""

import numpy as np
import pytest

from tessera_b200._abi import MAT_FLUID, density_particles, make_params
from tessera_b200.session import Session

pytestmark = pytest.mark.gpu

H, DT, BULK = 2.0**-6, 2.0**-14, 2.0**13
PRODUCTS = 2 * 2.0**-24
# the errors that the CUDA math functions document (ulps of at most 2^-23), times how
# much of them the difference from one keeps
NEAR = PRODUCTS + 2 * 2.0**-23 + 1.2 * 2.0**-24 + 1.2 * 2.0**-23  # expm1 1 ulp (and its product), e rounded, log 1 ulp
STRONG = PRODUCTS + 2.0**-24 + 4 * 2.0**-23 * 1.02  # power 4 ulp, below 1/50 of it one is


@pytest.mark.parametrize("gamma", [4.0, 7.0, 11.0])
@pytest.mark.parametrize("lo,hi,bound", [(0.97, 0.9999, NEAR), (0.04, 0.35, STRONG)])
def test_pressure_of_a_compressed_fluid(gamma, lo, hi, bound):
    at = np.arange(8, 56, 6)
    cells = np.stack(np.meshgrid(at, at, at, indexing="ij"), -1).reshape(-1, 3)
    n = len(cells)
    p = density_particles(cells * H, H / 4, 1000.0, MAT_FLUID, (BULK, gamma, 0.0, 0.0))
    J = np.linspace(lo, hi, n).astype(np.float32)
    p.deformation[:] = np.eye(3).reshape(9)
    p.deformation[:, 0] = J
    params = make_params(H, max_substep=1e-3, gravity=(0.0, 0.0, 0.0), bounds=((0, 0, 0), (1, 1, 1)))
    nodes, values = Session(params, p, DT).debug_p2g()
    momentum = {tuple(c): v[1] for c, v in zip(nodes, values)}
    got = np.array([momentum[(x + 1, y, z)] for x, y, z in cells], dtype=np.float64)
    J = J.astype(np.float64)
    want = 9 / 128 * (H / 2) ** 3 * H * BULK * np.expm1(-gamma * np.log(J)) * J
    worst = np.abs(got / want - 1).max()
    assert worst < bound, (worst, bound)
