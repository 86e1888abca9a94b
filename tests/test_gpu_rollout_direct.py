"""The direct path of the rollout's adjoint (a CTA that gathers or scatters node
by node, without a shared-memory tile), reached as ordinary programs reach it: a
loss on one tracked particle, which then dominates its CTA's velocity adjoints,
and particles too far apart for their CTA's box to fit the tile.

Checked against central differences of the f64 oracle (1e-3 relative, the bar
of the other adjoint tests), between checkpoint intervals, which decide what the
adjoint replays beside its sweep, and whole against kernel by kernel; these
must change the gradients only by the f32 order of the node sums: 1e-7 relative
per sum, over 2 x SUBSTEPS substeps below 1e-5 of the largest component."""

import numpy as np
import pytest

from oracle import oracle as O
from tessera_b200 import _native, scenes
from tessera_b200._abi import MAT_ELASTIC, density_particles, make_params
from tessera_b200.adjoint import Rollout

pytestmark = pytest.mark.gpu
SUBSTEPS = 12
FD = 1e-3  # step of the differences: absolute for velocities, relative for moduli


def stretched(parts, seed):
    """The particles with a deformation 2 % off the identity, so that the moduli act from the first substep."""
    rng = np.random.default_rng(seed)
    F = np.eye(3) + rng.uniform(-0.02, 0.02, (parts.count, 3, 3))
    parts.deformation[:] = F.transpose(0, 2, 1).reshape(parts.count, 9)
    return parts


def final_positions(params, parts, dt, v0, E):
    p = parts.copy()
    p.velocity[:] = v0
    p.material_params[:, 0] = E
    world = O.OracleWorld(params, p)
    for _ in range(SUBSTEPS):
        world.substep_fixed(dt)
    return world.particles().position


def check_gradients(params, parts, dt, tracked, seed):
    """Gradients of a loss on the particles `tracked`, for several checkpoint intervals."""
    rng = np.random.default_rng(seed)
    n = parts.count
    v0, E = parts.velocity.copy(), np.linspace(4e3, 6e3, n)
    weight = np.zeros((n, 3))
    weight[tracked] = rng.normal(size=(len(tracked), 3))

    ref = None
    for every in (SUBSTEPS, 1, 2, 5):
        sim = Rollout(params, parts, dt, SUBSTEPS, checkpoint_every=every)
        for stepwise in (False, True):
            if stepwise:
                assert _native.lib().tmpm_debug_rollout_whole(sim._h) == 3  # both sweeps were one launch
                _native.lib().tmpm_debug_rollout_stepwise(sim._h)
            for _ in range(2):  # the second pass replays the captured launches
                sim.forward(v0, E)
                got = sim.backward(weight)
                ref = ref or got
                for a, b in zip(got, ref):
                    assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max(), (every, stepwise)
        sim.close()

    gv, gE = ref
    assert np.abs(gE).max() > 0
    for _ in range(3):
        d, e = rng.normal(size=(n, 3)), rng.normal(size=n)
        diff = (final_positions(params, parts, dt, v0 + FD * d, E) - final_positions(params, parts, dt, v0 - FD * d, E))
        fd = float((diff * weight).sum() / (2 * FD))
        assert abs(fd - float((gv * d).sum())) < 1e-3 * max(abs(fd), 0.1 * np.abs(gv).max()), fd
        diff = (final_positions(params, parts, dt, v0, E * (1 + FD * e))
                - final_positions(params, parts, dt, v0, E * (1 - FD * e)))
        fd = float((diff * weight).sum() / (2 * FD))
        assert abs(fd - float((gE * E * e).sum())) < 1e-3 * max(abs(fd), 0.1 * np.abs(gE * E).max()), fd


@pytest.mark.parametrize("count", [129, 512])
def test_loss_on_one_particle(count):
    """Compact CTAs (their boxes fit the tile), one dominant particle, a fixed particle beside it."""
    sc = scenes.adjoint_block(cells=4, substeps=SUBSTEPS)
    parts = stretched(sc.particles.select(np.arange(count)), count)
    parts.fixed[5] = 1
    check_gradients(sc.params, parts, sc.dt, [count // 2], seed=count)


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("loss", ["all", "one"])
def test_scattered_particles(loss, fixed):
    """Touching pairs spread over 26 x 26 cells: no CTA's box fits its tile.  Rows are
    ordered by x first, so the last CTA's (partial, hence in order) second warp
    holds the 32 particles of the third group, all of them fixed or none."""
    h = 1.0 / 32
    rng = np.random.default_rng(3)
    groups = []
    for count, lo, hi in ((64, 0.12, 0.35), (16, 0.45, 0.5), (16, 0.6, 0.65), (16, 0.75, 0.8)):
        first = np.column_stack([rng.uniform(lo, hi, count), rng.uniform(0.1, 0.9, (count, 2))])
        groups.append(np.stack([first, first + rng.uniform(-0.4 * h, 0.4 * h, first.shape)], 1).reshape(-1, 3))
    params = make_params(h, bounds=((0, 0, 0), (1, 1, 1)))
    parts = stretched(density_particles(np.concatenate(groups), h / 4, 1000.0, MAT_ELASTIC, (5e3, 0.3),
                                        velocity=(0.1, 0.2, -0.3)), 4)
    if fixed:
        parts.fixed[160:192] = 1
    tracked = np.arange(parts.count) if loss == "all" else [200]
    check_gradients(params, parts, 1e-4, tracked, seed=5)
