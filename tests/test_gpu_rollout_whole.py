"""Whole-rollout launches of the differentiable rollout: the forward against the
oracle and the gradients of one checkpoint interval against another's, at CTA
edges and where the last segment is shorter than the others.

The checkpoint interval only decides what the adjoint replays, so gradients of
two intervals differ by the f32 summation order of the node sums alone: 1e-7
relative per sum, over 2 x 21 substeps below 1e-5 of the largest component."""

import numpy as np
import pytest

from oracle import oracle as O
from tessera_b200 import _native, scenes
from tessera_b200.adjoint import Rollout

pytestmark = pytest.mark.gpu
SUBSTEPS = 21


def gradients(sc, parts, every):
    sim = Rollout(sc.params, parts, sc.dt, SUBSTEPS, checkpoint_every=every)
    n = parts.count
    E = np.linspace(4e3, 6e3, n)
    out = []
    for _ in range(2):  # the second pass replays the captured launches
        x, v = sim.forward(parts.velocity, E)
        g = 2.0 * (x.mean(0) - np.asarray(sc.info["target"])) / n
        out.append((x, v) + sim.backward(np.tile(g, (n, 1))))
    assert _native.lib().tmpm_debug_rollout_whole(sim._h) == 3  # both sweeps ran as one launch
    sim.close()
    return E, out


@pytest.mark.parametrize("count", [1, 127, 128, 129, 512])
def test_gradients_do_not_depend_on_the_checkpoint_interval(count):
    sc = scenes.adjoint_block(cells=4, substeps=SUBSTEPS)
    parts = sc.particles.select(np.arange(count))
    if count > 8:
        parts.fixed[5] = 1
    E, ref = gradients(sc, parts, SUBSTEPS)
    cpu_parts = parts.copy()
    cpu_parts.material_params[:, 0] = E
    cpu = O.OracleWorld(sc.params, cpu_parts)
    for _ in range(SUBSTEPS):
        cpu.substep_fixed(sc.dt)
    e = cpu.particles()
    assert np.linalg.norm(e.position - ref[0][0], axis=1).max() < 4e-5
    assert np.linalg.norm(e.velocity - ref[0][1], axis=1).max() < 4e-4
    for every in (1, 2, 5, 8, 20):
        _, got = gradients(sc, parts, every)
        for run in got + ref[1:]:
            for a, b in zip(run, ref[0]):
                assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max() + 1e-30
