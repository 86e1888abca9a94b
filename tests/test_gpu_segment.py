"""Whole-segment launches (small scenes: one cooperative launch per segment) and
the fluid's one-component F between the first and last G2P of a segment, against
the f64 oracle with the resident tolerances of the reference (gpu.rs:3699-3703;
twice the 8-substep bounds for the longer runs, as in the launch-shape tests)."""

import numpy as np
import pytest

from oracle import oracle as O
from tessera_b200 import _native, scenes
from tessera_b200._abi import MAT_ELASTIC, MAT_FLUID, ParticleArrays, density_particles, make_params
from tessera_b200.batch import Batch
from tessera_b200.session import Session

pytestmark = pytest.mark.gpu
H = 1.0 / 32


def block(count, material, prm, seed=1):
    """`count` particles of a jittered lattice above the floor, moving down, with a non-spherical F."""
    rng = np.random.default_rng(seed)
    pos = scenes.lattice((0.3, 0.3, 2 * H), (0.3 + 6 * H, 0.3 + 6 * H, 8 * H), H / 2, rng, 0.5)
    assert len(pos) >= count
    p = density_particles(pos[:count], H / 4, 1000.0, material, prm, velocity=(0.1, -0.05, -0.4))
    F = np.eye(3) + rng.uniform(-0.02, 0.02, (count, 3, 3))
    p.deformation[:] = F.transpose(0, 2, 1).reshape(count, 9)
    return p


def assert_whole(sim):
    """Every segment of the session or batch ran as one launch."""
    L = _native.lib()
    fn = L.tmpm_debug_batch_segments if isinstance(sim, Batch) else L.tmpm_debug_session_segments
    whole, stepwise = _native.segment_launches(fn, sim._h)
    assert whole > 0 and stepwise == 0, (whole, stepwise)


def check(cpu, got, steps):
    e, k = cpu.particles(), 1 if steps <= 8 else 2
    assert np.linalg.norm(e.position - got.position, axis=1).max() < k * 2e-5
    assert np.linalg.norm(e.velocity - got.velocity, axis=1).max() < k * 2e-4
    assert np.linalg.norm(e.deformation - got.deformation, axis=1).max() < k * 2e-4


@pytest.mark.parametrize("shape", [0, 1, 3, 4])
@pytest.mark.parametrize("count", [1, 127, 129, 256, 257, 1500])
def test_segment_tracks_the_oracle_at_chunk_edges(shape, count):
    params = make_params(H, bounds=((0, 0, 0), (1, 1, 1)))
    p = block(count, MAT_ELASTIC, (5e3, 0.3))
    cpu = O.OracleWorld(params, p)
    s = Session(params, p, 1e-4, launch_shape=shape)
    for steps in (1, 2, 9):  # segments of one substep, of two, and one replayed from a graph
        s.step(steps)
        for _ in range(steps):
            cpu.substep_fixed(1e-4)
    check(cpu, s.particles(), 12)
    assert_whole(s)


@pytest.mark.parametrize("steps", [1, 2, 3, 17])
def test_fluid_deformation_survives_segment_ends(steps):
    """A fluid with any F, a fixed particle and an elastic one beside it: every
    component of F is current after each segment, whatever its length, also
    where a re-sort moves the rows between segments."""
    params = make_params(H, bounds=((0, 0, 0), (1, 1, 1)))
    fluid = block(700, MAT_FLUID, (1e4, 7.0, 0.01, 0.25))
    fluid.fixed[3] = 1
    solid = block(100, MAT_ELASTIC, (5e3, 0.3), seed=2)
    solid.position[:, 0] += 0.3
    p = ParticleArrays.concat([fluid, solid])
    cpu = O.OracleWorld(params, p)
    s = Session(params, p, 5e-5, resort_interval=3)
    for _ in range(2):
        s.step(steps)
        for _ in range(steps):
            cpu.substep_fixed(5e-5)
        got = s.particles()
    check(cpu, got, 2 * steps)
    assert_whole(s)
    assert np.allclose(got.deformation[3], fluid.deformation[3], atol=1e-7)  # a fixed particle keeps its F


def test_fluid_deformation_of_uneven_batch_scenes():
    """Scenes of one batch end at different substeps: each writes all of F at its own last one."""
    made = [(make_params(H, bounds=((0, 0, 0), (1, 1, 1))), block(n, MAT_FLUID, (1e4, 7.0, 0.01, 0.25), seed=n))
            for n in (300, 700, 40)]
    batch = Batch()
    ids = [batch.add_scene(params, p, 5e-5) for params, p in made]
    steps = dict(zip(ids, (1, 6, 3)))
    batch.run(steps)
    batch.run(steps)
    for sid, (params, p) in zip(ids, made):
        cpu = O.OracleWorld(params, p)
        for _ in range(2 * steps[sid]):
            cpu.substep_fixed(5e-5)
        check(cpu, batch.particles(sid), 2 * steps[sid])
    assert_whole(batch)


def test_sessions_of_several_threads_share_the_gpu():
    """Whole-segment launches of several sessions, each on its own stream from its
    own thread, with more particles between them than the GPU holds at once: every
    session gets the result it gets alone."""
    import threading

    made = [scenes.elastic_block(seed=k, lo=(0.3, 0.3, 0.3), hi=(0.3 + s, 0.3 + s, 0.3 + s)) for k, s in
            ((1, 0.3), (2, 0.28), (3, 0.1))]

    def frames(sc, out, k):
        s = Session(sc.params, sc.particles, sc.dt, launch_shape=0)
        for _ in range(12):
            s.submit_steps(16)
        s.synchronize()
        out[k] = s.particles()
        sessions.append(s)

    alone, together, sessions = [None] * 3, [None] * 3, []
    for k, sc in enumerate(made):
        frames(sc, alone, k)
    threads = [threading.Thread(target=frames, args=(sc, together, k)) for k, sc in enumerate(made)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s in sessions:
        assert_whole(s)
    for a, b in zip(alone, together):
        # 192 substeps apart only by the order of the f32 node sums
        assert np.abs(a.position - b.position).max() < 4e-5
        assert np.abs(a.velocity - b.velocity).max() < 4e-4 * max(1.0, np.abs(a.velocity).max())
