"""CPU tests of what the library asks of the device: its host code runs against a
fake CUDA runtime (tests/native/fake_cudart.cpp: device memory on the heap, no
kernel runs, every operation logged with its stream), linked with the library's
own objects, in a process of its own."""

import os
import shutil
import subprocess
import sys

import pytest

from tessera_b200 import _native

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
OBJECTS = os.path.join(ROOT, "_build", "tmpm")
SOURCES = os.path.join(ROOT, "tessera_b200", "csrc")

PRELUDE = """
import ctypes as C, sys
import numpy as np
sys.path.insert(0, {root!r})
from tessera_b200 import _native, scenes
_native.LIB_PATH = {lib!r}
L = _native.lib()
L.fake_log.restype = C.c_char_p
L.fake_memory.argtypes = [C.c_void_p, C.c_size_t, C.c_int]

def log():
    lines = L.fake_log().decode().splitlines()
    L.fake_clear_log()
    return lines

def count(lines, *words):
    return sum(all(w in line for w in words) for line in lines)
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    if shutil.which("nvcc") is None or shutil.which("g++") is None:
        pytest.skip("nvcc or g++ not available")
    _native.build()  # the objects, where they are not up to date
    lib = str(tmp_path_factory.mktemp("fake") / "libtmpm_fake.so")
    include = os.path.join(os.path.dirname(os.path.dirname(shutil.which("nvcc"))), "include")
    objects = sorted(os.path.join(OBJECTS, f[:-3] + ".o") for f in os.listdir(SOURCES) if f.endswith(".cu"))
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", include, "-o", lib,
                    os.path.join(HERE, "native", "fake_cudart.cpp"), *objects, "-lpthread", "-Wl,-z,defs"],
                   check=True, timeout=600)

    def run(body):
        r = subprocess.run([sys.executable, "-c", PRELUDE.format(root=ROOT, lib=lib) + body], capture_output=True,
                           text=True, timeout=300, cwd=ROOT)
        assert r.returncode == 0, r.stdout + r.stderr

    return run


@pytest.mark.parametrize("refuse", [0, 1, 2, 3])
def test_rollout_whose_cooperative_launch_is_refused_runs_kernel_by_kernel(run, refuse):
    """Refused when issued (1; 3: which also ends the capture) or when its graph
    is launched (2), a whole-rollout launch must not be answered with whatever
    the result buffers held: the sweep runs kernel by kernel, then and later."""
    run(f"""
from tessera_b200.adjoint import Rollout
sc = scenes.adjoint_block(cells=2, substeps=4)
sim = Rollout(sc.params, sc.particles, sc.dt, 4, checkpoint_every=3)
L.fake_refuse_cooperative({refuse})
for call in range(2):
    log()
    x, v = sim.forward(sc.particles.velocity, np.full(sc.particles.count, 5e3))
    done = log()
    whole = 0 if {refuse} else 1
    assert count(done, "cooperative", "k_rollout_forward") == whole, done
    assert count(done, "kernel", "k_p2g") == (0 if whole else 4), done
    if not whole:
        assert np.allclose(x, sc.particles.position)  # after an even count, the buffer that began as the initial state (no kernel ran)
    sim.backward(np.ones((sc.particles.count, 3)))
    done = log()
    assert count(done, "cooperative", "k_rollout_backward") == whole, done
    assert count(done, "kernel", "k_p2g_back") == (0 if whole else 4), done
""")


@pytest.mark.parametrize("device", [0, 1])
@pytest.mark.parametrize("with_keys", [False, True])
@pytest.mark.parametrize("offset", [0, 2])
def test_binning_writes_only_words_of_its_own_device(run, device, with_keys, offset):
    """The last pass stores to the caller's buffers itself only where a kernel may:
    aligned memory of the current device.  Another device's memory is reached by
    copies, which need no peer access."""
    run(f"""
n = 300
pos = np.random.default_rng(1).uniform(0, 1, (3, n)).astype(np.float32)
own, out = np.zeros(n + 1, np.uint32), np.zeros(n + 1, np.uint32)
L.fake_memory(pos.ctypes.data, pos.nbytes, 0)
L.fake_memory(own.ctypes.data, own.nbytes, 0)
L.fake_memory(out.ctypes.data, out.nbytes, {device})
order, keys = (own.ctypes.data, out.ctypes.data + {offset}) if {with_keys} else (out.ctypes.data + {offset}, None)
assert L.tmpm_sort_by_block_noalloc(pos.ctypes.data, n, n, 1 / 64, order, keys, None) == 0, L.tmpm_last_error()
done = log()
assert count(done, "kernel", "k_small_pass") == 3
direct = {device} == 0 and {offset} == 0
assert count(done, "copy kind=3", "dst=%#x " % order) == (0 if direct else 1), done
if keys:
    assert count(done, "copy kind=3", "dst=%#x " % keys) == (0 if direct else 1), done
""")


# the words after each grid table's block count (two tables): cleared, then one set
# to ~0, on the stream of the segment that reads them, before it
TABLE_WORDS = """
    lines = log()
    first = next(i for i, line in enumerate(lines) if "k_segment" in line)
    stream = lines[first].split("stream=")[1]
    assert stream != "(nil)"
    cleared = [line.split("dst=")[1].split()[0] for line in lines[:first]
               if line.startswith("set") and "bytes=16 " in line and line.endswith("stream=" + stream)]
    marked = ["set dst=%#x bytes=4 stream=%s" % (int(p, 16) + 4, stream) for p in cleared]
    assert sum(m in lines[:first] for m in marked) == 2, lines[:first]
"""


def test_table_words_are_set_on_the_stream_that_reads_them(run):
    run("""
def check():
""" + TABLE_WORDS + """
from tessera_b200.batch import Batch
from tessera_b200.session import Session
sc = scenes.batch_scene(3, cells=4)
s = Session(sc.params, sc.particles, sc.dt)
s.submit_steps(3)
check()
b = Batch()
b.run({b.add_scene(sc.params, sc.particles, sc.dt): 3})
check()
""")


def test_uploads_are_ordered_before_the_kernels_that_read_them(run):
    """No host-to-device copy on the legacy stream: from pageable memory it may
    return before its data has arrived, and non-blocking streams do not wait for it."""
    run("""
from tessera_b200._abi import Obstacle, TmpmRigidBody, TmpmRigidMapping
from tessera_b200.batch import Batch
from tessera_b200.session import Session
sc = scenes.batch_scene(3, cells=4)
s = Session(sc.params, sc.particles, sc.dt, obstacles=[Obstacle.sphere((0.5, 0.5, 0.9), 0.05)])
s.rigid_attach([TmpmRigidBody.make((0.5, 0.5, 0.9), 2.0, inverse_inertia=(5.0, 5.0, 5.0))], [TmpmRigidMapping.make(0)])
s.rigid_step(2)
b = Batch()
b.run({b.add_scene(sc.params, sc.particles, sc.dt): 3})
from tessera_b200.adjoint import Rollout
sc = scenes.adjoint_block(cells=2, substeps=4)
Rollout(sc.params, sc.particles, sc.dt, 4).forward()
lines = log()
assert count(lines, "copy kind=1") > 10
assert count(lines, "copy kind=1", "stream=(nil)") == 0, [l for l in lines if "(nil)" in l]
""")


@pytest.mark.parametrize("refuse", [0, 1, 2, 3])
def test_segment_whose_cooperative_launch_is_refused_runs_kernel_by_kernel(run, refuse):
    """As for a rollout: captured segments of a session (16 substeps) and launched ones (2), and a batch's."""
    run(f"""
from tessera_b200.batch import Batch
from tessera_b200.session import Session
sc = scenes.batch_scene(3, cells=4)
L.fake_refuse_cooperative({refuse})
s = Session(sc.params, sc.particles, sc.dt, launch_shape=0)
b = Batch(launch_shape=0)
scene = b.add_scene(sc.params, sc.particles, sc.dt)
log()
for steps in (16, 2, 16):
    for call in (lambda: s.step(steps), lambda: b.run({{scene: steps}})):
        call()
        done = log()
        # refused only when a graph is launched, a segment without one still goes whole at first
        if {refuse} == 0:
            assert count(done, "cooperative", "k_segment") == 1, done
            assert count(done, "kernel", "k_grid") == 0, done
        else:
            assert count(done, "cooperative", "k_segment") == 0, done
            assert count(done, "kernel", "k_grid") == steps, done
assert s.substeps() == 34 and b.substeps(scene) == 34
""")


def test_whole_segments_leave_room_for_other_streams(run):
    """A segment that held every SM until its end would keep a read of another scene
    waiting; with 2 x 148 CTAs resident at once, five are left (rounded up from 1/64)."""
    run("""
from tessera_b200._abi import MAT_ELASTIC, density_particles, make_params
from tessera_b200.batch import Batch
from tessera_b200.session import Session
h = 1 / 64
params = make_params(h, bounds=((0, 0, 0), (1, 1, 1)))
pos = scenes.lattice((0.2, 0.2, 0.2), (0.55, 0.55, 0.55), h / 2, np.random.default_rng(0), 0.5)
pos = np.concatenate([pos, pos + 1e-3])
for count, whole in ((291 * 256, 1), (291 * 256 + 1, 0)):
    assert len(pos) >= count
    p = density_particles(pos[:count], h / 4, 1000.0, MAT_ELASTIC, (5e3, 0.3))
    s, b = Session(params, p, 1e-4, launch_shape=0), Batch(launch_shape=0)
    s.submit_steps(2)
    b.submit({b.add_scene(params, p, 1e-4): 2})
    for sim, fn in ((s, L.tmpm_debug_session_segments), (b, L.tmpm_debug_batch_segments)):
        assert _native.segment_launches(fn, sim._h) == (whole, 1 - whole), (count, sim)
""")
