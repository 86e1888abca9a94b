"""The four-kernel sort of up to 2^18 keys (allocation-free binning, re-sorts of
sessions and batches): keys and stable order against the f32 binning restated in
numpy, bit for bit, at the edges of its tiles and at its largest size."""

import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from tessera_b200 import _native, scenes
from tessera_b200._abi import TMPM_OK
from tessera_b200.batch import Batch

pytestmark = pytest.mark.gpu


def keys_of(pos, cell_width):
    """27-bit sort key: Morton code of the 4^3 block (21 bits), then of the cell inside it."""
    inv_h = np.float32(1.0) / np.float32(cell_width)
    cell = np.floor(pos * inv_h - np.float32(0.5)).astype(np.int64)
    block, key = cell >> 2, np.zeros(pos.shape[1], dtype=np.uint32)
    for bit in range(7):
        for a in range(3):
            key |= (((block[a] >> bit) & 1) << (6 + 3 * bit + 2 - a)).astype(np.uint32)
    for bit in range(2):
        for a in range(3):
            key |= (((cell[a] >> bit) & 1) << (3 * bit + 2 - a)).astype(np.uint32)
    return key


@pytest.mark.parametrize("count", [1, 31, 2047, 2048, 2049, 70_001, 262_143, 262_144])
@pytest.mark.parametrize("spread", [0.02, 1.0])
def test_small_sort_is_the_stable_order(count, spread):
    import torch

    rng = np.random.default_rng(count)
    pos = rng.uniform(-0.1 * spread, spread, (3, count)).astype(np.float32)
    h = 1.0 / 96
    dev = torch.from_numpy(pos).cuda()
    out = torch.full((2, count + 2), 7, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    for shift in (0, 1):  # word-aligned outputs at any offset, and a call on used scratch
        st = _native.lib().tmpm_sort_by_block_noalloc(
            C.c_void_p(dev.data_ptr()), count, count, h, C.c_void_p(out[0, shift:].data_ptr()),
            C.c_void_p(out[1, shift:].data_ptr()), C.c_void_p(stream))
        assert st == TMPM_OK, _native.lib().tmpm_last_error()
        got = out.cpu().numpy().view(np.uint32)[:, shift:shift + count]
        keys = keys_of(pos, h)
        order = np.argsort(keys, kind="stable")
        assert np.array_equal(got[0], order) and np.array_equal(got[1], keys[order])
        assert (out.cpu().numpy()[:, shift + count:] == 7).all()


def test_batch_resort_keeps_scenes_apart():
    """30-bit keys (scene, block; three 10-bit passes): a removed scene's rows go, the others track the oracle."""
    made = [scenes.batch_scene(40 + k, cells=4 + k) for k in range(3)]
    b = Batch()
    ids = [b.add_scene(s.params, s.particles, s.dt) for s in made]
    b.run({i: 2 for i in ids})
    b.remove_scene(ids[1])
    keep = [(ids[0], made[0]), (ids[2], made[2])]
    b.run({i: 3 for i, _ in keep})
    for sid, s in keep:
        w = O.OracleWorld(s.params, s.particles)
        for _ in range(5):
            w.substep_fixed(s.dt)
        assert np.linalg.norm(b.particles(sid).position - w.particles().position, axis=1).max() < 2e-5
