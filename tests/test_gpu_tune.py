"""The autotuner and the launch shapes it chooses between.

Every tile shape and block size of the solver iteration, and every block size of block matching,
must give the same bytes as the oracle (each element keeps the reference's operation order
whatever the tiling); the tuned table must round-trip through its JSON cache.
"""
import json

import numpy as np
import pytest

import oracle_lib as O
import twixtor_b200 as tw
from twixtor_b200 import synth

pytestmark = pytest.mark.gpu

SHAPES = [(0, 256), (0, 512), (1, 256), (1, 512), (2, 512), (2, 256)]


@pytest.fixture(scope="module")
def dev():
    tw.build()
    d = tw.Device(0)
    yield d
    d.close()


def _pair(w, h, fmt, seed):
    depth = {0: 8, 1: 16, 2: 32}[fmt]
    frames = synth.moving_clip(w, h, 2, depth=depth, seed=seed, square=48, square_velocity=(3.0, 2.0))
    n = w * h * 4
    return O.from_frame(frames[:n], w, h, fmt), O.from_frame(frames[n:], w, h, fmt)


@pytest.mark.parametrize("tile,threads", SHAPES)
@pytest.mark.parametrize("size", [(481, 271), (160, 96), (1920, 1080)])
def test_every_iteration_shape_is_bit_exact(dev, tile, threads, size):
    w, h = size
    if size == (1920, 1080) and (tile, threads) not in [(1, 512), (2, 512)]:
        pytest.skip("1080p: the shapes the tuner picks there")
    a, b = _pair(w, h, 0, seed=w + h)
    s = tw.FlowSettings()
    _, _, levels = tw.flow_geometry(s, w, h)
    for lw, lh in levels:
        dev.tuning_set(lw, lh, tile, threads, 256, 256)
    try:
        fab, fba, _ = dev.solve_pair(a, b, w, h, 0, s)
    finally:
        dev.tuning_clear()
    wab, wba, _ = O.solve_pair(a, b, w, h, 0)
    assert fab.tobytes() == wab.tobytes() and fba.tobytes() == wba.tobytes()


@pytest.mark.parametrize("rows,cols", [(128, 512), (512, 128), (1024, 64), (32, 1024)])
def test_every_block_matching_block_size_is_bit_exact(dev, rows, cols):
    w, h = 481, 271
    a, b = _pair(w, h, 1, seed=7)
    s = tw.FlowSettings()
    _, _, levels = tw.flow_geometry(s, w, h)
    for lw, lh in levels:
        dev.tuning_set(lw, lh, 0, 256, rows, cols)
    try:
        fab, fba, _ = dev.solve_pair(a, b, w, h, 1, s)
    finally:
        dev.tuning_clear()
    wab, wba, _ = O.solve_pair(a, b, w, h, 1)
    assert fab.tobytes() == wab.tobytes() and fba.tobytes() == wba.tobytes()


def test_autotune_table_round_trips_and_keeps_the_bytes(dev, tmp_path):
    path = str(tmp_path / "tune.json")
    s = tw.FlowSettings()
    n = dev.autotune(s, 1920, 1080, path=path)
    _, _, levels = tw.flow_geometry(s, 1920, 1080)
    assert n == len(levels)
    table = json.load(open(path))
    assert set(table["levels"]) == {f"{lw}x{lh}" for lw, lh in levels}
    with tw.Device(0) as other:
        assert other.autotune(s, 1920, 1080, path=path) == 0  # everything came from the cache
        assert json.loads(other.tuning_table()) == table
    # a clip rendered with the tuned shapes is the oracle's
    w, h, nf = 160, 96, 6
    dev.autotune(s, w, h)
    frames = synth.moving_clip(w, h, nf, depth=8, seed=3)
    tp = tw.TimeParams(speed_percent=50.0)
    sels = [tw.select(tp, k, w, h) for k in range(8)]
    got = dev.retime_clip(tw.RetimeSettings(), frames, nf, sels, w, h, 0)
    want = O.retime_clip(frames, nf, w, h, 0, O.retime_params(speed=50.0), 8)
    dev.tuning_clear()
    assert got.tobytes() == want.tobytes()


def test_tuning_entries_are_checked(dev):
    for bad in [(-1, 256, 256, 256), (3, 256, 256, 256), (0, 1024, 256, 256), (0, 100, 256, 256), (0, 256, 2048, 256)]:
        with pytest.raises(tw.BadParam):
            dev.tuning_set(64, 48, *bad)


@pytest.mark.parametrize("tile", ["16x16", "32x64", "32x32", "64x32", "64x64"])
@pytest.mark.parametrize("threads", [256, 512])
@pytest.mark.parametrize("size", [(15, 17), (31, 63), (32, 64), (33, 65), (161, 131)])
@pytest.mark.parametrize("points", [None, (-1.0, -1.0)])
@pytest.mark.parametrize("above_first", [False, True])
def test_every_shape_of_a_table_at_the_ends_of_its_tiles(dev, tmp_path, tile, threads, size, points, above_first):
    """Levels a pixel smaller and larger than one or several tiles with each shape a saved table can hold (the
    defaults choose 32 x 64 only for levels of more than 148 tiles of 32 x 32). The points put vectors of
    exactly -1.0, the sentinel of the border rule, near the corners."""
    w, h = size
    rng = np.random.RandomState(w * 3 + h)
    x = np.kron(rng.randint(0, 256, ((h + 2) // 3, (w + 2) // 3, 4)), np.ones((3, 3, 1)))[:h, :w].astype(np.uint8)
    y = np.roll(x, 1, axis=1)
    y[:, 0] = rng.randint(0, 256, (h, 4))
    x, y = np.ascontiguousarray(x).reshape(-1), np.ascontiguousarray(y).reshape(-1)
    pairs = None
    if points:
        at = np.array([[1.0, 1.0], [w - 1.0, 1.0], [1.0, h - 1.0], [w / 2, h / 2]], np.float32)
        pairs = np.concatenate([at, at + np.float32(points)], 1).astype(np.float32)
    want, xl, yl, _, _, ud, uw = O.solve_pyramids_with(x, y, w, h, 0, None, None, pairs, quality=5, above_first=above_first)
    s = tw.FlowSettings(quality=5, taps_above_first=above_first)
    levels = tw.flow_geometry(s, w, h)[2]
    path = tmp_path / "tune.json"
    try:
        for lw, lh in levels:
            dev.tuning_set(lw, lh, 0, threads, 256, 256)
        path.write_text(dev.tuning_table().replace('"32x32"', f'"{tile}"'))
        dev.tuning_clear()
        assert dev.autotune(s, w, h, path=str(path)) == 0
        assert [v["iter_tile"] for v in json.loads(dev.tuning_table())["levels"].values()] == [tile] * len(levels)
        got, _ = dev.solve_pyramids(s, w, h, xl, yl, None, None, ud, uw)
    finally:
        dev.tuning_clear()
    assert got.tobytes() == want.tobytes()
