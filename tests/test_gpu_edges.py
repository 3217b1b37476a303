"""The device kernels at the sizes and values where their fast paths end, against the oracle, bit for bit:
every integer sample, lerps between the ends of a depth's range, points on and across the image's border."""
import numpy as np
import pytest

import oracle_lib as O
import twixtor_b200 as tw

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    tw.build()
    d = tw.Device(0)
    yield d
    d.close()


def same(a, b):
    return np.asarray(a).view(np.uint8).tobytes() == np.asarray(b).view(np.uint8).tobytes()


def integer_pixels(fmt):
    """Pairs (colour, alpha): all of the 8 bit depth, for 16 bits every alpha with colours around it."""
    if fmt == 0:
        c, a = np.meshgrid(np.arange(256), np.arange(256))
    else:
        a = np.arange(65536).repeat(4).reshape(-1, 4)
        c = np.stack([a[:, 0], a[:, 0] // 2, a[:, 0] * 3 + 1, np.full(65536, 65535)], 1) & 0xffff
    return c.reshape(-1), a.reshape(-1)


@pytest.mark.parametrize("fmt", [0, 1])
def test_every_sample_at_the_image_boundary(dev, fmt):
    c, a = integer_pixels(fmt)
    w = 256
    h = c.size // w
    top = 255 if fmt == 0 else 65535
    wire = np.stack([c, top - c, c ^ 1, a], 1).astype(tw.DTYPES[fmt]).reshape(-1)
    assert same(dev.from_frame(wire, w, h, fmt), O.from_frame(wire, w, h, fmt))
    eng = np.stack([a, c, top - c, c ^ 1], 1).astype(tw.DTYPES[fmt]).reshape(-1)
    assert same(dev.to_frame(eng, w, h, fmt), O.to_frame(eng, w, h, fmt))


@pytest.mark.parametrize("fmt", [0, 1, 2])
@pytest.mark.parametrize("size", [(2, 2), (33, 5), (129, 67)])
@pytest.mark.parametrize("wa,interp", [(0.3, 1), (0.5, 1), (1.5, 1), (0.6, 0)])
def test_warps_between_the_ends_of_the_range(dev, fmt, size, wa, interp):
    """Samples at 0 and at the top of the depth (or random), vectors that reach, touch and cross the border."""
    w, h = size
    rng = np.random.RandomState(w + fmt)
    top = {0: 255, 1: 65535, 2: 1.0}[fmt]
    ends = [(rng.randint(0, 2, w * h * 4) * top).astype(tw.DTYPES[fmt]) for _ in range(2)]
    full = [(rng.random_sample(w * h * 4) * top).astype(tw.DTYPES[fmt]) for _ in range(2)]
    flows = [rng.uniform(-4.0, 4.0, w * h * 2).astype(np.float32) for _ in range(2)]
    for f in flows:
        f[::7] = np.round(f[::7])
        f[::11] = 0.0
    for a, b in (ends, full):
        got = dev.compose_vectors(tw.EngineSettings(), tw.Selection(wa=np.float32(wa), interp=interp), a, b, w, h, fmt,
                                  flows[0], flows[1], (w, h))
        assert same(got, O.compose_vectors(a, b, w, h, fmt, flows[0], flows[1], w, h, np.float32(wa), interp))
