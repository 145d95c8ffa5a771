"""The device's Halton digits over the whole index range: every dimension at
indices around the powers of two and at the 32-bit limit, against a numpy
float32 restatement of the permuted radical inverse (integer digits, so the
results must be equal bit for bit)."""
import numpy as np
import pytest

import ymrt_b200 as Y
from ymrt_b200 import scenes

pytestmark = pytest.mark.gpu


def radical_inverse(index: int, base: int, perm: np.ndarray) -> np.float32:
    f = np.float32
    inv, scale, total = f(1) / f(base), f(1), 0
    while index:
        index, digit = divmod(index, base)
        total = (total * base + int(perm[digit])) & 0xFFFFFFFFFFFFFFFF
        scale = f(scale * inv)
    tail = f(f(f(perm[0]) * scale) * inv) / f(f(1) - inv)
    x = f(f(f(np.uint64(total)) * scale) + f(tail))
    return max(f(0.000001), min(x, f(0.999999)))


def test_every_dimension_at_index_limits(ctx, cornell_path, halton_perm):
    scene = Y.Scene(ctx, Y.HostScene(cornell_path, 64, 64), halton_perm)
    # samples whose global indices straddle 2^8, 2^16, 2^31, 2^32 and 2^40
    step = int(scene.halton([0], [0], [1], 0)[0][0]) - int(scene.halton([0], [0], [0], 0)[0][0])
    samples = sorted({0, 1, 2, (1 << 31) - 1} |
                     {max(0, min((1 << b) // step + k, (1 << 31) - 1)) for b in (8, 16, 31, 32, 40) for k in (-1, 0, 1)})
    n = len(samples)
    px, py = np.arange(n) * 7 % 64, np.arange(n) * 13 % 64
    index, _, dims = scene.halton(px, py, samples, 1000)
    assert index.max() > (1 << 32) and index.min() < (1 << 16)
    primes = scenes.first_primes()
    first = np.concatenate([[0], np.cumsum(primes.astype(np.int64))]).astype(np.int64)
    d = [2 + k if k < 998 else 2 + k - 998 for k in range(1000)]
    want = np.array([[radical_inverse(int(i), int(primes[k]), halton_perm[first[k]:first[k + 1]]) for k in d]
                     for i in index], np.float32)
    assert np.array_equal(dims.view(np.uint32), want.view(np.uint32))
    scene.close()


def plain_inverse(index: int, base: int) -> np.float32:
    f = np.float32
    inv, scale, total = f(1) / f(base), f(1), 0
    while index:
        index, digit = divmod(index, base)
        total = total * base + digit
        scale = f(scale * inv)
    return max(f(0.000001), min(f(f(np.uint64(total)) * scale), f(0.999999)))


@pytest.mark.parametrize("width,height", [(1, 1), (2, 3), (16, 9), (33, 28)])
@pytest.mark.parametrize("sample", [0, 1, 1000, 1 << 20, (1 << 31) - 1])
def test_pixel_enumeration_and_jitter(ctx, cornell_path, halton_perm, width, height, sample):
    """Every pixel's global index lands in that pixel (the enumerator's
    property), and its jitter is the two plain radical inverses, scaled, minus
    the pixel, up to the last sample number an int holds."""
    scene = Y.Scene(ctx, Y.HostScene(cornell_path, width, height), halton_perm)
    sx, sy, ex, ey = 1, 1, 0, 0
    while sx < width:
        sx, ex = sx * 2, ex + 1
    while sy < height:
        sy, ey = sy * 3, ey + 1
    px, py = (v.ravel() for v in np.meshgrid(np.arange(width), np.arange(height)))
    index, jitter, _ = scene.halton(px, py, np.full(px.size, sample), 0)
    f = np.float32
    for k in range(px.size):
        i = int(index[k])
        assert i // (sx * sy) == sample
        for axis, (base, scale, digits, p) in enumerate(((2, sx, ex, px[k]), (3, sy, ey, py[k]))):
            v, r = i, 0
            for _ in range(digits):
                v, d = divmod(v, base)
                r = r * base + d
            assert r == p
            want = f(plain_inverse(i, base) * f(scale)) - f(p)
            assert jitter[k][axis] == min(max(f(want), f(0.000001)), f(0.999999))
    scene.close()
