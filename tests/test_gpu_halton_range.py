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
