"""Deposits of wide splats (radius over 1.4), which are composited from the tile's
sorted records instead of per-texel lists: record counts at the edges of the
sorted runs (32) and of the window (576), and radii from just above the rule's
line to boxes larger than a tile.  Texels within 1e-6 of the restatement, the
bound of every deposit test: the blend's operations and their order are the
same."""
import numpy as np
import pytest

import ggb_cases as K

pytestmark = pytest.mark.gpu


def crowded(n, seed, spread):
    """n short arcs within `spread` of one direction, one or two samples each."""
    rng = np.random.default_rng(seed)
    a = np.array([0.05, 0.03, 1.0]) + rng.uniform(-spread, spread, size=(n, 3))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    b = a + rng.uniform(-0.01, 0.01, size=(n, 3))
    b /= np.linalg.norm(b, axis=1, keepdims=True)
    return a.astype(np.float32), b.astype(np.float32), rng.uniform(0.05, 1.0, size=(n, 4)).astype(np.float32)


@pytest.mark.parametrize("radius", [1.4375, 2.5])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 575, 576, 577, 1300])
def test_wide_deposit_record_counts(gpu, orc32, n, radius):
    prev, pos, col = crowded(n, n, 0.2)
    a = K.deposit(gpu, 40, prev, pos, col, radius=radius)
    b = K.deposit(orc32, 40, prev, pos, col, radius=radius)
    assert np.max(np.abs(a["faces"] - b["faces"])) <= 1e-6


@pytest.mark.parametrize("R,radius", [(1, 1.5), (15, 1.375), (17, 3.0), (33, 7.5), (50, 16.0), (64, 40.0)])
def test_wide_deposit_radii(gpu, orc32, R, radius):
    prev, pos, col = K.random_arcs(700, 11, 0.3)
    a = K.deposit(gpu, R, prev, pos, col, fade_steps=3, radius=radius)
    b = K.deposit(orc32, R, prev, pos, col, fade_steps=3, radius=radius)
    assert np.max(np.abs(a["faces"] - b["faces"])) <= 1e-6


@pytest.mark.parametrize("radius", [0.75, 1.0, 1.25, 1.375])
@pytest.mark.parametrize("n,spread", [(40, 0.01), (200, 0.02), (500, 0.02), (575, 0.05), (576, 0.05), (577, 0.05),
                                      (900, 0.2), (1200, 0.01), (2500, 0.2)])
def test_dense_lists(gpu, orc32, n, spread, radius):
    """Narrower splats on a few texels: lists of 16 to several hundred entries,
    tiles of one to several windows; bound as above."""
    prev, pos, col = crowded(n, n + 1, spread)
    a = K.deposit(gpu, 40, prev, pos, col, radius=radius)
    b = K.deposit(orc32, 40, prev, pos, col, radius=radius)
    assert np.max(np.abs(a["faces"] - b["faces"])) <= 1e-6
