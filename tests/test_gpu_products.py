"""Products at the edges of their tiles: the persistent CTA pairs of more than 256 rows (tiles, k remainders, k splits, rounds), the f32 decode kernel."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    (257, 256, 64),     # the smallest batch that takes them, half a stage of k
    (272, 255, 72),     # rows of a tile past the matrix, k that ends inside a slab
    (300, 384, 200),    # the second CTA of the last pair without weight rows
    (512, 1024, 4096),  # k splits
    (513, 130, 136),    # one row in the last token tile
    (700, 8, 1096),     # fewer weight rows than a quarter of a warpgroup
    (2065, 18, 2048),   # one weight tile: a router's columns, k splits
    (3072, 16, 1032),   # the most tokens of one weight tile that pairs take
    (3073, 18, 1032),   # ... and single CTAs from there on
    (300, 128, 72),
    (300, 129, 72),
    (1031, 6400, 136),  # more than one round of the 74 pairs, ragged
    (512, 9728, 264),   # two tiles more than a round: the last ones in pieces
    (2065, 2432, 392),  # nine token tiles: a group of eight and one more
]


@pytest.fixture(scope="module")
def backend(pkg):
    return pkg.CudaBackend(0)


@pytest.mark.parametrize("rows,n,k", SHAPES)
def test_products_of_many_rows(pkg, backend, rows, n, k):
    rng = np.random.default_rng(rows * 7 + n)
    from oracle import binding as oracle
    x, w = (oracle.round_to_bf16(rng.standard_normal(s).astype(np.float32)) for s in ((rows, k), (n, k)))
    got = pkg.ops.linear(backend, x, w, None, pkg.DType.BF16)
    exact, size = x.astype(np.float64) @ w.T.astype(np.float64), np.abs(x).astype(np.float64) @ np.abs(w).T.astype(np.float64)
    # products of bf16 are exact in f32; an MMA adds 16 of them and the accumulator, each sum cut off below 2^-23 of what stands in it at most,
    # and a k split one rounding more
    bound = (k / 16 + 8) * 2.0 ** -23 * size
    assert np.all(np.abs(got - exact) <= bound), float(np.max(np.abs(got - exact) / bound))


@pytest.mark.parametrize("rows,n,k,splits", [(300, 64, 512, 1), (1280, 16, 2048, 4), (2048, 18, 2048, 4), (3072, 16, 2048, 3), (3073, 16, 2048, 4), (8192, 128, 1024, 2)])
def test_one_weight_tile_is_split_along_k(pkg, backend, rows, n, k, splits):
    """Routers: a single weight tile, so k splits are what fills the chip, whatever the number of tokens."""
    ms, used = ctypes.c_float(), ctypes.c_uint32()
    pkg.errors.check(pkg._ffi.lib().orion_cuda_linear_bench(backend._h, rows, k, n, 1, 1, ctypes.byref(ms), ctypes.byref(used)))
    assert used.value == splits


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 64, 65])
@pytest.mark.parametrize("n,k", [(1, 4), (17, 100), (130, 128), (16, 132), (33, 684), (15, 6)])
def test_f32_products_of_few_rows_are_bit_exact(pkg, backend, rows, n, k):
    """The kernel of decode batches, its neighbours in rows and k it does not take: one chain of additions per output, whatever the tile."""
    from oracle import binding as oracle
    rng = np.random.default_rng(rows * 7 + n + k)
    x, w = rng.standard_normal((rows, k)).astype(np.float32), rng.standard_normal((n, k)).astype(np.float32)
    assert np.array_equal(pkg.ops.linear(backend, x, w), oracle.linear(x, w))


@pytest.mark.parametrize("rows,n", [(32, 40001), (33, 32499), (33, 32500), (57, 20312), (64, 20313), (65, 400)])
def test_f32_products_on_both_sides_of_the_rule_are_bit_exact(pkg, backend, rows, n):
    """More than 32 rows against a large vocabulary go to the tiles of 64 x 64 outputs."""
    from oracle import binding as oracle
    rng = np.random.default_rng(rows + n)
    x, w = rng.standard_normal((rows, 20)).astype(np.float32), rng.standard_normal((n, 20)).astype(np.float32)
    assert np.array_equal(pkg.ops.linear(backend, x, w), oracle.linear(x, w))
