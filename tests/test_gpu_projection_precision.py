"""FP32 sums of the CUDA-core projections hold 256 products at most; the rest is double-float.

Chains of 8 products a lane (7 rounded additions; the first product and the additions round together) and a
tree over 32 lanes (5 more) are off by (8 + 5) 2^-24 of the sum of the products' sizes at most.
Constant vectors are the worst case for a chain: every lane rounds alike, and at the constants below
chains of 128 are off by 1.9e-6."""
import numpy as np
import pytest

import gdmr

pytestmark = pytest.mark.gpu

BOUND = 13 * 2.0 ** -24
CONSTANTS = np.array([0.985774994, 0.7071068, 0.61803399, 0.9857, 0.51, 0.8415, 0.5403, 0.9093, 0.4161, 0.1411, 0.99, 0.7568,
                      0.6536, 0.9589, 0.2837, 0.2794], np.float32)


@pytest.mark.parametrize("variant", [0, 9])
@pytest.mark.parametrize("n,k,nsys", [
    (884736, 24, 16),       # one warp a tile of outputs
    (500001, 16, 8),        # two warps a tile, odd n
    (1800000, 4, 2),        # four
    (200, 24, 33),          # three groups of systems, two chunks of rows
])
def test_sums_of_constants(variant, n, k, nsys):
    c = CONSTANTS[np.arange(nsys) % CONSTANTS.size]
    W = np.ones((k, n), np.complex64)
    W[1::2] = 1j
    Y = np.repeat(c[:, None], n, axis=1).astype(np.complex64)
    gdmr.tune_force(variant, -1)
    try:
        got = gdmr.projection_check(W, Y)
    finally:
        gdmr.tune_force(-1, -1)
    exact = n * c.astype(np.float64)[:, None] * np.where(np.arange(k) % 2 == 0, 1.0, -1j)[None]
    err = (np.abs(got - exact) / np.abs(exact)).max()
    print(f"n {n} k {k} nsys {nsys} variant {variant}: {err:.2e}")
    assert err <= BOUND


@pytest.mark.parametrize("n,k,nsys", [(262144, 24, 16), (100345, 16, 5), (50000, 32, 64)])
def test_sums_of_gaussians(n, k, nsys):
    rng = np.random.default_rng(4)
    W, Y = (rng.standard_normal((q, n), np.float32) + 1j * rng.standard_normal((q, n), np.float32) for q in (k, nsys))
    gdmr.tune_force(9, -1)
    try:
        got = gdmr.projection_check(W, Y)
    finally:
        gdmr.tune_force(-1, -1)
    exact = Y.astype(np.complex128) @ W.conj().T.astype(np.complex128)
    size = np.linalg.norm(Y, axis=1)[:, None] * np.linalg.norm(W, axis=1)[None]
    assert (np.abs(got - exact) / size).max() <= BOUND
