"""GPU float64 Gram (update_gram) through the C ABI against numpy float64."""
import numpy as np
import pytest

import alto_b200 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,rank", [(1, 1), (7, 3), (1000, 8), (4096, 16), (100000, 32), (33333, 64),
                                       (5000, 100), (2000, 128), (0, 16)])
def test_gram_matches_float64(rows, rank):
    import torch

    rng = np.random.default_rng(rows + rank)
    U = rng.uniform(-1, 1, (rows, rank)).astype(np.float32)
    G = A.gram(torch.tensor(U, device="cuda")).cpu().numpy()
    ref = U.astype(np.float64).T @ U.astype(np.float64)
    np.testing.assert_allclose(G, ref, rtol=1e-12, atol=1e-12 * max(1.0, np.abs(ref).max()))
    assert np.array_equal(G, G.T)


def test_gram_rejects_large_rank():
    import torch

    with pytest.raises(A.AltoError) as e:
        A.gram(torch.zeros((4, 129), device="cuda"))
    assert e.value.status == A.ERR_UNSUPPORTED


@pytest.mark.parametrize("rank", [1, 7, 8, 9, 16, 17, 24, 25, 31, 32, 33, 63, 64, 65, 127])
@pytest.mark.parametrize("rows", [1, 3, 8, 63, 65, 515])
def test_gram_at_tile_edges(rows, rank):
    """Tiles of 8 columns and steps of 4 rows, with remainders in both; products
    of float32 values are exact in float64, so the bound is that of adding 515 terms
    in any order (515 * 2^-53 * the sum of absolute values < 6e-14 of it)."""
    import torch

    U = np.random.default_rng(rows * 131 + rank).uniform(-1, 1, (rows, rank)).astype(np.float32)
    G = A.gram(torch.tensor(U, device="cuda")).cpu().numpy()
    V = U.astype(np.float64)
    assert np.all(np.abs(G - V.T @ V) <= 2 * 6e-14 * (np.abs(V).T @ np.abs(V)))
    assert np.array_equal(G, G.T)
