"""The device fuzzy-kNN construction (si_fuzzy_graph, csrc/fuzzy.cu) against
the reference's stage fixtures (tests/generate_fixtures.py:70-182) and the
oracle (oracle/fuzzy_oracle.py): exact kNN, smooth-kNN sigma / rho, and the
pruned fuzzy union, on the datasets whose stage inputs are committed."""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import GOLDEN
from oracle import fuzzy_oracle as F

pytestmark = pytest.mark.gpu


def _npz(ds, name):
    return np.load(GOLDEN / ds / f"{name}.npz", allow_pickle=False)


@pytest.mark.parametrize("ds", ["blobs_connected_200", "moons_200", "near_dupes_100"])
def test_fuzzy_graph_stages_match_fixtures(gpu_ctx, ds):
    import spectral_init_b200 as si
    x = _npz(ds, "step0_raw_data")["X"]
    ref1 = _npz(ds, "step1_knn_exact")
    ref2 = _npz(ds, "step2_smooth_knn_exact")
    k = int(ref1["n_neighbors"])
    g, (idx, dist, sig, rho) = si.fuzzy_graph(x, k, ctx=gpu_ctx, return_stages=True)
    if ds == "near_dupes_100":
        # the generator forms distances as |x|^2 - 2 x.y + |y|^2 clipped at 0,
        # so near-duplicate pairs carry cancellation noise (zeros there where
        # the device's difference form gives ~2e-7); rho follows the first
        # positive distance and is not pinned for those rows, nor is which
        # duplicate is a neighbour
        assert np.allclose(dist, ref1["knn_dists"], rtol=1e-6, atol=1e-6)
        return
    assert np.allclose(dist, ref1["knn_dists"], rtol=1e-6, atol=1e-7)
    assert np.allclose(rho, ref2["rhos"], rtol=1e-6, atol=1e-7)
    assert np.allclose(sig, ref2["sigmas"], rtol=1e-5, atol=1e-7)  # +inf rows included
    assert np.array_equal(idx, ref1["knn_indices"])
    ref5 = sp.load_npz(GOLDEN / ds / "step5a_pruned_exact.npz").tocsr()
    ref5.sort_indices()
    assert np.array_equal(g.indptr, ref5.indptr) and np.array_equal(g.indices, ref5.indices)
    assert np.allclose(g.data, ref5.data, rtol=2e-6, atol=1e-7)


def test_fuzzy_graph_matches_oracle_on_a_larger_cloud(gpu_ctx):
    """3000 points of a 6-cluster mixture in 10-D, k = 15: the device graph
    equals the oracle's (structure exactly, values to f32 rounding)."""
    import spectral_init_b200 as si
    rng = np.random.default_rng(5)
    centres = rng.normal(0, 4, (6, 10))
    x = np.concatenate([rng.normal(0, 1, (500, 10)) + c for c in centres])
    g = si.fuzzy_graph(x, 15, ctx=gpu_ctx)
    ref = F.fuzzy_graph(x, 15)
    ref.sort_indices()
    assert np.array_equal(g.indptr, ref.indptr) and np.array_equal(g.indices, ref.indices)
    assert np.allclose(g.data, ref.data, rtol=2e-6, atol=1e-7)
    assert (g != g.T).nnz == 0


@pytest.mark.parametrize("n,d,k", [(2, 1, 1), (17, 3, 16), (64, 16, 5), (65, 17, 17), (129, 1, 32), (700, 50, 15),
                                   (4097, 33, 16)])
def test_knn_tile_edges_and_ties(gpu_ctx, n, d, k):
    """Exact neighbours at the edges of query, candidate and feature tiles.
    Integer coordinates: squared distances are exact and full of ties, which
    go to the smaller index."""
    import spectral_init_b200 as si
    rng = np.random.default_rng(n + d)
    x = rng.integers(0, 4, (n, d)).astype(np.float64)
    _, (idx, dist, _, _) = si.fuzzy_graph(x, k, ctx=gpu_ctx, return_stages=True)
    sq = (x * x).sum(1)
    for s in range(0, n, 512):
        d2 = sq[s:s + 512, None] + sq[None, :] - 2.0 * (x[s:s + 512] @ x.T)  # exact in f64
        d2[np.arange(d2.shape[0]), np.arange(s, s + d2.shape[0])] = np.inf
        want = np.argsort(d2, axis=1, kind="stable")[:, :k]
        assert np.array_equal(idx[s:s + 512], want)
        assert np.array_equal(dist[s:s + 512], np.sqrt(np.take_along_axis(d2, want, 1)).astype(np.float32))


def test_fuzzy_graph_with_a_hub(gpu_ctx):
    """Points in random directions around one centre, which is everybody's
    nearest neighbour: its row is far longer than a warp sorts."""
    import spectral_init_b200 as si
    rng = np.random.default_rng(11)
    v = rng.normal(size=(1500, 40))
    x = np.concatenate([np.zeros((1, 40)), v / np.linalg.norm(v, axis=1, keepdims=True)
                        * rng.uniform(1.0, 1.2, (1500, 1))])
    g = si.fuzzy_graph(x, 5, ctx=gpu_ctx)
    ref = F.fuzzy_graph(x, 5)
    ref.sort_indices()
    assert np.max(np.diff(g.indptr)) > 1000
    assert np.array_equal(g.indptr, ref.indptr) and np.array_equal(g.indices, ref.indices)
    assert np.allclose(g.data, ref.data, rtol=2e-6, atol=1e-7)
