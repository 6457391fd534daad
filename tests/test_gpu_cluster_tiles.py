"""The clustering kernels at the edges of their tiles (rows and columns per block, columns per
round, clusters per block, flattened row length): alphas, norms, centres, representatives,
weights and assignments equal the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,clusters", [(1, 1, 1), (1, 33, 5), (5, 31, 4), (7, 32, 9), (8, 257, 63), (9, 256, 64),
                                                (31, 255, 65), (33, 300, 17), (64, 2049, 66), (67, 4100, 130)])
def test_tiles_match_oracle(ctx, oracle_built, rows, cols, clusters):
    import torch
    from oracle import Oracle
    from renzoku_b200 import rzk
    rng = np.random.default_rng(rows * 10000 + cols)
    m = (rng.gamma(0.3, 1.0, (cols, rows, 3)) * (rng.random((cols, rows, 1)) < 0.6)).astype(np.float32)
    mat = torch.from_numpy(m).cuda()
    cb = rzk.ClusterBuilderCuda()
    for got, want in zip(cb.alphas(mat), Oracle.ltm_alphas(m)):
        assert np.array_equal(got.cpu().numpy(), want)
    for got, want in zip(cb.cluster_by_sampling(mat, clusters, 7), Oracle.cluster_by_sampling(m, clusters, 7)):
        assert np.array_equal(got, want)
