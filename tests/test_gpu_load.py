"""Uploads: the records' row layout, counts and frequencies at ragged record lengths, and matrices
large enough for the chunked host copies in both directions."""
import numpy as np
import pytest

import pcaone_b200 as pb

pytestmark = pytest.mark.gpu


def counts_of(packed, N):
    codes = np.stack([packed >> s & 3 for s in (0, 2, 4, 6)], 2).reshape(packed.shape[0], -1)[:, :N]
    n00, n10, n01 = ((codes == c).sum(1) for c in (0, 2, 1))
    return 2 * n00 + n10, N - n01


# record bytes 1, 2, 3, 5, 16, 17, 64, 65 (every start alignment), then more than 8 MiB in all: chunks of
# whole records, the last one ragged, tiny and long records, and records longer than a chunk
@pytest.mark.parametrize("N,M", [(1, 7), (5, 300), (12, 33), (17, 1001), (64, 40), (65, 129), (256, 50), (257, 77),
                                 (4099, 9003), (17, 1800003), (100003, 411), (4200001, 71)])
def test_load_layout_counts_and_frequencies(gpu, N, M):
    rng = np.random.default_rng(N + M)
    packed = rng.integers(0, 256, (M, (N + 3) // 4), dtype=np.uint8)
    gpu.load_bed(packed, N)
    a, c = gpu.counts()
    ra, rc = counts_of(packed, N)
    np.testing.assert_array_equal(a, ra)
    np.testing.assert_array_equal(c, rc)
    F = np.divide(ra * 0.5, rc, out=np.zeros(M), where=rc > 0)
    np.testing.assert_array_equal(gpu.allele_freq(), F)
    perm = rng.permutation(M).astype(np.int32)
    gpu.permute(perm)
    a, c = gpu.counts()
    np.testing.assert_array_equal(a, ra[perm])
    np.testing.assert_array_equal(c, rc[perm])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_large_likelihoods_and_results_round_trip(gpu, dtype):
    """Likelihoods above the chunked copies' threshold give the posterior of the same values loaded
    in small pieces would: F after one sweep against numpy; loadings of a wide matrix come back
    orthonormal (all chunks of the read-back present)."""
    N, M = 61, 140003
    rng = np.random.default_rng(1)
    g = rng.dirichlet(np.ones(3), size=(M, N)).astype(dtype)
    P = np.ascontiguousarray(g[:, :, :2].reshape(M, 2 * N)).T
    gpu.load_gl(P)
    F, it = gpu.gl_freq(1, 1e-6)
    assert it == 1
    p = g.astype(np.float64)
    p0, p1 = p[:, :, 0] * 0.75 ** 2, p[:, :, 1] * 2 * 0.25 * 0.75
    p2 = (1 - p[:, :, 0] - p[:, :, 1]) * 0.25 ** 2
    np.testing.assert_allclose(F, ((p1 + 2 * p2) / (p0 + p1 + p2)).sum(1) / (2 * N), rtol=1e-12)
    gpu.gl_update()
    r = gpu.rsvd(k=10, svd=1, maxp=2, tol=0.0, precision="fp32", standardize=False)
    np.testing.assert_allclose(r.V.T @ r.V, np.eye(10), atol=1e-9)


def test_large_context_reuse_keeps_padding(gpu):
    """A smaller matrix loaded after a larger one on the same context: counts of the new one."""
    for N, M in ((4099, 9003), (203, 1500), (4098, 9001)):
        packed = np.random.default_rng(M).integers(0, 256, (M, (N + 3) // 4), dtype=np.uint8)
        gpu.load_bed(packed, N)
        a, c = gpu.counts()
        ra, rc = counts_of(packed, N)
        np.testing.assert_array_equal(a, ra)
        np.testing.assert_array_equal(c, rc)
    assert pb.lib() is not None
