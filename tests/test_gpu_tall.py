"""The FP64 passes on tall matrices (Omega update, epoch tail) through RSVD runs at every column
tile count and at the edges of their row split, against the oracle's Householder QR."""
import numpy as np
import pytest

from oracle import pcaone_oracle as O
from tests.test_gpu_rsvd import random_bed

pytestmark = pytest.mark.gpu

# (samples, k, oversamples): l = k + oversamples covers 1 to 8 column tiles of 8, full and ragged;
# the rows end inside an 8-row group, a CTA's 64 rows, and a cluster's 512 rows
CASES = [(67, 1, 1), (64, 2, 6), (65, 4, 5), (71, 3, 13), (511, 7, 10), (512, 12, 12), (513, 10, 21), (1025, 16, 24),
         (777, 20, 27), (4099, 24, 32), (130, 28, 29), (20003, 32, 32)]


@pytest.mark.parametrize("N,k,os_", CASES)
@pytest.mark.parametrize("svd", [1, 2])
def test_rsvd_widths_and_row_edges(gpu, N, k, os_, svd):
    M = 700
    bed = random_bed(N, M, seed=N + k, miss=0.01)
    gpu.load_bed(bed.packed, N)
    kw = dict(k=k, oversamples=os_, maxp=3, tol=0.0, svd=svd, bands=4)
    r = gpu.rsvd(precision="fp64", **kw)
    _, S, U, V, _, epochs = O.run_pca(bed, shuffle=False, **kw)
    assert r.epochs == epochs
    # unstructured data: singular values within a factor of 10 of one another, so the sketch's
    # condition number stays below 1e3 and CholeskyQR2 (error eps cond^2) below 1e-9
    np.testing.assert_allclose(r.S, S, rtol=1e-9)
    np.testing.assert_allclose(r.U.T @ r.U, np.eye(k), atol=1e-9)
    np.testing.assert_allclose(r.V.T @ r.V, np.eye(k), atol=1e-9)


@pytest.mark.parametrize("N,k,os_", [(40, 1, 1), (203, 4, 10), (1000, 20, 21), (5003, 12, 20)])
@pytest.mark.parametrize("rand,seed", [(1, 101), (0, 101), (1, 0), (0, 7), (1, 2147483647), (1, -5)])
def test_sketch_drawn_on_the_device(gpu, N, k, os_, rand, seed):
    """One epoch from the seeded sketch (a fraction of a CTA's candidates to several hundred CTAs):
    singular values of Z^T Omega's range depend on every value of Omega."""
    bed = random_bed(N, 400, seed=5, miss=0.0)
    gpu.load_bed(bed.packed, N)
    kw = dict(k=k, oversamples=os_, maxp=0, tol=0.0, svd=1, seed=seed, rand=rand)
    r = gpu.rsvd(precision="fp64", **kw)
    Z, _ = O.standardized_from_bed(bed)  # one epoch by hand: the oracle's loop needs two
    G = Z.T @ O.omega(seed, N, k + max(os_, k), rand)
    R = np.linalg.qr(G)[1]
    S = np.linalg.svd(np.linalg.solve(R.T, (Z @ G).T), compute_uv=False)[:k]
    np.testing.assert_allclose(r.S, S, rtol=1e-9)
