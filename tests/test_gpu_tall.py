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
