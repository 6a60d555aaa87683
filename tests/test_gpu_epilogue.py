"""The missing-entry sums of the second product with two, four and eight warps to a row, in each of their
forms: general (any width, products), FP32 row sums (RSVD) and weighted row sums (EMU)."""
import numpy as np
import pytest

import pcaone_b200 as pb
from oracle import pcaone_oracle as O
from tests.test_gpu_product import TOL, rel_col_err

pytestmark = pytest.mark.gpu

# A row's mean of 256, 512 and 1024 entries is where a row gets two, four and eight warps (few rows here)
WARPS = {1: 600, 2: 1000, 4: 2000, 8: 4000}  # SNPs at a missing rate of 0.3: 180, 300, 600, 1200 entries


def populations(N, M, pops, seed, miss=0.3):
    """Strongly separated populations; missing rates of the samples from a third to five thirds of the
    mean, one sample complete and one almost empty."""
    rng = np.random.default_rng(seed)
    anc = rng.uniform(0.2, 0.8, (M, 1))
    freq = np.clip(anc + 0.25 * rng.standard_normal((M, pops)), 0.03, 0.97)
    p = freq[:, np.arange(N) % pops]
    g = (rng.random((M, N)) < p).astype(int) + (rng.random((M, N)) < p)
    codes = np.array([3, 2, 0], dtype=np.uint8)[g]
    rate = miss * rng.uniform(1 / 3, 5 / 3, N)
    rate[0], rate[N // 2] = 0.0, 0.98
    codes[rng.random((M, N)) < rate] = 1
    pad = np.full((M, (N + 3) // 4 * 4), 3, dtype=np.uint8)
    pad[:, :N] = codes
    pad = pad.reshape(M, -1, 4)
    return O.Bed(N, M, (pad[:, :, 0] | pad[:, :, 1] << 2 | pad[:, :, 2] << 4 | pad[:, :, 3] << 6).astype(np.uint8))


@pytest.mark.parametrize("precision", ["mixed", "fp32", "fp64"])
@pytest.mark.parametrize("warps", list(WARPS))
@pytest.mark.parametrize("N,l", [(61, 7), (203, 20)])
def test_products(gpu, precision, warps, N, l):
    bed = populations(N, WARPS[warps], 4, N + warps)
    gpu.load_bed(bed.packed, N)
    Z, _ = O.standardized_from_bed(bed)
    B = np.random.default_rng(l).standard_normal((bed.M, l))
    assert rel_col_err(gpu.product(B, precision=precision), Z @ B) <= TOL[precision]


@pytest.mark.parametrize("precision,tol", [("mixed", 1e-5), ("fp32", 1e-5)])
@pytest.mark.parametrize("warps", list(WARPS))
@pytest.mark.parametrize("N,k", [(61, 2), (203, 10)])
def test_rsvd_row_sums(gpu, precision, tol, warps, N, k):
    """Widths of 12 and 20, one run of all SNPs."""
    bed = populations(N, WARPS[warps], k + 1, N + warps)
    gpu.load_bed(bed.packed, N)
    kw = dict(k=k, svd=1, maxp=4, tol=0.0)
    r = gpu.rsvd(precision=precision, **kw)
    np.testing.assert_allclose(r.S, O.run_pca(bed, shuffle=False, **kw)[1], rtol=tol)


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("warps", list(WARPS))
@pytest.mark.parametrize("N,k", [(61, 2), (203, 10)])
def test_emu_weighted_row_sums(gpu, precision, warps, N, k):
    bed = populations(N, WARPS[warps], k + 1, N + warps)
    kw = dict(k=k, svd=1, maxp=4, tol=0.0, maxiter=2, tolem=0.0)
    eig = pb.run_emu(gpu, bed.packed, N, precision=precision, **kw)[0]
    np.testing.assert_allclose(eig, O.run_emu(bed, **kw)[0], rtol=1e-5)
