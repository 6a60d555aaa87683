"""GPU tests of the standardised decode-GEMM products through the C ABI, each precision
against the FP64 numpy restatement of Z (oracle): Z^T B and Z B."""
import numpy as np
import pytest

import pcaone_b200 as pb
from oracle import pcaone_oracle as O
from tests.test_gpu_rsvd import random_bed

pytestmark = pytest.mark.gpu

# max |err| / max |ref| per output column. mixed: int8 tensor cores with the sketch as three
# 8-bit fixed-point pieces per column (21 bits below the column maximum); bf16: split BF16
# hi+lo pairs (16 significant bits), FP32 accumulation.
TOL = {"fp64": 1e-12, "fp32": 2e-6, "mixed": 5e-6, "bf16": 5e-5}


def rel_col_err(got, ref):
    return float((np.abs(got - ref).max(axis=0) / np.abs(ref).max(axis=0)).max())


@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed", "bf16"])
@pytest.mark.parametrize("N,M,l", [(1003, 2500, 40), (517, 777, 20), (2048, 1300, 7), (300, 4100, 64)])
def test_products_match_dense(gpu, prec, N, M, l):
    bed = random_bed(N, M, seed=N * 7 + l, miss=0.02)
    Z, F = O.standardized_from_bed(bed)
    gpu.load_bed(bed.packed, N)
    rng = np.random.default_rng(l)
    B1 = rng.standard_normal((N, l))
    got1 = gpu.product_t(B1, precision=prec)
    assert rel_col_err(got1, Z.T @ B1) <= TOL[prec]
    B2 = rng.standard_normal((M, l))
    got2 = gpu.product(B2, precision=prec)
    assert rel_col_err(got2, Z @ B2) <= TOL[prec]


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
@pytest.mark.parametrize("N,M,l", [(1003, 2500, 40), (2048, 1300, 7), (300, 4100, 64)])
def test_int8_pipeline_variants_match_dense(gpu, monkeypatch, variant, N, M, l):
    """Every pipeline variant of the int8 decode-GEMM (the autotuner's choices), pinned one at
    a time: codes through shared memory or from global memory, one- or two-chunk units (wide
    sketches, l = 64, have the one-chunk forms 0 and 2 only)."""
    monkeypatch.setenv("PCAONE_I8_VARIANT", str(variant))
    bed = random_bed(N, M, seed=N * 3 + l + variant, miss=0.02)
    Z, F = O.standardized_from_bed(bed)
    gpu.load_bed(bed.packed, N)
    rng = np.random.default_rng(l + variant)
    B1 = rng.standard_normal((N, l))
    assert rel_col_err(gpu.product_t(B1, precision="mixed"), Z.T @ B1) <= TOL["mixed"]
    B2 = rng.standard_normal((M, l))
    assert rel_col_err(gpu.product(B2, precision="mixed"), Z @ B2) <= TOL["mixed"]


@pytest.mark.parametrize("prec", ["fp64", "mixed", "bf16"])
def test_products_unstandardised_haploid(gpu, prec):
    bed = random_bed(640, 900, seed=3, miss=0.05)
    codes = O.decode_codes(bed)
    F = O.allele_freq(codes)
    Zc = O.centered_matrix(codes, F)
    gpu.load_bed(bed.packed, bed.N)
    B = np.random.default_rng(0).standard_normal((bed.N, 12))
    assert rel_col_err(gpu.product_t(B, precision=prec, standardize=False), Zc.T @ B) <= TOL[prec]
    Zh = O.standardize(Zc, F, ploidy=1)
    assert rel_col_err(gpu.product_t(B, precision=prec, ploidy=1), Zh.T @ B) <= TOL[prec]


@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed", "bf16"])
def test_gram_product_matches_dense(gpu, prec):
    """The IRAM operator Z (Z^T X) in one device call against the oracle's Z."""
    bed = random_bed(777, 3001, seed=21, miss=0.02)
    Z, F = O.standardized_from_bed(bed)
    gpu.load_bed(bed.packed, bed.N)
    X = np.random.default_rng(3).standard_normal((bed.N, 5))
    got = gpu.gram_product(X, precision=prec)
    assert rel_col_err(got, Z @ (Z.T @ X)) <= 2 * TOL[prec]


@pytest.mark.parametrize("N,M", [(64, 63), (65, 129), (127, 2049), (2051, 128), (300, 4100)])
@pytest.mark.parametrize("l", [1, 2, 3, 8, 9, 24, 41, 64])
def test_fp64_products_at_tile_and_chunk_edges(gpu, N, M, l):
    """The FP64 products at the edges of their row tiles (64 and 128), K chunks (64, spans of 2048)
    and column tiles, in the matrix-vector (l <= 2) and the tensor form."""
    bed = random_bed(N, M, seed=N + M + l, miss=0.03)
    gpu.load_bed(bed.packed, N)
    Z, _ = O.standardized_from_bed(bed)
    rng = np.random.default_rng(l)
    for Zx, got in ((Z.T, gpu.product_t), (Z, gpu.product)):
        B = rng.standard_normal((Zx.shape[1], l))
        ref = Zx @ B
        # sums of at most 4100 terms of order 1: error below 4100 * 2^-53 of the largest
        np.testing.assert_allclose(got(B, precision="fp64"), ref, rtol=0, atol=1e-12 * np.abs(ref).max())
    X = rng.standard_normal((N, l))
    ref = Z @ (Z.T @ X)
    np.testing.assert_allclose(gpu.gram_product(X, precision="fp64"), ref, rtol=0, atol=1e-12 * np.abs(ref).max())


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-9), ("fp32", 1e-5)])
@pytest.mark.parametrize("N,M,bands,k", [(203, 1501, 8, 4), (130, 641, 16, 1), (513, 4099, 4, 16)])
def test_simt_window_runs_match_oracle(gpu, precision, tol, N, M, bands, k):
    """winSVD on the FP32 and FP64 back ends, whose windows run as one product: uneven windows."""
    bed = random_bed(N, M, seed=N, miss=0.02)
    gpu.load_bed(bed.packed, N)
    kw = dict(k=k, svd=2, bands=bands, maxp=5, tol=0.0)
    r = gpu.rsvd(precision=precision, **kw)
    S = O.run_pca(bed, shuffle=False, **kw)[1]
    np.testing.assert_allclose(r.S, S, rtol=tol)


@pytest.mark.parametrize("precision", ["mixed", "fp32", "fp64"])
@pytest.mark.parametrize("N,M,l", [(61, 3000, 8), (300, 900, 20), (777, 4500, 15)])
def test_products_with_uneven_missing_rates(gpu, precision, N, M, l):
    """Z B where the samples' missing counts run from none to almost all SNPs: rows summed by one
    warp, by a whole CTA, and empty ones."""
    rng = np.random.default_rng(N)
    bed = random_bed(N, M, seed=N, miss=0.0)
    codes = O.decode_codes(bed).copy()
    rate = np.where(np.arange(N) % 5 == 0, 0.0, rng.beta(1, 4, N))
    rate[3] = 0.99
    miss = rng.random((M, N)) < rate
    miss[:, :8] &= np.arange(M)[:, None] % 7 != 0
    codes = np.where(miss if codes.shape == miss.shape else miss.T, 1, codes).astype(np.uint8)
    snp_major = codes if codes.shape == (M, N) else codes.T
    pad = np.zeros((M, (N + 3) // 4 * 4), dtype=np.uint8)
    pad[:, :N] = snp_major
    pad = pad.reshape(M, -1, 4)
    bed = O.Bed(N, M, (pad[:, :, 0] | pad[:, :, 1] << 2 | pad[:, :, 2] << 4 | pad[:, :, 3] << 6).astype(np.uint8))
    gpu.load_bed(bed.packed, N)
    Z, _ = O.standardized_from_bed(bed)
    B = rng.standard_normal((M, l))
    assert rel_col_err(gpu.product(B, precision=precision), Z @ B) <= TOL[precision]
    X = rng.standard_normal((N, l))
    assert rel_col_err(gpu.product_t(X, precision=precision), Z.T @ X) <= TOL[precision]


def test_mixed_operand_maxima_across_calls(gpu):
    """The window operand's column maxima are cleared by the epilogue that used them last: an RSVD, a
    product with a much larger operand and the RSVD again give the first RSVD's results."""
    bed = random_bed(333, 2100, seed=8, miss=0.02)
    gpu.load_bed(bed.packed, bed.N)
    kw = dict(k=4, svd=2, bands=8, maxp=4, tol=0.0, precision="mixed")
    a = gpu.rsvd(**kw)
    B = 1e6 * np.random.default_rng(2).standard_normal((bed.M, 14))
    gpu.product(B, precision="mixed")
    gpu.gram_product(1e6 * np.ones((bed.N, 14)), precision="mixed")
    b = gpu.rsvd(**kw)
    np.testing.assert_allclose(b.S, a.S, rtol=1e-6)
    S = O.run_pca(bed, k=4, svd=2, bands=8, maxp=4, tol=0.0, shuffle=False)[1]
    np.testing.assert_allclose(b.S, S, rtol=1e-6)


def test_fp32_product_over_long_k(gpu):
    """Enough rows that K is not split: the FP32 sums run over 256 codes at most whatever the length
    of K, so the error stays below 2^-24 sqrt(256 / 2) of a column's size (0.29 units a rounding,
    random walk), where one sum over 8192 would be five times that."""
    N, M, l = 8192, 38000, 64
    packed = np.random.default_rng(6).integers(0, 256, (M, N // 4), dtype=np.uint8)
    gpu.load_bed(packed, N)
    B = np.random.default_rng(7).standard_normal((N, l))
    ref = gpu.product_t(B, precision="fp64")
    assert rel_col_err(gpu.product_t(B, precision="fp32"), ref) <= 2.0 ** -24 * np.sqrt(128)
