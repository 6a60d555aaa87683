"""Large host copies on the GPU: memory the caller has pinned, several contexts copying at once, and what
a context that is loaded again keeps of the matrix before."""
import threading

import numpy as np
import pytest

import pcaone_b200 as pb
from tests.test_gpu_load import counts_of

pytestmark = pytest.mark.gpu


def records(N, M, seed):
    return np.random.default_rng(seed).integers(0, 256, (M, (N + 3) // 4), dtype=np.uint8)


def pinned(a):
    torch = pytest.importorskip("torch")
    t = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True)
    out = t.numpy().view(a.dtype).reshape(a.shape)
    out[...] = a
    return out, t


@pytest.mark.parametrize("N,M", [(17, 1800003), (4099, 70001)])
def test_pinned_records_and_likelihoods(N, M):
    """Records pinned by the caller (several pieces of 64 MiB, the last ragged): counts as from pageable
    memory; likelihoods in both types: the same frequencies."""
    a = records(N, M, 1)
    p, _keep = pinned(a)
    with pb.GpuContext(0) as c:
        c.load_bed(p, N)
        got = c.counts()
        for x, y in zip(got, counts_of(a, N)):
            np.testing.assert_array_equal(x, y)
        for dtype in (np.float32, np.float64):
            P = np.random.default_rng(2).random((60001, 2 * 101)).astype(dtype) / 2.5
            c.load_gl(P.T)
            F = c.gl_freq(3, 0.0)[0]
            q, _k = pinned(P)
            c.load_gl(q.T)
            np.testing.assert_array_equal(c.gl_freq(3, 0.0)[0], F)


def test_pinned_and_pageable_results(gpu):
    N, M = 301, 30011
    gpu.load_bed(records(N, M, 3), N)
    ref = gpu.residuals()
    assert ref.nbytes > 32 << 20
    out, _keep = pinned(np.full_like(ref, np.nan))
    gpu._check(pb.lib().pcaone_gpu_residuals(gpu._h, None, None, None, 0, 0, M, pb._ptr(out)))
    np.testing.assert_array_equal(out, ref)


def test_contexts_copy_at_once():
    """Uploads and results of four contexts on four host threads, which share the pinned slots: as each
    alone."""
    shapes = [(301, 30011), (1003, 50021), (64, 600000), (4099, 9003)]
    failures = []

    def results(t):
        N, M = shapes[t]
        out = []
        with pb.GpuContext(0) as c:
            for i in range(3):
                c.load_bed(records(N, M, 10 * t + i), N)
                out += [*c.counts(), c.residuals()]
        return out

    alone = [results(t) for t in range(4)]

    def work(t):
        try:
            for x, y in zip(results(t), alone[t]):
                np.testing.assert_array_equal(x, y)
        except BaseException as e:  # noqa: BLE001 - reported by the test
            failures.append((t, e))

    th = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for x in th:
        x.start()
    for x in th:
        x.join()
    assert not failures, failures


def test_reloaded_context_agrees_with_a_fresh_one(gpu, monkeypatch):
    """A smaller matrix after a larger one, twice, with samples and SNPs that end inside a word and a row
    tile: what the products, a permutation and an RSVD read of the rows, their padding and the rows past
    the last SNP is that of a fresh context, bit for bit (one pipeline of the int8 product: the tuner's choice is by time)."""
    monkeypatch.setenv("PCAONE_I8_VARIANT", "0")
    for N, M in ((4099, 9003), (203, 1500), (4098, 9001), (61, 777)):
        a = records(N, M, N)
        rng = np.random.default_rng(M)
        X, Y, perm = rng.standard_normal((N, 5)), rng.standard_normal((M, 5)), rng.permutation(M).astype(np.int32)

        def results(c):
            c.load_bed(a, N)
            out = [c.product_t(X, precision=p) for p in ("mixed", "fp32", "fp64")]
            out += [c.product(Y, precision=p) for p in ("mixed", "fp32", "fp64")]
            c.permute(perm)
            out += list(c.counts())
            r = c.rsvd(k=3, svd=2, bands=8, maxp=4, tol=0.0, precision="fp64")
            return out + [r.U, r.S, r.V]

        with pb.GpuContext(0) as fresh:
            ref = results(fresh)
        for x, y in zip(results(gpu), ref):
            np.testing.assert_array_equal(x, y)
