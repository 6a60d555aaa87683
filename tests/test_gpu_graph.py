"""Steady epochs are launched as graphs: a capture that the runtime refuses falls back to direct launches
with the same results, so only a count shows it."""
import ctypes

import numpy as np
import pytest

import pcaone_b200 as pb
from oracle import pcaone_oracle as O
from tests.test_gpu_rsvd import random_bed

pytestmark = pytest.mark.gpu


def graph_epochs(ctx):
    fn = getattr(pb.lib(), "_ZN2pg12graph_epochsEPK10pcaone_ctx")
    fn.restype = ctypes.c_int64
    return fn(ctx._h)


# epochs 0 to 8; bodies are steady from epoch 2 on (2^2 >= 4 bands), the first of them runs directly
@pytest.mark.parametrize("precision", ["mixed", "bf16"])
@pytest.mark.parametrize("svd", [1, 2])
def test_steady_epochs_run_as_graphs(gpu, capfd, precision, svd):
    bed = random_bed(333, 2100, seed=8, miss=0.02)
    gpu.load_bed(bed.packed, bed.N)
    kw = dict(k=4, svd=svd, bands=4, maxp=8, tol=0.0)
    before = graph_epochs(gpu)
    r = gpu.rsvd(precision=precision, verbose=True, **kw)
    assert r.epochs == 9
    assert graph_epochs(gpu) - before == 6
    assert "not launched as graphs" not in capfd.readouterr().err
    S = O.run_pca(bed, shuffle=False, **kw)[1]
    np.testing.assert_allclose(r.S, S, rtol=1e-5)
    gpu.rsvd(precision="fp32", **kw)  # launched directly by design
    assert graph_epochs(gpu) - before == 6
