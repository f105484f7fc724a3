"""Markers packed a second time under a running chain: markers with missing
genotypes need up to four times the pair sums of markers without."""
import numpy as np
import pytest

import oracle_lib as O
from bayesrrcmd_gb300 import gpu, plink

pytestmark = pytest.mark.gpu
S1 = [[0.01, 0.001, 0.0001]]


@pytest.mark.parametrize("kind", [gpu.KIND_DENSE, gpu.KIND_RAGGED, gpu.KIND_EIGEN])
@pytest.mark.parametrize("form,rtol", [(gpu.FORM_FP64, 1e-10), (gpu.FORM_FP32C, 1e-9)])
def test_sweep_after_packing_markers_with_missing_genotypes(gpu_lib, kind, form, rtol):
    N, M = 900, 4_200
    beds = []
    for miss in (0.0, 0.02):
        g, _ = plink.synth_genotypes(N, M, 5 + kind, missing=miss)
        beds.append(plink.encode_bed(g))
    y, _, _ = plink.synth_phenotype(g, 5, 30, 0.5)
    ch = gpu.Chain(gpu.ChainConfig(N=N, M=M, kind=kind, form=form, S=S1, seed=7, gram=-1 if form == gpu.FORM_FP32C else 0))
    ch.pack_bed(beds[0])
    ch.set_phenotype(y)
    ch.init()
    ch.iterate(1)
    ch.pack_bed(beds[1])
    oc = O.OracleChain(beds[1], N, y, S1, kind=kind, seed=7)
    oc.set_state(ch.state())
    order = O.permutation(7, 0, 50, M)
    u, z = O.marker_draws(7, 0, 50, M)
    ch.sweep(order, u, z)
    oc.sweep(order, u, z)
    s, o = ch.state(), oc.state()
    np.testing.assert_array_equal(s["comp"], o["comp"])
    nz = o["beta"] != 0
    np.testing.assert_allclose(s["beta"][nz], o["beta"][nz], rtol=rtol, atol=1e-13)
    np.testing.assert_allclose(s["eps"], o["eps"], rtol=0, atol=rtol)
    ch.close()
