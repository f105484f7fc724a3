"""Markers packed a second time under a running chain: markers with missing
genotypes need up to four times the pair sums of markers without, and the marker
Gram is another."""
import numpy as np
import pytest

import oracle_lib as O
from bayesrrcmd_gb300 import gpu, plink

pytestmark = pytest.mark.gpu
S1 = [[0.01, 0.001, 0.0001]]


@pytest.mark.parametrize("kind", [gpu.KIND_DENSE, gpu.KIND_RAGGED, gpu.KIND_EIGEN])
@pytest.mark.parametrize("form,rtol,gram", [(gpu.FORM_FP64, 1e-10, 0), (gpu.FORM_FP32C, 1e-9, -1),
                                            (gpu.FORM_FP32C, 1e-9, 1)])
def test_sweep_after_packing_markers_with_missing_genotypes(gpu_lib, kind, form, rtol, gram):
    if gram == 1 and kind != gpu.KIND_DENSE:
        pytest.skip("the Gram-blocked sweep is for dense markers")
    N, M = 900, 4_200
    beds = []
    for miss in (0.0, 0.02):
        g, _ = plink.synth_genotypes(N, M, 5 + kind, missing=miss)
        beds.append(plink.encode_bed(g))
    y, _, _ = plink.synth_phenotype(g, 5, 30, 0.5)
    ch = gpu.Chain(gpu.ChainConfig(N=N, M=M, kind=kind, form=form, S=S1, seed=7, gram=gram))
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


def test_failed_packing_needs_a_new_start(gpu_lib):
    N, M = 300, 40
    g, _ = plink.synth_genotypes(N, M, 3)
    bed = plink.encode_bed(g)
    bad = g.copy()
    bad[7] = 0                      # a marker that does not vary
    y, _, _ = plink.synth_phenotype(g, 3, 5, 0.5)
    ch = gpu.Chain(gpu.ChainConfig(N=N, M=M, S=S1, seed=7))
    ch.pack_bed(bed)
    ch.set_phenotype(y)
    ch.init()
    ch.iterate(1)
    with pytest.raises(gpu.BrrError) as e:
        ch.pack_bed(plink.encode_bed(bad))
    assert e.value.code == -5
    with pytest.raises(gpu.BrrError) as e:
        ch.iterate(1)
    assert e.value.code == -1
    ch.pack_bed(bed)
    ch.init()
    ch.iterate(2)
    oc = O.OracleChain(bed, N, y, S1, seed=7)
    oc.iterate(0)
    oc.iterate(1)
    np.testing.assert_array_equal(ch.state()["comp"], oc.state()["comp"])
    np.testing.assert_allclose(ch.state()["eps"], oc.state()["eps"], rtol=0, atol=1e-11)
    ch.close()
