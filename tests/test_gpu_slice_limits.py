"""Multi-instance runs whose slices lie between the shared memory a CTA of the
whole-round sweep has beside its static arrays and 220 KB: 94 chunks of 64
individuals at 8 markers per round need 224,912 bytes, 70 chunks at 32 markers and
five groups 225,056.  They run on more CTAs, in narrower rounds or on the restart
sweep; every individual is on one of 152 CTAs.  Bars of the multi-instance tests."""
import numpy as np
import pytest

import oracle_lib as O
from bayesrrcmd_gb300 import gpu, plink

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [gpu.KIND_DENSE, gpu.KIND_RAGGED])
@pytest.mark.parametrize("N,groups,width", [(152 * 94 * 64, 1, 0), (152 * 70 * 64, 5, 32)])
def test_largest_slices(gpu_lib, kind, N, groups, width):
    M = 24
    g, _ = plink.synth_genotypes(N, M, 9, missing=0.01, p_lo=0.05)
    bed = plink.encode_bed(g)
    y, _, _ = plink.synth_phenotype(g, 9, 6, 0.4)
    S = [[0.01, 0.001, 0.0001]] * groups
    group = (np.arange(M) % groups).astype(np.int32)
    m = gpu.Multi([gpu.ChainConfig(N=N, M=M, kind=kind, S=S, seed=3, spec_width=width)])
    m.pack_bed(0, bed)
    m.set_groups(0, group)
    m.set_phenotype(0, y)
    m.init()
    oc = O.OracleChain(bed, N, y, S, kind=kind, group=group, seed=3)
    for it in range(2):
        m.iterate(1)
        oc.iterate(it)
        s, o = m.state(0), oc.state()
        np.testing.assert_array_equal(s["comp"], o["comp"])
        nz = o["beta"] != 0
        np.testing.assert_allclose(s["beta"][nz], o["beta"][nz], rtol=1e-10)
        np.testing.assert_allclose(s["eps"], o["eps"], rtol=0, atol=1e-11)
    m.close()
