"""The Gram-blocked sweep on grids of few CTAs, where the dot warps gather the
staged Gram entries that the chore warp's lanes leave (below 80 CTAs at 64 markers
per block; more than one entry per thread below 20), against the FP64 oracle.

Bars of the FP32C form: components equal, beta within 1e-9 relative (num as a pair of
FP32 words, 2^-46 per change of a block), the residual within 1e-10."""
import numpy as np
import pytest

import oracle_lib as O
from bayesrrcmd_gb300 import gpu, plink

pytestmark = pytest.mark.gpu
S1 = [[0.01, 0.001, 0.0001]]


@pytest.mark.parametrize("N,M,grid", [(60, 200, 0), (1027, 193, 0), (2000, 321, 19), (4000, 330, 20), (6000, 200, 79),
                                      (6000, 200, 80)])
def test_blocked_sweep_of_few_slices_matches_oracle(gpu_lib, N, M, grid):
    g, _ = plink.synth_genotypes(N, M, 3 * N + M, missing=0.01, p_lo=0.1)
    bed = plink.encode_bed(g)
    y, _, _ = plink.synth_phenotype(g, 5, max(1, M // 20), 0.5)
    ch = gpu.Chain(gpu.ChainConfig(N=N, M=M, kind=gpu.KIND_DENSE, form=gpu.FORM_FP32C, S=S1, seed=4, gram=1, grid=grid))
    ch.pack_bed(bed)
    ch.set_phenotype(y)
    ch.init()
    oc = O.OracleChain(bed, N, y, S1, kind=0, seed=4)
    for it in range(3):
        ch.iterate(1)
        oc.iterate(it)
        s, o = ch.state(), oc.state()
        np.testing.assert_array_equal(s["comp"], o["comp"])
        np.testing.assert_allclose(s["beta"], o["beta"], rtol=1e-9, atol=1e-13)
        np.testing.assert_allclose(s["eps"], o["eps"], rtol=0, atol=1e-10)
    ch.close()
