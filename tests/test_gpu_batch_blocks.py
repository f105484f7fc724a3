"""The batched sweep at the edges of its blocks and of its division of chains over
warps, against the FP64 oracle: one block, a second block of one marker, full last
blocks (an odd and an even number of them), and few CTAs, whose resolver warps take
several chains each.

Bars: components equal; beta within 1e-9 relative (num is carried as a pair of
FP32 words, 2^-46 per step of a block, fixed point 2^-40 of the residual: N 2^-41 over
a num of order sqrt(N)); the residual within 1e-10 (one rounding of 2^-41 per change).
"""
import numpy as np
import pytest

import oracle_lib as O
from bayesrrcmd_gb300 import gpu, plink

pytestmark = pytest.mark.gpu
S1 = [[0.01, 0.001, 0.0001]]


@pytest.mark.parametrize("N,M,C,grid", [
    (330, 1, 32, 0),       # one marker
    (330, 32, 64, 0),      # one block
    (500, 33, 32, 0),      # a second block of one marker
    (901, 64, 64, 0),      # two blocks
    (900, 97, 64, 0),      # four blocks, the last of one marker
    (1000, 160, 64, 3),    # 21 or 22 chains per CTA, five or six per resolver warp
    (300, 70, 32, 1),      # one CTA
    (53_000, 40, 64, 0),   # the largest slices that fit 64 chains
])
def test_batch_blocks_match_oracle(gpu_lib, N, M, C, grid):
    g, _ = plink.synth_genotypes(N, M, 5 + M, missing=0.0, p_lo=0.05)
    bed = plink.encode_bed(g)
    ys = np.stack([plink.synth_phenotype(g, 100 + c, max(1, M // 8), 0.3 + 0.1 * (c % 5))[0]
                   for c in range(C)]).astype(np.float32)
    b = gpu.Batch(gpu.ChainConfig(N=N, M=M, S=S1, seed=9, chain=2, grid=grid), C)
    b.pack_bed(bed)
    b.set_phenotypes(ys)
    b.init()
    checked = (0, 1, C // 2, C - 1)
    oracles = {c: O.OracleChain(bed, N, ys[c], S1, seed=9, chain=2 + c, perm_chain=2) for c in checked}
    for it in range(3):
        b.iterate(1)
        for c, oc in oracles.items():
            oc.iterate(it)
            s, o = b.state(c), oc.state()
            what = f"iteration {it} chain {c}"
            np.testing.assert_array_equal(s["comp"], o["comp"], err_msg=what)
            np.testing.assert_array_equal(s["beta"] != 0, o["beta"] != 0, err_msg=what)
            np.testing.assert_allclose(s["beta"], o["beta"], rtol=1e-9, atol=1e-13, err_msg=what)
            np.testing.assert_allclose(s["eps"], o["eps"], rtol=0, atol=1e-10, err_msg=what)
            np.testing.assert_allclose(s["acum"], o["acum"], rtol=2e-6, atol=1e-12, err_msg=what)
    b.close()
