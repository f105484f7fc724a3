"""The warps of a round follow one another through words in shared memory (changes,
the FP64 warp's progress and answers, rows of pair products that arrive during
the round): sweeps with many changes a round give the same bits every time,
and the oracle's components."""
import numpy as np
import pytest

import oracle_lib as O
from bayesrrcmd_gb300 import gpu, plink

pytestmark = pytest.mark.gpu
S1 = [[0.01, 0.001, 0.0001]]


@pytest.mark.parametrize("kind", [gpu.KIND_DENSE, gpu.KIND_RAGGED, gpu.KIND_EIGEN])
@pytest.mark.parametrize("tokens", [0, 64])
def test_sweeps_with_many_changes_repeat_bit_for_bit(gpu_lib, kind, tokens):
    N, M = 1_500, 2_000
    g, _ = plink.synth_genotypes(N, M, 17 + kind, missing=0.01)
    bed = plink.encode_bed(g)
    y, _, _ = plink.synth_phenotype(g, 17, 60, 0.5)
    first = None
    for _ in range(4):
        ch = gpu.Chain(gpu.ChainConfig(N=N, M=M, kind=kind, S=S1, seed=7, async_batch=tokens))
        ch.pack_bed(bed)
        ch.set_phenotype(y)
        ch.init()
        ch.iterate(6)
        s = ch.state()
        ch.close()
        if first is None:
            first = s
        for k in ("beta", "comp", "acum", "eps"):
            np.testing.assert_array_equal(s[k], first[k], err_msg=k)
    oc = O.OracleChain(bed, N, y, S1, kind=kind, seed=7, async_batch=tokens)
    for it in range(6):
        oc.iterate(it)
    np.testing.assert_array_equal(first["comp"], oc.state()["comp"])
