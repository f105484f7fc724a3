"""Genetic values at the edges of the refresh kernel's tiles (128 individuals per
CTA, 64 markers at a time) against the same sums in NumPy, terms in the same
order: each step rounds once on the GPU (FMA) and twice in NumPy, so the two are
within 2 n 2^-53 of the sum of |b x|."""
import numpy as np
import pytest

from bayesrrcmd_gb300 import gpu, plink

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [gpu.KIND_DENSE, gpu.KIND_RAGGED])
@pytest.mark.parametrize("N,n", [(5, 0), (127, 1), (128, 63), (129, 64), (1027, 65), (300, 130)])
def test_xbeta_at_tile_edges(gpu_lib, kind, N, n):
    M = 140
    g, _ = plink.synth_genotypes(N, M, N + n, missing=0.02, p_lo=0.3)
    g[:, 0], g[:, 1], g[:, 2] = 0, 1, 2
    bed = plink.encode_bed(g)
    rng = np.random.default_rng(n)
    idx = rng.permutation(M)[:n].astype(np.uint32)
    b = rng.normal(size=n)
    with gpu.Chain(gpu.ChainConfig(N=N, M=M, kind=kind, S=[[0.01, 0.001]])) as ch:
        ch.pack_bed(bed)
        table, _ = ch.marker_table()
        out = ch.xbeta(idx, b)
    code = np.stack([(bed >> (2 * k)) & 3 for k in range(4)], 2).reshape(M, -1)[:, :N]
    want, size = np.zeros(N), np.zeros(N)
    for j, bj in zip(idx, b):
        if kind == gpu.KIND_DENSE:
            x = table[j][code[j]]
        else:
            x = (np.array([2.0, 0.0, 1.0, 0.0]) - table[j, 0])[code[j]] / table[j, 1]
            x[code[j] == 1] = 0.0
        want += bj * x
        size += np.abs(bj * x)
    np.testing.assert_array_less(np.abs(out - want), 2 * max(n, 1) * 2.0**-53 * size + 1e-300)
