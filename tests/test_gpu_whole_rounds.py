"""The whole-round sweep at the sizes where it can go wrong, against the FP64
oracle: slices of one and of several 64-individual chunks, rounds of less than
64 markers, every marker kind, round widths, a residual that outgrows its
fixed-point range, pair products of only the markers likely to change, and the
rules that choose widths and rounds.

Bars of one sweep from a shared state: components equal.  The residual is held
in units of 2^-56 of its range and every sum over it is exact, so num differs
from the oracle's, whose N-term FP64 sums carry at most N 2^-53, by less than
1e-11 relative at N <= 1e5; 1e-10 leaves a decade for the M updates of a sweep.
The FP32C form carries num as a pair of FP32 words (2^-46 each step of a
round): 1e-9.
"""
import numpy as np
import pytest

import oracle_lib as O
from bayesrrcmd_gb300 import gpu, plink

pytestmark = pytest.mark.gpu
S1 = [[0.01, 0.001, 0.0001]]


def data(N, M, seed, miss=0.02, p_lo=0.05):
    g, _ = plink.synth_genotypes(N, M, seed, missing=miss, p_lo=p_lo)
    y, _, _ = plink.synth_phenotype(g, seed, max(1, M // 20), 0.5)
    return plink.encode_bed(g), y


def chain(bed, N, y, kind, form, seed=7, **kw):
    ch = gpu.Chain(gpu.ChainConfig(N=N, M=bed.shape[0], kind=kind, form=form, S=S1, seed=seed, **kw))
    ch.pack_bed(bed)
    ch.set_phenotype(y)
    ch.init()
    return ch


def compare(s, o, form, scale=1.0):
    rtol = 1e-10 if form == gpu.FORM_FP64 else 1e-9
    np.testing.assert_array_equal(s["comp"], o["comp"])
    np.testing.assert_array_equal(s["beta"] != 0, o["beta"] != 0)
    np.testing.assert_allclose(s["beta"], o["beta"], rtol=rtol, atol=1e-13 * scale)
    np.testing.assert_allclose(s["eps"], o["eps"], rtol=0, atol=rtol * scale)
    np.testing.assert_allclose(s["sigmaE"], o["sigmaE"], rtol=rtol)


@pytest.mark.parametrize("kind", [gpu.KIND_DENSE, gpu.KIND_RAGGED, gpu.KIND_EIGEN])
@pytest.mark.parametrize("N,M,kw", [
    (61, 1, {}),                        # one slice, one marker
    (65, 64, {}),                       # two slices, one full round
    (9729, 65, {}),                     # one individual past 152 slices of 64; a last round of one marker
    (1027, 191, dict(spec_width=8)),
    (1030, 130, dict(grid=3)),          # several chunks per slice
    (523, 127, dict(cluster=4)),
])
def test_fp64_rounds_match_oracle(gpu_lib, kind, N, M, kw):
    bed, y = data(N, M, seed=N + M + kind)
    ch = chain(bed, N, y, kind, gpu.FORM_FP64, **kw)
    oc = O.OracleChain(bed, N, y, S1, kind=kind, seed=7)
    for it in range(3):
        ch.iterate(1)
        oc.iterate(it)
        compare(ch.state(), oc.state(), gpu.FORM_FP64)
    ch.close()


@pytest.mark.parametrize("kind", [gpu.KIND_DENSE, gpu.KIND_RAGGED, gpu.KIND_EIGEN])
@pytest.mark.parametrize("form", [gpu.FORM_FP64, gpu.FORM_FP32C])
def test_residual_that_outgrows_its_range(gpu_lib, kind, form):
    """Effects of 150 in the state, which a small sigmaG shrinks away, make the
    residual leave, within one sweep, the range it was given at the sweep's start."""
    N, M = 700, 150
    bed, y = data(N, M, seed=3 + kind)
    oc = O.OracleChain(bed, N, y, S1, kind=kind, seed=7)
    ch = chain(bed, N, y, kind, form, **({} if form == gpu.FORM_FP64 else dict(gram=-1)))
    oc.iterate(0)
    st = oc.state()
    st["beta"][::50] = 150.0
    st["comp"][::50] = 1
    st["sigmaG"][:] = 1e-6
    ch.set_state(st)
    oc.set_state(st)
    order = O.permutation(7, 0, 50, M)
    u, z = O.marker_draws(7, 0, 50, M)
    ch.sweep(order, u, z)
    oc.sweep(order, u, z)
    s, o = ch.state(), oc.state()
    scale = np.abs(o["eps"]).max()
    assert scale > 200
    compare(s, o, form, scale)
    ch.close()


@pytest.mark.parametrize("kind,form", [(gpu.KIND_DENSE, gpu.FORM_FP64), (gpu.KIND_EIGEN, gpu.FORM_FP64),
                                       (gpu.KIND_RAGGED, gpu.FORM_FP32C)])
def test_rounds_with_the_products_of_likely_markers_only(gpu_lib, kind, form):
    """N M >= 5e8: a change of a marker whose products were not formed ends its
    round early; the first sweep of a chain has many."""
    N, M = 120_001, 4_200
    bed, y = data(N, M, seed=29, miss=0.0 if kind == gpu.KIND_DENSE else 0.01)
    ch = chain(bed, N, y, kind, form)
    oc = O.OracleChain(bed, N, y, S1, kind=kind, seed=7)
    for it in range(2):
        ch.iterate(1)
        oc.iterate(it)
        compare(ch.state(), oc.state(), form)
    assert ch.timing()[2] >= -(-M // 64)
    ch.close()


@pytest.mark.parametrize("M", [4095, 4096])
@pytest.mark.parametrize("kind", [gpu.KIND_DENSE, gpu.KIND_RAGGED])
def test_fp32c_width_rule(gpu_lib, kind, M):
    """Rounds of 64 with pair products from 4,096 markers on; below, 32 markers
    and, for dense markers, rounds that end at a change."""
    N = 400
    bed, y = data(N, M, seed=M)
    ch = chain(bed, N, y, kind, gpu.FORM_FP32C, gram=-1)
    oc = O.OracleChain(bed, N, y, S1, kind=kind, seed=7)
    for it in range(2):
        ch.iterate(1)
        oc.iterate(it)
        compare(ch.state(), oc.state(), gpu.FORM_FP32C)
    rounds = ch.timing()[2]
    if M >= 4096:
        assert rounds == -(-M // 64)
    elif kind == gpu.KIND_RAGGED:
        assert rounds >= -(-M // 32)
    ch.close()
