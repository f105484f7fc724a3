"""Residuals that no fixed-point grid holds as finely as FP64 does: a phenotype
value far from the others, values that are not finite.  Such sweeps run on the
restart sweep, in every variant that the whole-round sweep has.

Bars against the FP64 oracle are those of the chain tests, 1e-10 relative; of
the residual absolute at the outlier's size."""
import numpy as np
import pytest

import oracle_lib as O
from bayesrrcmd_gb300 import gpu, plink

pytestmark = pytest.mark.gpu
S1 = [[0.01, 0.001, 0.0001]]
KINDS = [gpu.KIND_DENSE, gpu.KIND_RAGGED, gpu.KIND_EIGEN]


def data(N, M, seed, sd, miss=0.01):
    """Genotypes, and a normal phenotype with one value `sd` standard deviations out."""
    g, _ = plink.synth_genotypes(N, M, seed, missing=miss, p_lo=0.05)
    y, _, _ = plink.synth_phenotype(g, seed, max(1, M // 20), 0.5)
    y[17] = sd / np.sqrt(1.0 - sd * sd / N)
    return g, plink.encode_bed(g), y


def chain(bed, N, y, kind, form=gpu.FORM_FP64, **kw):
    ch = gpu.Chain(gpu.ChainConfig(N=N, M=bed.shape[0], kind=kind, form=form, S=S1, seed=7, **kw))
    ch.pack_bed(bed)
    ch.set_phenotype(y)
    ch.init()
    return ch


def compare(s, o, what=""):
    np.testing.assert_array_equal(s["comp"], o["comp"], err_msg=what)
    nz = o["beta"] != 0
    np.testing.assert_allclose(s["beta"][nz], o["beta"][nz], rtol=1e-10, err_msg=what)
    np.testing.assert_allclose(s["sigmaE"], o["sigmaE"], rtol=1e-10, err_msg=what)
    np.testing.assert_allclose(s["eps"], o["eps"], rtol=0, atol=1e-11 * np.abs(o["eps"]).max(), err_msg=what)


@pytest.mark.parametrize("kind", KINDS)
def test_residual_is_rounded_no_more_than_in_fp64(gpu_lib, kind):
    """Three sweeps from shared draws against eps - sum dBeta x of the chain's own
    effects in extended precision.  A change of the residual in FP64 rounds each value
    to its spacing s, an error of s / sqrt(12) in the root mean square if it is
    random; 1.5 times that over n changes is the bar.  A grid of 2^-51 (the finest
    below 2^62 for a value of 250 with three bits of headroom) has 4.5 times."""
    N, M = 100_003, 60
    g, bed, y = data(N, M, 5 + kind, 250.0)
    ch = chain(bed, N, y, kind)
    table, counts = ch.marker_table()
    s = ch.state()
    exact = s["eps"].astype(np.longdouble)
    n = 0
    for it in range(3):
        order = O.permutation(7, 0, it, M)
        u, z = O.marker_draws(7, 0, it, M)
        old = s["beta"]
        ch.sweep(order, u, z)
        s = ch.state()
        for j in np.flatnonzero((old != 0) | (s["beta"] != 0)):
            dB = np.longdouble(old[j]) - np.longdouble(s["beta"][j])
            if kind == gpu.KIND_DENSE:
                x = table[j][[3, 2, 0, 1]]                        # genotype 0, 1, 2, missing
            else:
                x = np.append((np.arange(3) - table[j, 0]) / table[j, 1], 0.0)
            exact += dB * x.astype(np.longdouble)[np.where(g[j] < 0, 3, g[j])]
            n += 1
    assert n > 0
    err = np.delete((s["eps"] - exact).astype(np.float64), 17)
    spacing = np.spacing(np.abs(np.delete(s["eps"], 17)))
    assert np.sqrt((err ** 2).mean()) < 1.5 * np.sqrt(n * (spacing ** 2).mean() / 12)
    ch.close()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("kw", [{}, dict(grid=40), dict(cluster=16), dict(spec_width=64), dict(async_batch=20)])
def test_outlier_chain_matches_oracle(gpu_lib, kind, kw):
    N, M = 40_009, 130
    _, bed, y = data(N, M, 15 + kind, 150.0)
    ch = chain(bed, N, y, kind, **kw)
    oc = O.OracleChain(bed, N, y, S1, kind=kind, seed=7, async_batch=kw.get("async_batch", 0))
    for it in range(3):
        ch.iterate(1)
        oc.iterate(it)
        compare(ch.state(), oc.state(), f"iteration {it}")
        if "async_batch" not in kw:
            # a round per change: the restart sweep
            assert ch.timing()[2] > -(-M // 64) + 10
    ch.close()


def test_outlier_instances_match_their_oracles(gpu_lib):
    """Two instances of a multi-instance run leave the common sweep, one stays."""
    shapes = [(40_009, 90, gpu.KIND_DENSE, 150.0), (3_001, 120, gpu.KIND_DENSE, 5.0), (41_003, 70, gpu.KIND_RAGGED, 170.0)]
    probs = [(N, M, kind) + data(N, M, 31 + k, sd)[1:] for k, (N, M, kind, sd) in enumerate(shapes)]
    m = gpu.Multi([gpu.ChainConfig(N=N, M=M, kind=kind, S=S1, seed=3, chain=k) for k, (N, M, kind, _, _) in enumerate(probs)])
    for k, (N, M, kind, bed, y) in enumerate(probs):
        m.pack_bed(k, bed)
        m.set_phenotype(k, y)
    m.init()
    m.iterate(2)
    m.tune(1)                       # four iterations
    m.iterate(1)
    for k, (N, M, kind, bed, y) in enumerate(probs):
        oc = O.OracleChain(bed, N, y, S1, kind=kind, seed=3, chain=k)
        for it in range(7):
            oc.iterate(it)
        compare(m.state(k), oc.state(), f"instance {k}")
    m.close()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("form", [gpu.FORM_FP64, gpu.FORM_FP32C])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_residual_that_is_not_finite_is_refused(gpu_lib, kind, form, value):
    N, M = 700, 150
    _, bed, y = data(N, M, 23 + kind, 5.0)
    ch = chain(bed, N, y, kind, form, **({} if form == gpu.FORM_FP64 else dict(gram=-1)))
    ch.iterate(1)
    st = ch.state()
    st["eps"][5] = value
    ch.set_state(st)
    before = ch.state()
    with pytest.raises(gpu.BrrError) as e:
        ch.sweep(O.permutation(7, 0, 50, M), *O.marker_draws(7, 0, 50, M))
    assert e.value.code == -6
    after = ch.state()
    for k in ("beta", "comp", "acum", "eps"):
        np.testing.assert_array_equal(after[k], before[k], err_msg=k)
    ch.close()
