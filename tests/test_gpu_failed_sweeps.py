"""A sweep that ends with a status leaves effects, components, P(component 0) and,
where the sweep writes it to a buffer of its own, the residual as they were
before it."""
import numpy as np
import pytest

import oracle_lib as O
from bayesrrcmd_gb300 import gpu, plink

pytestmark = pytest.mark.gpu
S1 = [[0.01, 0.001, 0.0001]]
RANGE, TIMEOUT = -6, -4


def data(N, M, seed, miss=0.02):
    g, _ = plink.synth_genotypes(N, M, seed, missing=miss, p_lo=0.05)
    y, _, _ = plink.synth_phenotype(g, seed, max(1, M // 20), 0.5)
    return plink.encode_bed(g), y


def chain(bed, N, y, **kw):
    ch = gpu.Chain(gpu.ChainConfig(N=N, M=bed.shape[0], S=S1, seed=7, **kw))
    ch.pack_bed(bed)
    ch.set_phenotype(y)
    ch.init()
    return ch


def unchanged(a, b, names=("beta", "comp", "acum")):
    for k in names:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("kind", [gpu.KIND_DENSE, gpu.KIND_RAGGED, gpu.KIND_EIGEN])
@pytest.mark.parametrize("form", [gpu.FORM_FP64, gpu.FORM_FP32C])
def test_refused_residual_leaves_the_state(gpu_lib, kind, form):
    """The first marker of the sweep holds an effect of 3e16, which a tiny sigmaG
    takes away whole (num^2 h stays below 20, far from the 700 guards): the residual
    leaves every grid and the range of the dot products that follow."""
    N, M = 300, 150
    bed, y = data(N, M, seed=3 + kind)
    ch = chain(bed, N, y, kind=kind, form=form, **({} if form == gpu.FORM_FP64 else dict(gram=-1)))
    ch.iterate(2)
    st = ch.state()
    order = O.permutation(7, 0, 50, M)
    u, z = O.marker_draws(7, 0, 50, M)
    st["beta"][order[0]] = 3e16
    st["comp"][order[0]] = 1
    st["sigmaG"][:] = 1e-35
    ch.set_state(st)
    before = ch.state()
    with pytest.raises(gpu.BrrError) as e:
        ch.sweep(order, u, z)
    assert e.value.code == RANGE
    unchanged(ch.state(), before, ("beta", "comp", "acum", "eps"))
    ch.close()


@pytest.mark.parametrize("miss", [0.0, 0.02])
def test_blocked_sweep_that_ran_out_of_time_leaves_the_effects(gpu_lib, miss):
    """The waits of the third sweep run out before its first block is decided."""
    N, M = 1500, 300
    bed, y = data(N, M, seed=11, miss=miss)
    ch = chain(bed, N, y, form=gpu.FORM_FP32C, gram=1)
    ch.iterate(2)
    before = ch.state()
    ch.set_wait_limit(50_000_000, 1)
    with pytest.raises(gpu.BrrError) as e:
        ch.iterate(1)
    assert e.value.code == TIMEOUT
    unchanged(ch.state(), before)
    ch.close()


def test_batched_sweep_that_ran_out_of_time_leaves_the_effects(gpu_lib):
    """The same for the chains of a batch."""
    N, M, C = 1000, 96, 32
    bed, y = data(N, M, seed=12, miss=0.0)
    rng = np.random.default_rng(12)
    b = gpu.Batch(gpu.ChainConfig(N=N, M=M, form=gpu.FORM_FP32C, S=S1, seed=4), C)
    b.pack_bed(bed)
    b.set_phenotypes(np.stack([y + 0.1 * rng.normal(size=N) for _ in range(C)]))
    b.init()
    b.iterate(2)
    before = [b.state(c) for c in range(C)]
    b.set_wait_limit(50_000_000, 1)
    with pytest.raises(gpu.BrrError) as e:
        b.iterate(1)
    assert e.value.code == TIMEOUT
    for c in range(C):
        unchanged(b.state(c), before[c])
    b.close()
