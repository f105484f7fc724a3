"""Component decisions of the FP64 form with u next to P(component 0).

One marker, residual c x, so that num is a sum of positive terms; P(component 0) =
1 / (1 + exp(D)) with D = log pi_1 - log pi_0 - log(1 + sigmaG (N-1) S / sigmaE) / 2 +
num^2 / (2 den sigmaE) between 400 and 600 moves by 2 D of a relative change of num.
In FP64 num carries two roundings, D half a dozen of at most 2^-53 of itself: under 1e-12
of P, usually 3e-13.  A num of 48 bits (2^-49 of itself) moves P by up to 2.1e-12,
one from double-float products (2^-44) by 6e-11.  u lies 1.5e-12 of P to either side."""
import numpy as np
import pytest

from bayesrrcmd_gb300 import gpu, plink

pytestmark = pytest.mark.gpu
N, S = 400, 0.01


@pytest.mark.parametrize("kind", [gpu.KIND_DENSE, gpu.KIND_RAGGED])
@pytest.mark.parametrize("kw", [{}, dict(async_batch=1), dict(cluster=2)])
def test_draws_next_to_the_boundary(gpu_lib, kind, kw):
    rng = np.random.default_rng(11)
    g, _ = plink.synth_genotypes(N, 1, 3)
    ch = gpu.Chain(gpu.ChainConfig(N=N, M=1, kind=kind, S=[[S]], seed=1, **kw))
    ch.pack_bed(plink.encode_bed(g))
    ch.set_phenotype(rng.normal(size=N).astype(np.float32))
    ch.init()
    table = ch.marker_table()[0][0]
    if kind == gpu.KIND_DENSE:
        x = table[[3, 2, 0]][g[0]]
    else:
        x = (g[0] - table[0]) / table[1]
    L = np.longdouble
    st = ch.state()
    st["pi"][0, :2] = 0.5
    st["sigmaG"][:], st["sigmaE"], st["mu"] = 1.0, 1.0, 0.0
    den = L(N - 1) + 1 / L(S)
    bad = []
    for trial in range(120):
        st["eps"] = rng.uniform(1.6, 1.94) * x
        st["epsSum"] = float(st["eps"].sum())
        if kind == gpu.KIND_DENSE:
            num = (x.astype(L) * st["eps"].astype(L)).sum()
        else:
            num = ((g[0] - L(table[0])) * st["eps"].astype(L)).sum() / L(table[1])
        D = num * num / (2 * den) - np.log1p(L(N - 1) * L(S)) / 2
        assert 390 < D < 620
        for side in (-1, 1):
            u = float(np.exp(-D) * (1 + side * L(1.5e-12)))
            ch.set_state(st)
            ch.sweep(np.zeros(1, np.uint32), np.array([u]), np.zeros(1))
            if ch.state()["comp"][0] != (1 if side > 0 else 0):
                bad.append((trial, side))
    assert not bad, (len(bad), bad[:5])
    ch.close()
