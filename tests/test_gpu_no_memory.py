"""Chains whose device allocations are refused at initialisation, from the n-th on:
the sweep runs without the buffers it did not get (rounds that end at their first
change without pair products, the restart sweep without a second residual) and
follows the FP64 oracle.  No memory is filled: in a process of its own a stand-in
for cudaMalloc refuses the calls."""
import subprocess
import sys
import textwrap
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
TESTS = Path(__file__).resolve().parent

SETUP = """
    import ctypes, sys
    sys.path[:0] = [{tests!r}, {root!r}]
    budget = ctypes.CDLL({lib!r}, mode=ctypes.RTLD_GLOBAL).cuda_budget
    budget.argtypes = [ctypes.c_long]
    import numpy as np
    import oracle_lib as O
    from bayesrrcmd_gb300 import gpu, plink
    S1 = [[0.01, 0.001, 0.0001]]
    def data(N, M, seed):
        g, _ = plink.synth_genotypes(N, M, seed, missing=0.01, p_lo=0.05)
        y, _, _ = plink.synth_phenotype(g, seed, max(1, M // 20), 0.5)
        return plink.encode_bed(g), y
    def compare(s, o, rtol):
        np.testing.assert_array_equal(s["comp"], o["comp"])
        nz = o["beta"] != 0
        np.testing.assert_allclose(s["beta"][nz], o["beta"][nz], rtol=rtol, atol=1e-13)
        np.testing.assert_allclose(s["acum"], o["acum"], rtol=0, atol=1e-5 if rtol > 1e-9 else 1e-9)
        np.testing.assert_allclose(s["eps"], o["eps"], rtol=0, atol=max(rtol, 1e-11))
"""

CHAIN = """
    N, M = {N}, 150
    for kind in (gpu.KIND_DENSE, gpu.KIND_RAGGED, gpu.KIND_EIGEN):
        bed, y = data(N, M, 3 + kind)
        for kw in ({kws}):
            ch = gpu.Chain(gpu.ChainConfig(N=N, M=M, kind=kind, S=S1, seed=7, gram=-1, **kw))
            ch.pack_bed(bed)
            ch.set_phenotype(y)
            budget({calls})
            ch.init()
            budget(-1)
            oc = O.OracleChain(bed, N, y, S1, kind=kind, seed=7, async_batch=kw.get("async_batch", 0))
            for it in range(3):
                ch.iterate(1)
                oc.iterate(it)
                compare(ch.state(), oc.state(), 1e-7 if kw.get("form") == gpu.FORM_FP32C else 1e-10)
                if not kw.get("async_batch"):
                    assert ch.timing()[2] > -(-M // 64) + 10      # a round per change
            ch.close()
"""

TIMEOUT = """
    N, M = 1_500, 150
    bed, y = data(N, M, 3)
    for kw in (dict(), dict(cluster=8)):
        ch = gpu.Chain(gpu.ChainConfig(N=N, M=M, S=S1, seed=7, **kw))
        ch.pack_bed(bed)
        ch.set_phenotype(y)
        budget(0)
        ch.init()
        budget(-1)
        ch.set_wait_limit(50_000_000, 1)
        try:
            ch.iterate(1)
            raise SystemExit("no timeout")
        except gpu.BrrError as e:
            assert e.code == -4
        ch.set_wait_limit(2_000_000_000, 0)
        ch.init()
        oc = O.OracleChain(bed, N, y, S1, kind=0, seed=7)
        for it in range(2):
            ch.iterate(1)
            oc.iterate(it)
        compare(ch.state(), oc.state(), 1e-10)
        assert ch.timing()[2] > -(-M // 64) + 10
        ch.close()
    m = gpu.Multi([gpu.ChainConfig(N=N, M=M, S=S1, seed=3, chain=k) for k in range(2)])
    for k in range(2):
        m.pack_bed(k, bed)
        m.set_phenotype(k, y)
    budget(0)
    m.init()
    budget(-1)
    m.set_wait_limit(50_000_000, 1, instance=1)
    try:
        m.iterate(1)
        raise SystemExit("no timeout")
    except gpu.BrrError as e:
        assert e.code == -4
    m.set_wait_limit(2_000_000_000, 0)
    m.init()
    m.iterate(2)
    for k in range(2):
        oc = O.OracleChain(bed, N, y, S1, kind=0, seed=3, chain=k)
        oc.iterate(0)
        oc.iterate(1)
        compare(m.state(k), oc.state(), 1e-10)
    m.close()
"""

MULTI = """
    shapes = [(2_500, 300, gpu.KIND_DENSE), (1_203, 150, gpu.KIND_RAGGED), (5_000, 100, gpu.KIND_EIGEN)]
    probs = [(N, M, kind) + data(N, M, 40 + k) for k, (N, M, kind) in enumerate(shapes)]
    m = gpu.Multi([gpu.ChainConfig(N=N, M=M, kind=kind, form={form}, S=S1, seed=3, chain=k)
                   for k, (N, M, kind, _, _) in enumerate(probs)])
    for k, (N, M, kind, bed, y) in enumerate(probs):
        m.pack_bed(k, bed)
        m.set_phenotype(k, y)
    budget({calls})
    m.init()
    m.iterate(1)
    budget(-1)
    m.tune(1)
    m.iterate(1)
    for k, (N, M, kind, bed, y) in enumerate(probs):
        oc = O.OracleChain(bed, N, y, S1, kind=kind, seed=3, chain=k)
        for it in range(6):
            oc.iterate(it)
        compare(m.state(k), oc.state(), {rtol})
    m.close()
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("budget") / "libcuda_budget.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(out), str(TESTS / "cuda_budget.c"), "-ldl"], check=True)
    return str(out)


def run(code, lib, **kw):
    text = textwrap.dedent(SETUP.format(tests=str(TESTS), root=str(TESTS.parent), lib=lib) + code.format(**kw))
    r = subprocess.run([sys.executable, "-c", text], capture_output=True, text=True, timeout=200)
    assert r.returncode == 0, r.stderr[-3000:]


# FP64: six buffers (residual, records), then the pair sums and the pair products
@pytest.mark.parametrize("calls", [0, 4, 6, 7])
def test_chain(gpu_lib, lib, calls):
    run(CHAIN, lib, calls=calls, N=1_500, kws="dict(), dict(grid=1), dict(cluster=8), dict(async_batch=20), dict(spec_width=8)")


@pytest.mark.parametrize("calls", [0, 5])
def test_fp32c_chain(gpu_lib, lib, calls):
    run(CHAIN, lib, calls=calls, N=1_500, kws="dict(form=gpu.FORM_FP32C, pair_rounds=-1), dict(form=gpu.FORM_FP32C, cluster=4)")


# a second or third instance without its buffers takes the others to the restart sweep
@pytest.mark.parametrize("form,rtol", [("gpu.FORM_FP64", 1e-10), ("gpu.FORM_FP32C", 1e-7)])
@pytest.mark.parametrize("calls", [0, 3, 6, 11, 17])
def test_multi(gpu_lib, lib, calls, form, rtol):
    run(MULTI, lib, calls=calls, form=form, rtol=rtol)


def test_waits_of_the_restart_sweep_run_out_and_the_chain_recovers(gpu_lib, lib):
    run(TIMEOUT, lib)
