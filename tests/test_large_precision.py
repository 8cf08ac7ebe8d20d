"""Large-scene precision (the 2x2-domain square of the precision workload at
half size: 4096x4096 cells, strips of transform length 4096): FP32 GPU
against the FP64 oracle, next to the float oracle's own distance from FP64."""
import numpy as np
import pytest

from parity import rel

pytestmark = pytest.mark.gpu


def test_large_square_fp32_vs_fp64(oracle_mod):
    from openpstd_gb300 import scenes
    from openpstd_gb300.kernel import PSTDKernel
    steps = 3
    conf = scenes.large_square(1, half=2048, steps=steps, n_receivers=16)
    k = PSTDKernel()
    k.initialize_kernel(conf)
    k.advance(steps)
    k.synchronize()
    o64 = oracle_mod.OracleScene(conf, 64)
    o64.run(steps, threads=oracle_mod.max_threads())
    o32 = oracle_mod.OracleScene(conf, 32)
    o32.run(steps, threads=oracle_mod.max_threads())
    # after a few steps the pulse has not reached the receivers (their series
    # are round-off), so the whole fields are compared
    for d in range(4):                               # the four air domains
        for f in ("p0", "vx", "vy"):
            w = o64.snapshot(d, f)
            e, fl = rel(k.snapshot(d, f), w), rel(o32.snapshot(d, f), w)
            print(d, f, "gpu vs f64", e, "f32 oracle vs f64", fl)
            assert e <= max(1e-5, 3 * fl + 1e-6), (d, f, e, fl)


FORMS = [f"4096:{i}" for i in range(15) if i != 4] + ["chain 0", "chain 1", "chain 2", "serving"]   # 4: not tuned


@pytest.fixture(scope="module")
def large_reference(oracle_mod):
    """The scene, its FP64 fields and the float oracle's distance to them."""
    from openpstd_gb300 import scenes
    conf = scenes.large_square(1, half=2048, steps=3, n_receivers=16)
    out = {}
    o64, o32 = oracle_mod.OracleScene(conf, 64), oracle_mod.OracleScene(conf, 32)
    o64.run(3, threads=oracle_mod.max_threads())
    o32.run(3, threads=oracle_mod.max_threads())
    for d in range(4):
        for f in ("p0", "vx", "vy"):
            w = o64.snapshot(d, f)
            out[d, f] = w, rel(o32.snapshot(d, f), w)
    return conf, out


@pytest.mark.parametrize("form", FORMS)
def test_every_form_the_plan_may_choose(large_reference, monkeypatch, form):
    """The same bound for each variant of length 4096 that the autotuner may
    choose, for the chained families and for the serving configuration."""
    from openpstd_gb300.kernel import PSTDKernel
    conf, want = large_reference
    monkeypatch.setenv("PSTD_AUTOTUNE", "0")
    key, value = ("PSTD_CHAIN", form[-1]) if form.startswith("chain") else ("PSTD_PLAN", form)
    monkeypatch.setenv(key, value)
    k = PSTDKernel()
    k.initialize_kernel(conf)
    k.advance(3)
    k.synchronize()
    info = k.plan_info()
    assert "chained launches (forced)" in info if key == "PSTD_CHAIN" else "pinned by PSTD_PLAN" in info
    for (d, f), (w, fl) in want.items():
        e = rel(k.snapshot(d, f), w)
        assert e <= max(1e-5, 3 * fl + 1e-6), (d, f, e, fl)
    k.close()
