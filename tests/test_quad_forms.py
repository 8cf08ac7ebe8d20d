"""The four-strip stage kernels (stage_quad.cuh) and the chained launch form
(stage_chain.cu) against the oracle: every compiled variant of every transform
length, on scenes whose strips are odd in number and length, whose interface
runs start at odd strips (unaligned columns, unaligned neighbours) and whose
partial PML domains carry copy jobs.  Tolerance: that of the other parity
tests (fields within 2x the float oracle's own distance to FP64)."""
import ctypes

import numpy as np
import pytest

from parity import rel
from test_gpu_parity import check_parity

# transform length -> the two domains (cells), the second's offset along the shared edge, PML cells
SCENES = {32: (13, 14, 13, 15, 9, 10), 64: (21, 25, 29, 26, 9, 20)}
SCENES.update({L: (n, 61, 97, 75, 21, 50) for L, n in
               {128: 50, 256: 181, 512: 333, 1024: 611, 2048: 1203, 4096: 2003, 8192: 4101}.items()})


def _quads(L):
    from openpstd_gb300 import _lib
    buf, n = ctypes.create_string_buffer(1 << 14), ctypes.c_int32()
    assert _lib.lib().pstd_stage_variants(L, buf, 1 << 14, ctypes.byref(n)) == 0
    return [int(line.split(" ", 1)[0]) for line in buf.value.decode().splitlines() if " quad" in line]


def _offset_pair(L, steps=8, tall=False):
    """Two domains that share part of an edge, so that strip runs start at odd
    strips, the first with x strips of transform length L; tall: the same
    turned by a right angle."""
    from openpstd_gb300 import scenes
    from openpstd_gb300.config import PSTDConfiguration
    nx, ny, mx, my, off, pml = SCENES[L]
    conf = PSTDConfiguration()
    scenes.base_settings(conf, steps, dx=0.2, pml=pml)
    e = dict(left=0.6, right=0.4, top=0.8, bottom=0.5)
    rects = [(0, 0, nx, ny), (nx, off, mx, my)]
    if tall:
        rects = [(y, x, h, w) for x, y, w, h in rects]
    conf.Domains = [scenes._domain(*r, 0.2, e) for r in rects]
    conf.Speakers = [((r[0] + r[2] / 2 + 0.25) * 0.2, (r[1] + r[3] / 2 + 0.25) * 0.2, 0.0) for r in rects]
    conf.Receivers = []
    return conf


def test_variants_listed(pstd_lib):
    for L in SCENES:
        assert _quads(L), L


@pytest.mark.gpu
@pytest.mark.parametrize("tall", [False, True])
@pytest.mark.parametrize("L", sorted(SCENES))
def test_every_quad_variant(oracle_mod, monkeypatch, L, tall):
    conf = _offset_pair(L, tall=tall)
    monkeypatch.setenv("PSTD_AUTOTUNE", "0")
    for i in _quads(L):
        monkeypatch.setenv("PSTD_PLAN", f"{L}:{i}")
        k, rep = check_parity(oracle_mod, conf, 8, threads=16)
        assert "pinned by PSTD_PLAN" in k.plan_info()
        k.close()


@pytest.mark.gpu
@pytest.mark.parametrize("fam", [0, 1, 2])
@pytest.mark.parametrize("L", sorted(SCENES))
def test_chained_form(oracle_mod, monkeypatch, L, fam):
    monkeypatch.setenv("PSTD_CHAIN", str(fam))
    for tall in (False, True):
        k, rep = check_parity(oracle_mod, _offset_pair(L, tall=tall), 8, threads=16)
        assert "chained launches (forced)" in k.plan_info()
        k.close()


@pytest.mark.gpu
@pytest.mark.parametrize("fam", [0, 1, 2])
def test_chained_receivers_and_steps(oracle_mod, monkeypatch, fam):
    """Receivers, the first-step flag, reset and runs of 1, 2, 3, 7 steps in a
    row give what single steps give, bit for bit; the solve matches the oracle."""
    from openpstd_gb300 import scenes
    from openpstd_gb300.kernel import PSTDKernel
    monkeypatch.setenv("PSTD_CHAIN", str(fam))
    conf = scenes.l_shape(2, scale=0.2, steps=60)
    check_parity(oracle_mod, conf, 60, threads=16)
    k = PSTDKernel()
    k.initialize_kernel(conf)
    for _ in range(13):
        k.advance(1)
    want, p = k.receivers(), [k.snapshot(i, "px") for i in range(k.domain_count())]
    k.reset()
    for n in (1, 2, 3, 7):
        k.advance(n)
    assert np.array_equal(k.receivers(), want)
    assert all(np.array_equal(k.snapshot(i, "px"), p[i]) for i in range(k.domain_count()))
    assert rel(want, np.zeros_like(want)) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("env,chained", [({"PSTD_CHAIN": "0"}, True), ({"PSTD_AUTOTUNE": "0"}, False)])
def test_profile_counts_the_launches_of_its_form(monkeypatch, env, chained):
    from openpstd_gb300 import scenes
    from openpstd_gb300.kernel import PSTDKernel
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    k = PSTDKernel()
    k.initialize_kernel(scenes.l_shape(2, scale=0.2, steps=10))
    lengths = k.plan_info().count("L=")
    assert lengths >= 2
    got = k.profile_passes(3)
    assert got["stage_launches"] == 3 * 6 * (1 if chained else lengths)
    assert got["total_launches"] == 3 * k.work_counts()["launches_per_step"] == got["stage_launches"] + 3 * (1 if chained else 2)
    k.close()
