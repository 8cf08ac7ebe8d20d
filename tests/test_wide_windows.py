"""Windows of more than 32 cells (a patch error above 71 dB): more band
positions than the fused, staged and pipelined forms hold, so those are not
chosen (tests/test_plan_rules.py), and the other forms compute them.
Tolerances: those of the parity tests."""
import ctypes

import numpy as np
import pytest

from parity import rel
from test_gpu_parity import check_parity
from test_plan_rules import _windowed

pytestmark = pytest.mark.gpu


def _lshape(patch, steps=12):
    from openpstd_gb300 import scenes
    conf = scenes.l_shape(2, scale=0.25, steps=steps, pml=70)
    conf.Settings.SetPatchError(patch)
    assert 32 < conf.Settings.GetWindowSize() <= 70
    return conf


FORMS = {"untuned": {"PSTD_AUTOTUNE": "0"}, "tuned": {}, "chain0": {"PSTD_CHAIN": "0"}, "chain1": {"PSTD_CHAIN": "1"},
         "chain2": {"PSTD_CHAIN": "2"}, "merged": {"PSTD_MERGED": "1"}, "serving": {"PSTD_PLAN": "serving"}}


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("patch", [75.0, 100.0, 120.0])
def test_wide_window_parity(oracle_mod, monkeypatch, patch, form):
    for k, v in FORMS[form].items():
        monkeypatch.setenv(k, v)
    k, _ = check_parity(oracle_mod, _lshape(patch), 12, threads=16)
    k.close()


@pytest.mark.parametrize("patch,pml,n", [(75.0, 40, (53, 45)), (100.0, 70, (301, 187)), (100.0, 70, (700, 130))])
def test_wide_window_every_variant(oracle_mod, monkeypatch, patch, pml, n):
    """Every variant of every length present, pinned: parity, or refused."""
    from openpstd_gb300 import _lib
    from openpstd_gb300.kernel import PSTDKernel
    conf = _windowed(patch, n, pml)
    monkeypatch.setenv("PSTD_AUTOTUNE", "0")
    k = PSTDKernel()
    k.initialize_kernel(conf)
    lengths = sorted({x for i in range(k.domain_count()) for x in k.domain_info(i)["fft_length"] if x})
    k.close()
    ran = 0
    for L in lengths:
        buf, nv = ctypes.create_string_buffer(1 << 14), ctypes.c_int32()
        assert _lib.lib().pstd_stage_variants(L, buf, 1 << 14, ctypes.byref(nv)) == 0
        for i in range(nv.value):
            monkeypatch.setenv("PSTD_PLAN", f"{L}:{i}")
            try:
                k, _ = check_parity(oracle_mod, conf, 10, threads=16)
            except _lib.PSTDError as e:
                assert e.code == _lib.PSTD_ERR_UNSUPPORTED
                continue
            k.close()
            ran += 1
    assert ran > 10


def test_wide_window_noalloc_equals_create(monkeypatch):
    """pstd_solve_noalloc takes the same variants as pstd_create under PSTD_VARIANT=0."""
    import torch
    from openpstd_gb300 import _lib
    from openpstd_gb300.config import CConfig
    from openpstd_gb300.kernel import PSTDKernel
    conf = _windowed(100.0, (151, 97))
    conf.Receivers = [(15.05, 10.05, 0.0), (12.05, 10.05, 0.0)]
    monkeypatch.setenv("PSTD_VARIANT", "0")
    k = PSTDKernel()
    k.initialize_kernel(conf)
    k.advance(10)
    want, rec = k.snapshot(0, "p0"), k.receivers()
    cc = CConfig(conf)
    frame = torch.zeros(want.size, device="cuda")
    samples = torch.zeros(rec.size, device="cuda")
    _lib.check(_lib.lib().pstd_solve_noalloc(ctypes.byref(cc.c), 10, ctypes.c_void_p(frame.data_ptr()), frame.numel(),
                                             ctypes.c_void_p(samples.data_ptr()), samples.numel(), None))
    torch.cuda.synchronize()
    assert np.any(rec)
    assert rel(frame.cpu().numpy(), want.ravel()) <= 1e-5 and rel(samples.cpu().numpy(), rec.ravel()) <= 1e-5


@pytest.mark.parametrize("form", ["per_length", "merged", "lengths"])
def test_wide_windows_served(monkeypatch, form):
    """Scenes of different windows in one server equal their solo runs."""
    from openpstd_gb300 import scenes
    from openpstd_gb300.serving import Server
    from test_serving import _form_env, _solo
    _form_env(monkeypatch, form)
    # (per_length takes one variant for all strips of a length: both scenes wide there, as in the solo runs)
    other = _lshape(120.0, steps=30) if form == "per_length" else scenes.l_shape(1, scale=0.2, steps=30, pml=70)
    confs = [other, _lshape(100.0, steps=30)]
    with Server(256 << 20, max_scenes=4) as srv:
        first = srv.submit(confs[0], 14, final_frame=True)
        srv.tick(8)
        ids = [first, srv.submit(confs[1], 10, final_frame=True)]
        srv.run_until_idle(8)
        got = [srv.result(i) for i in ids]
    for (rec, frame), conf, n in zip(got, confs, (14, 10)):
        want_rec, want_frame = _solo(conf, n)
        assert rel(rec, want_rec) <= 1e-6 and rel(frame, want_frame) <= 1e-6


@pytest.mark.parametrize("form", ["untuned", "tuned", "chain2"])
@pytest.mark.parametrize("patch,cells", [(60.0, 26), (65.0, 28)])
def test_narrow_window_parity(oracle_mod, monkeypatch, patch, cells, form):
    """Windows below 32 cells: length 128 with strips the Toeplitz forms do not take."""
    from openpstd_gb300 import scenes
    conf = scenes.l_shape(2, scale=0.25, steps=12)
    conf.Settings.SetPatchError(patch)
    assert conf.Settings.GetWindowSize() == cells
    for k, v in FORMS[form].items():
        monkeypatch.setenv(k, v)
    k, _ = check_parity(oracle_mod, conf, 12, threads=16)
    k.close()
