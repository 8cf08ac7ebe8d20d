"""Rules of the job plan, on the CPU: what the host builds for a scene before
any launch (tests/cxx/plan_probe.cpp, compiled against the library)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
JK_COPY = 4


@pytest.fixture(scope="module")
def probe(pstd_lib, tmp_path_factory):
    from openpstd_gb300 import build
    so = str(tmp_path_factory.mktemp("cxx") / "plan_probe.so")
    libdir = os.path.join(ROOT, "openpstd_gb300")
    subprocess.check_call([build.NVCC, "-std=c++17", "-O1", "-shared", "-Xcompiler", "-fPIC", "-o", so,
                           os.path.join(ROOT, "tests", "cxx", "plan_probe.cpp"), "-I" + os.path.join(ROOT, "include"),
                           "-L" + libdir, "-lpstd_gb300", "-Xlinker", "-rpath=" + libdir])
    return ctypes.CDLL(so)


def _copying(steps=60, lr=("left",), n=(90, 73), shift=0):
    """A domain with locally-reacting edges, or (shift) two domains that share
    part of an edge: PML domains one of whose axes is not updated."""
    from openpstd_gb300 import scenes
    from openpstd_gb300.config import DomainConfEdge, PSTDConfiguration
    conf = PSTDConfiguration()
    scenes.base_settings(conf, steps, dx=0.2, pml=50)
    e = dict(left=0.6, right=0.4, top=0.8, bottom=0.5)
    rects = [(0, 0, *n)] + ([(n[0], shift, 61, n[1])] if shift else [])
    conf.Domains = [scenes._domain(*r, 0.2, e) for r in rects]
    for d in conf.Domains:
        for side in lr:
            name = side[0].upper()
            setattr(d, name, DomainConfEdge(getattr(d, name).Absorption, True))
    conf.Speakers = [((r[0] + r[2] / 2 + 0.25) * 0.2, (r[1] + r[3] / 2 + 0.25) * 0.2, 0.0) for r in rects]
    conf.Receivers = [((r[0] + 20.25) * 0.2, (r[1] + 20.25) * 0.2, 0.0) for r in rects]
    return conf


def test_window_of_every_patch_error(pstd_lib, oracle_mod):
    """The window is the same in the kernel, the oracle and the Python
    configuration, whatever machine the library is compiled for."""
    from openpstd_gb300 import _lib, scenes
    from openpstd_gb300.config import CConfig, PSTDConfiguration, c_domain_info
    for patch in range(30, 131):
        conf = PSTDConfiguration()
        scenes.base_settings(conf, 4, dx=0.2, pml=101)
        conf.Settings.SetPatchError(float(patch))
        conf.Domains = [scenes._domain(0, 0, 411, 411, 0.2, dict(left=0.6, right=0.4, top=0.8, bottom=0.5))]
        conf.Speakers = conf.Receivers = []
        cc, h, d = CConfig(conf), ctypes.c_void_p(), c_domain_info()
        _lib.check(pstd_lib.pstd_scene_build(ctypes.byref(cc.c), ctypes.byref(h)))
        try:
            _lib.check(pstd_lib.pstd_scene_domain_info(h, 0, ctypes.byref(d)))
        finally:
            pstd_lib.pstd_destroy(h)
        # kernel/KernelInterface.cpp:128-134 in exact arithmetic: halves round away from zero
        cells = 2 * ((7 * patch - 170 + 10) // 20)
        assert d.window[0] == conf.Settings.GetWindowSize() == oracle_mod.window_size(patch) == cells, patch


def _records(probe, conf, slot):
    from openpstd_gb300.config import CConfig
    cc = CConfig(conf)
    out = np.zeros((1 << 14, 3), dtype=np.int32)
    n = probe.probe_served_records(ctypes.byref(cc.c), slot, out.ctypes.data_as(ctypes.c_void_p), len(out))
    assert 0 < n <= len(out)
    return out[:n]


@pytest.mark.parametrize("conf", [dict(lr=("left",)), dict(lr=("left", "right")), dict(lr=(), shift=21)])
def test_served_records_carry_their_scene(probe, conf):
    """Every record of a served scene, copy jobs included, names the scene's
    slot: the serving loop skips a job by that scene's step count."""
    r = _records(probe, _copying(**conf), slot=5)
    assert np.any(r[:, 0] & JK_COPY)
    assert np.all(r[:, 1] == 5), r[r[:, 1] != 5]


def _plan(probe, conf):
    """[(L, wmin, wmax, first variant, [variant of PSTD_VARIANT=i], [tuned variants])] of a scene's lengths."""
    from openpstd_gb300.config import CConfig
    cc, buf = CConfig(conf), ctypes.create_string_buffer(1 << 17)
    rc = probe.probe_plan(ctypes.byref(cc.c), buf, len(buf))
    if rc:
        return rc, buf.value.decode()
    out = []
    for line in buf.value.decode().splitlines():
        key, rest = line.split(" ", 1)
        if key == "bucket":
            out.append([int(v) for v in rest.split()] + [None, [], []])
        elif key == "first":
            out[-1][3] = rest
        elif key == "forced":
            out[-1][4].append(rest.split(" ", 1)[1])
        else:
            out[-1][5].append(rest)
    return 0, out


def _windowed(patch, n=(301, 187), pml=70):
    """One domain, its strips and those of its PML domains in windows of the patch error's width."""
    from openpstd_gb300 import scenes
    from openpstd_gb300.config import PSTDConfiguration
    conf = PSTDConfiguration()
    scenes.base_settings(conf, 10, dx=0.2, pml=pml)
    conf.Settings.SetPatchError(patch)
    conf.Domains = [scenes._domain(0, 0, *n, 0.2, dict(left=0.6, right=0.4, top=0.8, bottom=0.5))]
    conf.Speakers = [(n[0] * 0.1, n[1] * 0.1, 0.0)]
    conf.Receivers = []
    return conf


# the forms that keep a strip's bands in slots of 32 floats a side
NARROW = (" fused c", " tma", " pipe")


def _narrow(name):
    return any(t in name for t in NARROW) and " quad" not in name


@pytest.mark.parametrize("patch,w,pml,n", [(72.0, 34, 40, (41, 50)), (75.0, 36, 50, (301, 187)), (100.0, 54, 70, (301, 187)),
                                           (100.0, 54, 70, (700, 1200)), (120.0, 68, 70, (2600, 5000))])
def test_wide_windows_get_no_narrow_form(probe, patch, w, pml, n):
    """A bucket with a window above 32 cells neither starts from, is forced to
    nor tunes a form whose band slots hold 32; the other buckets keep theirs."""
    rc, plan = _plan(probe, _windowed(patch, n, pml))
    assert rc == 0, plan
    assert max(b[2] for b in plan) == w
    for L, wmin, wmax, first, forced, tuned in plan:
        assert tuned and 0 < wmin <= wmax
        if wmax > 32:
            assert not [v for v in [first] + forced + tuned if _narrow(v)], (L, wmax)
        elif L >= 128:
            assert _narrow(first) and any(_narrow(v) for v in tuned)


def test_windows_up_to_32_start_from_variant_0(probe):
    import re
    from openpstd_gb300 import _lib
    seen = set()
    for n, pml in [((13, 14), 10), ((21, 25), 20), ((50, 90), 50), ((181, 333), 50), ((611, 1203), 50), ((2003, 4101), 50)]:
        rc, plan = _plan(probe, _windowed(70.0, n, pml))
        assert rc == 0, plan
        for L, _wmin, _wmax, first, forced, tuned in plan:
            buf, k = ctypes.create_string_buffer(1 << 14), ctypes.c_int32()
            assert _lib.lib().pstd_stage_variants(L, buf, 1 << 14, ctypes.byref(k)) == 0
            names = [line.split(" ", 1)[1] for line in buf.value.decode().splitlines()]
            assert first == names[0] and first in tuned
            fp32 = [v for v in names if not re.search(r"bf16x3|r16.16.16.2 tcgen05", v)]
            assert len(forced) == k.value and set(tuned) <= set(fp32)
            seen.add(L)
    assert seen == {32, 64, 128, 256, 512, 1024, 2048, 4096, 8192}


def test_pinned_plan_refused_where_the_window_is_too_wide(probe, monkeypatch):
    from openpstd_gb300 import _lib
    monkeypatch.setenv("PSTD_PLAN", "512:0")
    assert _plan(probe, _windowed(70.0))[0] == 0
    rc, msg = _plan(probe, _windowed(100.0))
    assert rc == _lib.PSTD_ERR_UNSUPPORTED and "does not take windows" in msg


@pytest.mark.parametrize("patch,w,n", [(60.0, 26, (50, 50)), (70.0, 32, (50, 50)), (75.0, 36, (50, 50)), (65.0, 28, (63, 90))])
def test_toeplitz_forms_for_their_own_window_only(probe, patch, w, n):
    """The tcgen05 Toeplitz forms compute a fixed tile of 32-cell windows; a
    bucket of length 128 with other windows is not offered them."""
    rc, plan = _plan(probe, _windowed(patch, n, pml=50))
    assert rc == 0, plan
    L, wmin, wmax, first, forced, tuned = plan[0]
    assert L == 128 and wmax == w
    has = [v for v in [first] + forced + tuned if "toeplitz" in v]
    assert bool(has) == (wmin == wmax == 32), has


def test_plan_cache_distinguishes_windows(probe):
    """Scenes of equal sizes and transform lengths at different patch errors
    do not share a tuned plan, and one that names a form of too narrow a window
    is not taken."""
    from openpstd_gb300.config import CConfig
    ccs = [CConfig(_windowed(p, (300, 300), pml=50)) for p in (60.0, 70.0, 75.0, 70.2)]
    sig = []
    for cc in ccs:
        buf = ctypes.create_string_buffer(1 << 16)
        n = probe.probe_signature(ctypes.byref(cc.c), buf, len(buf))
        assert 0 < n < len(buf)
        sig.append(buf.value)
    lengths = [[b[0] for b in _plan(probe, _windowed(p, (300, 300), pml=50))[1]] for p in (60.0, 70.0, 75.0)]
    assert lengths[0] == lengths[1] == lengths[2] == [128, 512]
    assert len(set(sig[:3])) == 3
    assert sig[3] == sig[1]               # 70.2 dB: the same 32 cells
    at70, at75 = ctypes.byref(ccs[1].c), ctypes.byref(ccs[2].c)
    assert probe.probe_plan_applies(at70, at70, 0) == 1      # variant 0: the fused form
    assert probe.probe_plan_applies(at70, at75, 0) == 0


def test_length_4096_tunes_every_form_within_the_limit(probe):
    """Every FP32 form of length 4096 may be timed, the four-strip ones (which
    the chained and served forms run) included, but the one whose round-off
    was measured above the limit of the large-scene test."""
    rc, plan = _plan(probe, _windowed(70.0, (2048, 2048), pml=50))
    assert rc == 0, plan
    L, _wmin, _wmax, _first, _forced, tuned = plan[-1]
    assert L == 4096
    assert "L4096 cs4 nt512 r16.16.16" not in tuned
    assert sum(" quad" in v for v in tuned) == 5 and sum(" fused c" in v for v in tuned) == 3
