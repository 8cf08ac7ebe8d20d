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
