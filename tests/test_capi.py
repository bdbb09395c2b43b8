"""The C-ABI library builds for sm_103a, loads, and exports every symbol include/hrt.h declares."""
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared():
    src = open(os.path.join(ROOT, "include", "hrt.h")).read()
    return sorted(set(re.findall(r"^\s*(?:int|void|size_t|int64_t|const char \*)\s*(hrt_\w+)\s*\(", src, re.M)))


def test_header_matches_binding():
    from helios_gb300 import _hrt
    assert declared() == sorted(_hrt.EXPORTS)


def test_library_exports_all(hrt_lib):
    for name in declared():
        assert hasattr(hrt_lib, name), name


def test_backend_name(hrt_lib):
    assert b"GB300" in hrt_lib.hrt_backend_name()


def test_no_cpu_fallback_path():
    """The product package never imports, loads or runs the oracle."""
    pkg = os.path.join(ROOT, "helios_gb300")
    pat = re.compile(r"(import\s+oracle|from\s+oracle|hrt_oracle|libhrt_oracle)")
    for dirpath, _, files in os.walk(pkg):
        for f in files:
            if f.endswith((".py", ".cu", ".cuh", ".h", ".cpp")):
                txt = open(os.path.join(dirpath, f)).read()
                assert not pat.search(txt), f


def test_server_budget_admits_a_scene_of_its_footprint(hrt_lib):
    """A scene's share of the server's memory budget is its records, trees and radiation buffers (529
    bytes a primitive, 68 more per band, and 8 MB); buffers that a solve can do without take no part in it."""
    import numpy as np

    from helios_gb300 import _hrt, scenes

    sc = scenes.mixed_canopy(2000, 2.0, seed=1)
    for short in (0, 1):
        srv = _hrt.Server(device=0, workers=1, hbm_budget=sc.n * (529 + 2 * 68) + (8 << 20) - short)
        srv.add_scene(0, sc.T, sc.ptype, sc.twosided, np.zeros((sc.n, 2)), np.zeros((sc.n, 2)))
        submit = lambda: srv.submit(1, 0, 0.0, [1, 1], (0.0, 0.0, 1.0), [1.0, 1.0], [1.0, 1.0], 4, 4, 0, 1)
        if short:
            with pytest.raises(_hrt.HrtError) as e:
                submit()
            assert e.value.code == _hrt.HRT_ENOMEM
        else:
            submit()
        del srv
