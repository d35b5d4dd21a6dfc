"""Library entries through the generated extension module against the same entries through ctypes (host-only entries: no GPU)."""
import ctypes as C

import pytest

from llmss_b200.ops import _lib, build, calls


@pytest.fixture(scope="module")
def both():
    lib = _lib.load()
    sigs = {**_lib._SIGS, **_lib._OPTIONAL}
    if calls.compiler() is None:
        pytest.skip("no C compiler or Python headers")
    assert calls.module_path(_lib.lib_path().parent, sigs).exists()
    plain = C.CDLL(_lib.LOADED_FROM)
    for name, (res, args) in sigs.items():
        fn = getattr(plain, name)
        fn.restype, fn.argtypes = res, args
    return lib, plain


def test_every_plain_entry_is_wrapped(both):
    lib, _ = both
    for name in calls.wrappable({**_lib._SIGS, **_lib._OPTIONAL}):
        assert not isinstance(getattr(lib, name), C._CFuncPtr), name


@pytest.mark.parametrize("name,args", [
    ("llmss_attn_decode_tc_pick_splits", (5, 32, 128, 4000)), ("llmss_attn_decode_scratch_floats", (1 << 20, 64, 256, 16)),
    ("llmss_linear_scan_chunked_floats", (1 << 30, 7, 64, 128, 128)), ("llmss_delta_scan_chunked_bytes", (-1, 3, 4))])
def test_same_results(both, name, args):
    lib, plain = both
    assert getattr(lib, name)(*args) == getattr(plain, name)(*args)


def test_same_results_through_addresses(both):
    got = []
    for side in both:
        d, g, t = C.c_float(), C.c_float(), C.c_int()
        assert side.llmss_moe_forms(788, 4, 16, 2048, 1024, 1024, C.addressof(d), C.addressof(g), C.addressof(t)) == 0
        got.append((d.value, g.value, t.value))
    assert got[0] == got[1]


@pytest.mark.parametrize("args", [(3, 4096, 4096, 1, 2, 0), (3, True, 4096, 1, 2, 0)])
def test_ctypes_objects_take_the_ctypes_function(both, args):
    lib, plain = both
    a, b = _lib.GemmPlan(), _lib.GemmPlan()
    assert lib.llmss_gemm_plan_query(*args, C.byref(a)) == plain.llmss_gemm_plan_query(*args, C.byref(b))
    assert [getattr(a, f) for f, _ in a._fields_] == [getattr(b, f) for f, _ in b._fields_]


def test_errors_as_through_ctypes(both):
    lib, plain = both
    bad = [None, 8, None, 8, None, None, 0, None, 8, 0, 4096, 4096, 0, 0, 0, 0, 0, None, None, None, 0, 0, None, None]       # M = 0
    assert lib.llmss_gemm_ex(*bad) == plain.llmss_gemm_ex(*bad) != 0
    assert "bad shape" in _lib.last_error()
    for args in (bad[:-1], [1.5] + bad[1:], bad[:1] + [8.0] + bad[2:]):
        kinds = []
        for side in (lib, plain):
            with pytest.raises((TypeError, C.ArgumentError)) as e:
                side.llmss_gemm_ex(*args)
            kinds.append(e.type)
        assert kinds[0] is kinds[1]


SIGS = {"llmss_version": (C.c_int, []), "llmss_gemm_set_pair": (C.c_int, [C.c_int])}


@pytest.fixture
def installed(tmp_path, monkeypatch):
    """A folder with a library that is current and no module."""
    monkeypatch.setattr(build, "LIB_DIR", tmp_path / "lib")
    monkeypatch.setattr(build, "OBJ_DIR", tmp_path / "obj")
    monkeypatch.setattr(build, "LIB_PATH", tmp_path / "lib" / "libllmss_b200.so")
    build.LIB_DIR.mkdir()
    build.LIB_PATH.write_bytes(b"")
    (build.LIB_DIR / "build.stamp").write_text(build.tree_digest())
    return build.LIB_DIR


def _tries(monkeypatch, what):
    n = []
    monkeypatch.setattr(build, "_build_locked", lambda *a: n.append(1) or build.LIB_PATH)
    assert what() == build.LIB_PATH
    return len(n)


def test_current_library_without_a_compiler_is_returned_untouched(installed, monkeypatch, capfd):
    monkeypatch.setattr(calls.shutil, "which", lambda name: None)
    assert _tries(monkeypatch, build.build_library) == 0
    assert sorted(f.name for f in installed.iterdir()) == ["build.stamp", "libllmss_b200.so"]
    assert capfd.readouterr() == ("", "")


def test_current_library_in_a_folder_that_takes_no_files(installed, monkeypatch):
    (installed / ".build.lock").mkdir()          # opening it to write raises OSError, as on a read-only file system
    assert _tries(monkeypatch, build.build_library) == 0
    with pytest.raises(OSError):                 # a library that has to be built still needs the folder
        build.build_library(force=True)


@pytest.mark.parametrize("why", ["compile", "folder"])
@pytest.mark.parametrize("stale", [False, True])
def test_a_module_that_cannot_be_built_does_not_stop_the_library(installed, monkeypatch, capfd, why, stale):
    if calls.compiler() is None:
        pytest.skip("no C compiler or Python headers")
    if why == "compile":
        monkeypatch.setattr(calls, "source", lambda sigs: "#error no such entry\n")
    else:
        build.OBJ_DIR.write_text("")             # mkdir raises
    assert _tries(monkeypatch, lambda: build.build_library(force=stale)) == int(stale)
    assert ("no such entry" if why == "compile" else "obj") in capfd.readouterr().err


def test_building_keeps_the_module_of_another_python(tmp_path):
    if calls.compiler() is None:
        pytest.skip("no C compiler or Python headers")
    other, old = tmp_path / "_llmss_calls.0123.cpython-39-other.so", calls.module_path(tmp_path, {})
    other.write_text("")
    old.write_text("")
    assert calls.build(tmp_path, tmp_path, SIGS)
    assert other.exists() and not old.exists() and calls.module_path(tmp_path, SIGS).exists()
    assert calls.attach(C.CDLL(_lib.LOADED_FROM or str(_lib.lib_path())), tmp_path, SIGS) == 1
