"""Library entries through the generated extension module against the same entries through ctypes (host-only entries: no GPU)."""
import ctypes as C

import pytest

from llmss_b200.ops import _lib, calls


@pytest.fixture(scope="module")
def both():
    lib = _lib.load()
    sigs = {**_lib._SIGS, **_lib._OPTIONAL}
    if not calls.module_path(_lib.lib_path().parent, sigs).exists():
        pytest.skip("built without a C compiler")
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
    ("llmss_linear_scan_chunked_floats", (1 << 30, 7, 64, 128, 128)), ("llmss_delta_scan_chunked_bytes", (-1, 3, 4)),
    ("llmss_moe_tile", ())])
def test_same_results(both, name, args):
    lib, plain = both
    if name == "llmss_moe_tile":          # results through addresses
        got = []
        for side in (lib, plain):
            d, g, t = C.c_float(), C.c_float(), C.c_int()
            assert side.llmss_moe_forms(788, 4, 16, 2048, 1024, 1024, C.addressof(d), C.addressof(g), C.addressof(t)) == 0
            got.append((d.value, g.value, t.value))
        assert got[0] == got[1]
        return
    assert getattr(lib, name)(*args) == getattr(plain, name)(*args)


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
