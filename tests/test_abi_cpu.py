"""The public header, the definitions and the ctypes signatures of the kernel library name the same arguments, on the CPU."""
import ctypes
import re
from pathlib import Path

import pytest

from llmss_b200.ops import _lib

ROOT = Path(__file__).resolve().parents[1]
SCALARS = {"int": "i32", "int32_t": "i32", "unsigned": "u32", "unsigned int": "u32", "uint32_t": "u32", "int64_t": "i64", "long long": "i64", "size_t": "u64",
           "unsigned long long": "u64", "uint64_t": "u64", "float": "f32", "double": "f64", "void": "void"}
POINTERS = {"llmss_stream_t", "cudaStream_t", "CUstream"}
CTYPES = {ctypes.c_int: "i32", ctypes.c_uint: "u32", ctypes.c_int64: "i64", ctypes.c_size_t: "u64", ctypes.c_ulonglong: "u64", ctypes.c_float: "f32",
          ctypes.c_double: "f64", None: "void"}


def _kind(text, named):
    """Machine type of a parameter (with its name) or a result (without)."""
    text = re.sub(r"\b(const|struct|extern)\b", " ", text).strip()
    if "*" in text or "[" in text:
        return "ptr"
    words = text.split()
    if named and len(words) > 1 and " ".join(words) not in SCALARS:
        words = words[:-1]
    name = " ".join(words)
    return "ptr" if name in POINTERS else SCALARS[name]


def _functions(source, pattern):
    source = re.sub(r"/\*.*?\*/", " ", source, flags=re.S)
    source = re.sub(r"//[^\n]*", " ", source)
    found = {}
    for m in re.finditer(pattern, source):
        params = " ".join(m.group(3).split())
        kinds = [] if params in ("", "void") else [_kind(p, True) for p in params.split(",")]
        found[m.group(2)] = (_kind(m.group(1), False), kinds)
    return found


DECLARED = _functions((ROOT / "include" / "llmss_b200.h").read_text(), r"([\w][\w \*]*?[\s\*])(llmss_\w+)\s*\(([^()]*)\)\s*;")
DEFINED = {}
for _path in sorted((ROOT / "csrc").glob("*.cu")):
    DEFINED.update(_functions(_path.read_text(), r"LLMSS_API\s+([\w][\w \*]*?[\s\*])(llmss_\w+)\s*\(([^()]*)\)\s*\{"))


def test_every_entry_is_declared_and_defined():
    assert len(DECLARED) > 100 and not set(DECLARED) - set(DEFINED)
    assert not set(DEFINED) - set(DECLARED)
    assert not set(_lib._SIGS) - set(DECLARED)


@pytest.mark.parametrize("name", sorted(DECLARED))
def test_arguments_agree(name):
    """A caller who compiles against the header hands over what the definition takes; so does the ctypes binding."""
    assert DECLARED[name] == DEFINED[name]
    if name in _lib._SIGS:
        result, args = _lib._SIGS[name]
        kind = lambda t: CTYPES[t] if t in CTYPES else "ptr"
        assert (kind(result), [kind(t) for t in args]) == DECLARED[name]
