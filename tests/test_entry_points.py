"""The library's entry points have one list of types: the header, which every translation unit includes, so that a definition that differs does not
compile.  The ctypes table names the same functions with the same types."""
import os
import re

from nsa_optim_b200.ops import build
from nsa_optim_b200.ops.signatures import SIGNATURES

CODES = {"int": "i", "unsigned": "u", "long": "l", "long long": "q", "float": "f", "void": "v"}


def _source(name):
    with open(os.path.join(build.SRC, name)) as f:
        return re.sub(r"/\*.*?\*/|//[^\n]*", "", f.read(), flags=re.S)


def _code(declaration, named=True):
    if "*" in declaration:
        return "s" if not named else "p"
    words = [w for w in declaration.split() if w != "const"]
    words = words[:-1] if named else words
    return "p" if words == ["cudaStream_t"] else CODES[" ".join(words)]


def _prototypes():
    text = "\n".join(line for line in _source("nsa_b200.h").splitlines() if not line.startswith("#"))
    return {m[2]: _code(m[1], False) + "".join(_code(a) for a in m[3].split(",") if a.strip() not in ("", "void"))
            for m in re.finditer(r"([\w\s*]+?)\b(nsa_\w+)\s*\(([^()]*)\)\s*;", text)}


def test_ctypes_table_agrees_with_the_header():
    assert _prototypes() == SIGNATURES


def test_every_translation_unit_includes_the_header():
    assert '#include "nsa_b200.h"' in _source("host.cuh")
    declared = set(_prototypes())
    for name in build.sources():
        text = _source(name)
        assert '#include "host.cuh"' in text, name
        assert set(re.findall(r'extern "C"[\w\s*]+?\b(nsa_\w+)\s*\(', text)) <= declared, name
