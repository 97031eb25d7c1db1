"""The declared argument types of the CUDA library's functions against their C definitions."""
import glob
import os
import re

import pippy_b200
from pippy_b200.ops import _lib

PKG = os.path.dirname(pippy_b200.__file__)


def _c_types():
    kinds = (("*", "p"), ("long long", "l"), ("int", "i"), ("float", "f"))
    table = {}
    for path in glob.glob(os.path.join(PKG, "csrc", "*.cu")):
        for name, args in re.findall(r"^(?:int|void|long long) (pb_\w+)\(([^)]*)\)", open(path).read(), re.M):
            if name in _lib.SIGNATURES:
                table[name] = "".join(next(code for word, code in kinds if word in a) for a in args.split(","))
    return table


def test_signatures_match_the_sources():
    assert _c_types() == _lib.SIGNATURES


def test_plain_numbers_only_go_to_declared_functions():
    """An undeclared function would get the low 32 bits of an address."""
    for path in glob.glob(os.path.join(PKG, "**", "*.py"), recursive=True):
        text = open(path).read()
        for m in re.finditer(r"lib\(\)\.(pb_\w+)\(", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[end], 0)
                end += 1
            call = text[m.end():end]
            if re.search(r"\b(addr|stream_addr|err_addr)\(", call):
                assert m.group(1) in _lib.SIGNATURES, (path, m.group(1))
