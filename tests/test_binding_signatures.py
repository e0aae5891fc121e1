"""The Python binding passes device pointers and streams as plain integers, so
every library function it calls must have declared argument types (an
undeclared one would take them as 32-bit ints)."""
import ctypes
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _header_prototypes():
    text = open(os.path.join(ROOT, "include", "megastation_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return {m[2]: (m[1], m[3]) for m in re.finditer(r"\b(mb_status|uint32_t|const char \*)\s*(mb_\w+)\(([^)]*)\);", text)}


def test_every_called_function_declares_its_arguments():
    from megastation_b200._lib import LIB
    used = set()
    for f in glob.glob(os.path.join(ROOT, "megastation_b200", "*.py")):
        used |= set(re.findall(r"LIB\.(mb_\w+)", open(f).read()))
    assert len(used) > 40
    for name in sorted(used):
        assert getattr(LIB, name).argtypes is not None, name


def test_declared_arguments_match_the_header():
    from megastation_b200._lib import LIB
    for name, (_, args) in _header_prototypes().items():
        decl = getattr(LIB, name).argtypes
        if decl is None:
            continue
        args = [a.strip() for a in args.split(",") if a.strip() and a.strip() != "void"]
        assert len(args) == len(decl), name
        for a, t in zip(args, decl):
            pointer = "*" in a or "[" in a
            is_ptr = t in (ctypes.c_void_p, ctypes.c_char_p) or hasattr(t, "contents")
            assert pointer == is_ptr, (name, a, t)
            if "uint64_t" in a and not pointer:
                assert t is ctypes.c_uint64, (name, a)
            if a.startswith("float ") and not pointer:
                assert t is ctypes.c_float, (name, a)
