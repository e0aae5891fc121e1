"""A kernel that is set up while its producer still runs reads the producer's
buffers with ordinary loads.  The non-coherent load (__ldg, const __restrict__)
promises data that stays as it is for the kernel's whole life, so it is left to
tables that are written when their handle is created."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "megastation_b200" / "csrc"

# what an __ldg may read: twiddles, pilot signs, descrambling bytes (spu points into p.seqb), the code's B^-1
TABLES = re.compile(r"(p\.tw|p\.pilot|p\.seqb|spu|h\.inv)\b")


def sources():
    files = sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])
    assert len(files) > 20
    return [(f.name, re.sub(r"//[^\n]*", "", f.read_text())) for f in files]


def test_non_coherent_loads_only_from_tables():
    found = 0
    for name, text in sources():
        for m in re.finditer(r"__ldg\(\s*", text):
            found += 1
            assert TABLES.match(text, m.end()), f"{name}: __ldg of {text[m.end():m.end() + 40]!r}"
    assert found


def test_no_other_non_coherent_loads():
    for name, text in sources():
        assert not re.search(r"__restrict__|ld\.global(\.\w+)*\.nc", text), name


def test_dependent_kernels_wait_before_anything_else():
    """Every kernel handed to pdl_launch() calls pdl_wait() before its first use of a pointer: it stands
    among the declarations at the head of the body."""
    texts = sources()
    heads = {}
    for _, text in texts:
        for m in re.finditer(r"__global__\s+void(?:\s+__launch_bounds__\([^)]*\))?\s+(\w+)\s*\([^{;]*\)\s*\{", text):
            heads[m.group(1)] = text[m.end():text.index("\n}", m.end())]
    waiting = {k for k, v in heads.items() if "pdl_wait();" in v}
    for k in waiting:
        before = heads[k].split("pdl_wait();")[0]
        for line in filter(None, (x.strip() for x in before.split(";"))):
            assert re.match(r"(extern\s+)?__shared__|constexpr|using|static_assert|namespace", line), f"{k}: {line!r}"
    launched = set()
    for _, text in texts:
        for m in re.finditer(r"pdl_launch\(", text):
            launched |= {w for w in re.findall(r"\b(\w+_kernel)\b", text[m.end():m.end() + 160])}
    assert len(launched) > 10 and launched <= waiting, launched - waiting
