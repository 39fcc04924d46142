"""The tile's samples are read by loads that the compiler may move (no memory clobber), so the order against the
barrier that completes the tile has to come from their addresses. Checked on the sources, since a compiler that
does not use its freedom hides a missing order: every such load's address comes from a TileAddr, and a TileAddr's
base passes through a statement that stays in order with barriers and memory accesses.
"""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "qtrk_b200" / "csrc"


def code(name: str) -> str:
    """A source without its comments."""
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def body(src: str, head: str) -> str:
    """The text between the braces that follow `head`."""
    i = src.index("{", src.index(head))
    depth = 0
    for j in range(i, len(src)):
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        if depth == 0:
            return src[i + 1:j]
    raise AssertionError(head)


def ordered(asm: str) -> bool:
    return "volatile" in asm.split("(")[0] and '"memory"' in asm


def test_the_base_of_every_tile_address_is_ordered():
    src = code("tile.cuh")
    if ordered(re.search(r"asm[^;]*ld\.shared[^;]*;", src).group(0)):
        return                                    # the loads themselves are in order
    ctor = body(src, "TileAddr(const uint32_t *tile, int ts)")
    after = ctor[ctor.index("base ="):]
    asm = re.search(r"asm[^;]*;", after)
    assert asm and ordered(asm.group(0)) and '"+r"(base)' in asm.group(0)


def test_every_sample_takes_its_address_from_a_tile_addr():
    calls = 0
    for name in ("tile.cuh", "adjoint.cu", "localize.cu", "gauss.cu", "zmatch_tc.cu", "com.cu"):
        src = code(name)
        if name == "tile.cuh":                    # the definitions of the loads and of the cells
            start, end = src.index("uint32_t tile_word("), src.index("word_pixel(")
            assert src[start:end].count("smem_addr(") == 1  # TileAddr's own
            src = src[:start] + src[end:]
        assert not re.search(r"\btile_(word|float)\b", src), name
        for first in re.findall(r"\bcells?2?<F>\(([^,]*),", src):
            calls += 1
            if not first.startswith("ta."):       # a variable: its own address
                assert re.search(rf"\b{first}\s*=\s*ta\.at\(", src), (name, first)
        # each function that samples builds its own TileAddr, so behind its caller's last barrier
        assert src.count("ta.at(") == 0 or re.search(r"const TileAddr ta\(img, ts\);", src), name
    assert calls >= 6
