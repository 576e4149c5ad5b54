"""What can be shown from the kernels' sources without a GPU."""

import re

import pytest

from deterministic_inference_b200.kernels.build import CSRC


def _braced(text: str, at: int) -> tuple:
    """(start, end) of the inside of the first brace at or after ``at``."""
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return start + 1, i
    raise AssertionError("unbalanced braces")


CALL = re.compile(r"(find_rows|load_tile|__syncthreads)\(([^()]*)\);")


def _calls(text: str) -> list:
    """(what, last argument) of the walk's calls in the order of the text."""
    return [(m.group(1), m.group(2).split(",")[-1].strip()) for m in CALL.finditer(text)]


def _walks():
    """The walks over key tiles of the mma.sync attention kernels: the calls in front of the loop, those of a turn that
    has a next tile and those of the last turn."""
    found = []
    for name in ("masked_attention_mma.cuh", "sigmoid_attention_mma.cuh"):
        text = (CSRC / name).read_text()
        for m in re.finditer(r"\n  find_rows\(it_begin\);", text):
            loop = text.index("for (int it = it_begin; it < it_end; ++it)", m.start())
            a, b = _braced(text, loop)
            body = text[a:b]
            when = body.index("if (it + 1 < it_end)")
            c, d = _braced(body, when)
            e, f = _braced(body, d)
            assert body[d + 1:e - 1].strip() == "else"
            found.append((f"{name}:{text.count(chr(10), 0, m.start()) + 2}", _calls(text[m.start():loop]),
                          _calls(body[:when] + body[c:d] + body[f:]), _calls(body[:when] + body[e:f] + body[f:])))
    return found


@pytest.mark.parametrize("where, ahead, turn, last", _walks(), ids=lambda x: x if isinstance(x, str) else "")
def test_row_offsets_of_key_tiles_are_not_written_while_they_are_read(where, ahead, turn, last):
    """The threads that find a tile's rows and those that copy them are other threads: between a write of an entry and
    a read of it, in either order, there is a barrier of the block, and a copy reads the tile that it asks for."""
    for it_begin in (0, 1, 4):
        for tiles in range(1, 7):
            it_end = it_begin + tiles
            steps = [(c, it_begin) for c in ahead]
            for it in range(it_begin, it_end):
                steps += [(c, it) for c in (turn if it + 1 < it_end else last)]
            entry, written, read, copied = {}, set(), set(), []
            for (what, arg), it in steps:
                if what == "__syncthreads":
                    written, read = set(), set()
                    continue
                value = eval(arg, {}, {"it_begin": it_begin, "it": it, "stage": it & 1})
                if what == "find_rows":
                    if value < it_end:
                        assert value & 1 not in read, f"{where}: {tiles} tiles, tile {value} found during a copy"
                        entry[value & 1] = value
                        written.add(value & 1)
                else:
                    assert value not in written, f"{where}: {tiles} tiles, a copy during the search for its rows"
                    read.add(value)
                    copied.append(entry[value])
            assert copied == list(range(it_begin, it_end)), where


def test_the_walks_are_there():
    assert len(_walks()) == 3


WIDTH = {"float2": 8, "uint2": 8, "int2": 8, "float4": 16, "uint4": 16, "int4": 16, "__nv_bfloat162": 4, "half2": 4}
TYPE = {"float": 4, "int": 4, "unsigned": 4, "double": 8, "long long": 8, "unsigned long long": 8, "__nv_bfloat16": 2}


def test_arrays_in_shared_memory_that_are_read_as_vectors_start_on_them():
    """An array in static shared memory is aligned to its elements; one whose elements are read or written several at a
    time says so."""
    declared = re.compile(r"__shared__ ((?:__align__\((\d+)\) )?)((?:unsigned |long )*\w+) ([^;]+);")
    seen = 0
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        text = re.sub(r"extern __shared__[^;]+;", "", path.read_text())
        for m in declared.finditer(text):
            kind = m.group(3).strip()
            align = int(m.group(2) or TYPE.get(kind, 0))
            if not align:
                continue                      # (a struct of its own)
            for name in re.findall(r"(\w+)\s*\[[^,]*", m.group(4)):
                for use in re.finditer(rf"reinterpret_cast<(?:const )?(\w+)\s*\*>\(&?{name}\b", text):
                    seen += 1
                    need = WIDTH.get(use.group(1), 16)
                    assert align % need == 0, f"{path.name}: {name} is read as {use.group(1)}, aligned to {align}"
    assert seen >= 2
