"""How the fp32 grouped GEMM cuts an expert's rows into tiles."""
import ctypes
import os
import re
import subprocess

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yamoe_b200", "csrc", "umma_f32.cuh")


def constant(name):
    return int(re.search(r"constexpr int (?:\w+ = \d+, )*%s = (\d+)" % name, open(SOURCE).read()).group(1))


@pytest.fixture(scope="module")
def tile_rows(tmp_path_factory):
    """The kernel's own function, compiled for the host."""
    function = re.search(r"[^\n]* int f32_tile_rows\(.*?\}\n", open(SOURCE).read(), re.S).group(0)
    folder = tmp_path_factory.mktemp("tiles")
    (folder / "tile.cpp").write_text(function + 'extern "C" int tile_rows(int rows, int cnt) { return f32_tile_rows(rows, cnt); }\n')
    subprocess.run(["g++", "-shared", "-fPIC", "-D__device__=", "-D__forceinline__=inline", "-o", str(folder / "tile.so"),
                    str(folder / "tile.cpp")], check=True)
    return ctypes.CDLL(str(folder / "tile.so")).tile_rows


def tiles_of(rows, most, tile_rows):
    """Widths of the tiles of an expert's `rows` (a multiple of 16), none of more than `most` rows."""
    cnt = -(-rows // most)
    return [min(tile_rows(rows, cnt), rows - i * tile_rows(rows, cnt)) for i in range(cnt)]


def test_tiles_cover_an_experts_rows(tile_rows):
    """Whatever the number of rows and the most that a tile may have: no tile is empty or too wide, together they cover
    the rows, and the first one is the widest, which is what the choice of the size reckons with."""
    for row_round in (16, 64):
        for rows in range(row_round, 4000, row_round):
            for i in range(constant("kF32Tiles")):
                most = constant("kF32N") - 16 * i
                tiles = tiles_of(rows, most, tile_rows)
                assert sum(tiles) == rows and min(tiles) > 0 and max(tiles) == tiles[0] <= most
                assert all(t % 16 == 0 for t in tiles)


def test_choice_and_walk_agree_on_the_width():
    """The cost of a candidate and the walk over the tiles take a tile's rows from one function."""
    text = open(SOURCE).read()
    cost = text[text.index("const int cap = kF32N"):text.index("s_cost[warp - 4] =")]
    walk = text[text.index("auto decode = "):text.index("auto give_up = ")]
    assert re.search(r"widest = max\(widest, f32_tile_rows\(rows, cnt\)\)", cost)
    assert re.search(r"step = f32_tile_rows\(rows, cnt\);", walk)
