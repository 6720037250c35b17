"""How the fp32 grouped GEMM cuts an expert's rows into tiles, and its widest tiles against the oracle."""
import ctypes
import os
import re
import subprocess

import pytest
import torch

from oracle import experts_oracle as orc

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yamoe_b200", "csrc", "umma_f32.cuh")
GRADS = ["d_hidden", "d_routing", "d_wgu", "d_bgu", "d_wd", "d_bd"]


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


def widths(counts, row_round, M, pairs, tile_rows):
    """Widths of the tiles that the kernel picks for a launch: the choice of s_cost, in Python."""
    rows = [-(-c // row_round) * row_round for c in counts]
    MT = -(-M // (2 * constant("kF32M")))
    best = None
    for i in range(constant("kF32Tiles")):
        tiles = [w for r in rows for w in tiles_of(r, constant("kF32N") - 16 * i, tile_rows)]
        cost = -(-len(tiles) * MT // pairs) * max(12 * max(tiles), constant("kConvClocks"))
        if best is None or cost <= best[0]:
            best = cost, set(tiles)
    return best[1]


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


#: rows per expert; H; a width that has to occur in: gate_up and down (rows rounded to 16), GLU gradient (to 64)
WIDE = {"160": ([145, 152, 159, 160] * 8, 512, 160, 160, 96), "144": ([129, 136, 143, 144] * 8, 512, 144, 144, 96),
        "two of 160": ([257, 300, 319, 320] * 4, 512, 160, 160, 160), "four of 144": ([513, 560, 575, 576] * 2 + [576], 512, 144, 144, 144)}


@pytest.mark.parametrize("name", WIDE)
def test_wide_tiles_are_chosen(name, tile_rows):
    counts, H, gate_up, down, glu_gradient = WIDE[name]
    assert gate_up in widths(counts, 16, 2 * H, 74, tile_rows)
    assert down in widths(counts, 16, H, 74, tile_rows)
    assert glu_gradient in widths(counts, 64, H, 74, tile_rows)


@pytest.mark.gpu
@pytest.mark.parametrize("name", WIDE)
def test_wide_tiles_against_64_bits(name):
    """Tiles of 144 and 160 rows in the forward, data-gradient and recomputing launches: the box of 80 rows, the planes of 10 KB
    and the last accumulator columns.  The bound is that of products of 24 bits (4 * 2^-23 a GEMM; two GEMMs, the
    activation and a gradient: 16 * 2^-23), so that a part taken from a wrong place would show."""
    import yamoe_b200
    counts, H = WIDE[name][:2]
    gen = torch.Generator().manual_seed(len(counts))
    E, T = len(counts), sum(counts)
    ridx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(T, generator=gen)][:, None]

    def normal(*shape, std):
        return torch.randn(*shape, generator=gen) * std

    args = [normal(T, H, std=1.0), ridx, torch.rand(T, 1, generator=gen) + 0.25, normal(E, H, 2 * H, std=H ** -0.5),
            normal(E, 2 * H, std=0.2), normal(E, H, H, std=H ** -0.5), normal(E, H, std=0.2)]
    grad = normal(T, H, std=1.0)
    dev = [a.cuda() for a in args]
    got = [yamoe_b200.experts(*dev, T, E, 1), *yamoe_b200.experts_backward(grad.cuda(), *dev, T, E, 1)]
    ref = [orc.experts_forward_oracle(*args, T, E, 1, compute_dtype=torch.float64),
           *orc.experts_backward_oracle(grad, *args, T, E, 1, compute_dtype=torch.float64)]
    for a, b, n in zip(got, ref, ["out"] + GRADS):
        assert ((a.cpu().double() - b).norm() / b.norm()).item() <= 16 * 2.0 ** -23, n
