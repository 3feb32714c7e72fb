"""How a batch is split into one- and two-board tiles, on the CPU: the kernels' own `Tiles` and the host's
`tile_launches`, compiled together.  Every board is in one tile, of one launch, whatever the batch, the option and the
way the length is known; both SMs of a pair have as many tiles; and no launch that has boards is left out."""
import os
import re
import subprocess

import pytest

from conftest import ROOT
from test_tile_schedule import definition

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#define __device__
TILES
RULE
template <int NB> int take(int n, int wave, int grid, int one, std::vector<int>& seen) {
    int boards = 0;
    for (int cta = 0; cta < grid; ++cta) {
        const Tiles<NB> t(n, wave, grid, cta, one), other(n, wave, grid, cta ^ 1, one);
        if (t.count() != other.count()) { std::printf("pair %d of %d: %d, %d tiles\n", cta, n, t.count(), other.count()); std::exit(1); }
        for (int k = 0; k < t.count(); ++k)
            for (int b = 0; b < NB; ++b)
                if (t.at(k) + b < n) { ++seen[t.at(k) + b]; ++boards; }
    }
    return boards;
}
int main(int argc, char** argv) {
    const int wave = std::atoi(argv[1]), one = std::atoi(argv[2]);
    for (int capacity : {1, 2, 3, wave - 1, wave, wave + 1, 2 * wave - 1, 2 * wave, 2 * wave + 1, 3 * wave, 3 * wave + 1, 4 * wave + 7, 9 * wave})
        for (int list = 0; list < 2; ++list)
            for (int n = list ? 0 : capacity; n <= capacity; n += list ? 1 + n / 7 : 1) {
                const TileLaunches made = tile_launches(capacity, wave, one, list);
                std::vector<int> seen(n + 1);
                const int in_twos = take<2>(n, wave, made.twos, one, seen);
                const int in_ones = take<1>(n, wave, made.ones, one, seen);
                for (int i = 0; i < n; ++i)
                    if (seen[i] != 1) { std::printf("board %d of %d (capacity %d): in %d tiles\n", i, n, capacity, seen[i]); return 1; }
                // the option's promise, and the two-board tiles' share
                if (n <= one * wave ? in_twos != 0 : one == 0 && in_ones != 0) { std::printf("%d boards on the wrong tiles\n", n); return 1; }
            }
    return 0;
}
"""


@pytest.mark.parametrize("one", [0, 1, 2, 8])
@pytest.mark.parametrize("wave", [2, 6, 148])
def test_every_board_is_in_one_tile(wave, one, tmp_path):
    text = open(os.path.join(ROOT, "brokefish_b200", "csrc", "bf_encoder_ws.cuh")).read()
    src, exe = tmp_path / "tiles.cpp", tmp_path / "tiles"
    rule = open(os.path.join(ROOT, "brokefish_b200", "csrc", "bf_encoder.cu")).read()
    rule = definition(rule, "struct TileLaunches") + "\n" + definition(rule, "TileLaunches tile_launches(")
    src.write_text(MAIN.replace("TILES", definition(text, "struct Tiles")).replace("RULE", rule))
    subprocess.run(["g++", "-std=c++17", "-w", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), str(wave), str(one)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_inputs_are_read_by_plain_loads():
    """One-board tiles beside two-board ones read what an earlier grid wrote behind a fence instead of a wait, which
    loads from memory that is taken to be constant are not bound by: only the network's tables are read so."""
    source = lambda name: re.sub(r"//.*", "", open(os.path.join(ROOT, "brokefish_b200", "csrc", name)).read())
    text, rest = source("bf_encoder_ws.cuh"), source("bf_encoder.cu")
    loads = re.findall(r"__ldg\((?:reinterpret_cast<[^>]*>\()?([^;]*?)\)", text)
    assert len(loads) >= 8 and all(re.match(r"p\.tail \+|emb \+|[gb]4 \+", what) for what in loads), loads
    assert re.findall(r"\* (?:emb|g4|b4) = (?:reinterpret_cast<[^>]*>\()?(p\.\w+)", text) == ["p.tail", "p.tail", "p.emb"]
    assert "__restrict__" not in text + definition(rest, "struct Params") + definition(rest, "__device__ __forceinline__ void expand_board(")
    assert "__ldg" not in definition(rest, "__device__ __forceinline__ void expand_board(")
    kernel = definition(text, "__global__ void __launch_bounds__(640, 1) encoder_ws_kernel(")
    assert kernel.index("__threadfence()") < kernel.index("p.leaf_count != nullptr) n_eval")
