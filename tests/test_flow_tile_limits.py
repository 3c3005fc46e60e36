"""Sizes that flow accumulation over tiles takes (csrc/codegen.hpp): the kernels number
rim slots, 256 a tile, in signed 32-bit integers, so a raster is taken only if all its
slots' numbers fit. Compiled from the header and compared with the formula in Python."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "map_b200", "csrc")

SIZES = [(1, 1), (64, 64), (65, 64), (46340, 46340), (8000, 8000), (1, 2 ** 29 - 64), (1, 2 ** 29 - 63), (1, 2 ** 29), (1, 2 ** 31 - 1),
         (2, 2 ** 30 - 1), (3, 2 ** 29 + 5), (2 ** 29, 3), (2 ** 29 - 64, 3), (4, 2 ** 29 - 64), (2 ** 31 - 1, 1), (65, 2 ** 24)]


def test_slots_fit_signed_32_bits(tmp_path):
    src = tmp_path / "limits.cpp"
    src.write_text('#include "codegen.hpp"\n#include <cstdio>\nint main() {\n' + "".join(
        '  std::printf("%%zu %%d\\n", mapb::spread_tiles(%d, %d), (int)mapb::spread_tiles_fit(%d, %d));\n' % (w, h, w, h)
        for w, h in SIZES) + "}\n")
    exe = str(tmp_path / "limits")
    subprocess.run(["g++", "-std=c++17", str(src), "-o", exe, "-I" + CSRC], check=True)
    got = [tuple(map(int, l.split())) for l in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()]
    for (w, h), (tiles, fit) in zip(SIZES, got):
        n = -(-w // 64) * -(-h // 64)
        assert tiles == n, (w, h)
        # the last slot of the last tile, and one past it as the loops' bound
        assert bool(fit) == (n * 256 <= 2 ** 31 - 1), (w, h)


def test_both_callers_ask():
    for name, calls in (("codegen_scan.cpp", 1), ("server.cpp", 1)):
        text = open(os.path.join(CSRC, name)).read()
        assert text.count("spread_tile_type(") - text.count("bool spread_tile_type(") >= calls
        assert "spread_tiles_fit(" in text
