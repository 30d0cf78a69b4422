"""The rule that picks the tiles of the router projection, against the times of both (us, 148 SMs, hidden size 2048)."""
import subprocess

from conftest import ROOT

# narrow tiles, fp32 weights, time with wide tiles, time with narrow tiles
MEASURED = [
    (152, 0, 232.3, 266.6), (256, 0, 235.9, 274.3), (296, 0, 240.0, 277.8), (300, 0, 446.0, 403.6), (384, 0, 449.1, 410.4),
    (444, 0, 452.9, 417.0), (512, 0, 456.6, 523.8), (592, 0, 463.7, 534.2), (600, 0, 666.1, 652.0), (672, 0, 673.3, 659.3),
    (768, 0, 680.1, 772.8), (888, 0, 688.7, 788.7), (1024, 0, 895.5, 914.8),
    (152, 1, 249.7, 262.8), (256, 1, 256.4, 270.3), (296, 1, 260.7, 276.2), (300, 1, 482.8, 395.3), (384, 1, 491.0, 398.8),
    (444, 1, 493.0, 406.4), (512, 1, 498.5, 521.7), (592, 1, 504.5, 528.6), (600, 1, 729.3, 643.8), (672, 1, 730.5, 650.1),
    (768, 1, 737.0, 767.9), (888, 1, 746.2, 784.2), (1024, 1, 976.9, 913.0),
]


def test_the_faster_tiles_are_taken(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include <cstdio>\n#include "router_tiles.hpp"\nint main() { int t, f; while (std::scanf("%d %d", &t, &f) == 2) '
                   'std::printf("%d\\n", (int)ffai::router_wide_tiles(t, 148, f)); }\n')
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "ffai_b200" / "csrc"), str(src), "-o", str(exe)], check=True)
    asked = [(t, f) for t, f, _, _ in MEASURED] + [(148, 0), (148, 1)]
    out = subprocess.run([str(exe)], input="".join(f"{t} {f}\n" for t, f in asked), capture_output=True, text=True, check=True)
    got = [int(v) for v in out.stdout.split()]
    assert got == [int(w < n) for _, _, w, n in MEASURED] + [0, 0]
