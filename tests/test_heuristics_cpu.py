"""Host-side choices of the launches (csrc/heuristics.hpp), swept over their range with a small C++ program: no GPU needed."""
import os
import subprocess
import textwrap

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "h100_gdn_cuda_b200", "csrc")


def run(tmp_path, body, head="", nvcc=False):
    """Compiles and runs `body` as main(); returns the lines it printed."""
    src = '#include <cstdio>\n#include "heuristics.hpp"\n' + head + "\nusing namespace gdn;\nint main() {\n" + textwrap.dedent(body) + "\n}\n"
    path, exe = str(tmp_path / ("h.cu" if nvcc else "h.cpp")), str(tmp_path / "h")
    with open(path, "w") as f:
        f.write(src)
    if nvcc:
        from h100_gdn_cuda_b200 import build
        cmd = [build.nvcc_path(), "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr"]
    else:
        cmd = ["g++", "-O1"]
    subprocess.check_call(cmd + ["-std=c++17", "-I", CSRC, path, "-o", exe])
    return subprocess.check_output([exe]).decode().splitlines()


def test_parts_of_one_token_units(tmp_path):
    """decode_split over 1 to 600 tiles per unit (dv has no upper limit at the C entry point): the parts divide the tiles, no CTA has two
    of them, what stays whole is whole rounds, and the launch's parameter holds the count (a byte did not: 256 tiles of one unit
    came out as 0 parts, 257 as 1)."""
    out = run(tmp_path, '''
        for (long long slots : {1ll, 2ll * 148, 3ll * 148, 4ll * 148})
            for (int tiles = 1; tiles <= 600; ++tiles)
                for (long long units : {1ll, 2ll, 7ll, 33ll, slots - 1, slots, slots + 1, 2 * slots + 5, 5 * slots + 1})
                    for (bool later : {false, true}) {
                        if (units < 1) continue;
                        const DecodeSplit d = decode_split(units * tiles, tiles, slots, later);
                        RecurrentParams p{};
                        p.split_parts = d.parts;
                        const bool ok = d.parts >= 1 && tiles % d.parts == 0 && d.whole % slots == 0 && d.whole <= units &&
                                        (d.parts == 1 || (units - d.whole) * d.parts <= slots) && p.split_parts == d.parts;
                        if (!ok) std::printf("slots %lld tiles %d units %lld later %d: whole %lld parts %d (%d)\\n", slots, tiles, units, later, d.whole, d.parts, (int)p.split_parts);
                    }
        const DecodeSplit one = decode_split(257, 257, 592, false), two = decode_split(512, 256, 592, false);
        std::printf("%d %d\\n", one.parts, two.parts);
    ''', '#include "kernels/recurrent.cuh"', nvcc=True)
    assert out == ["257 256"], out[:10]
