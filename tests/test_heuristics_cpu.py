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


def test_short_segment_plans(tmp_path):
    """prefill_segments_short for 1 to 64 chains of up to 640 chunks, without and with a limit of scratch: no sequence ends in an empty segment (the
    transition kernel takes all but the last for full ones), segments have 5 chunks or more, their CTAs find room side by side, the scratch is kept to, and packed plans
    have slots for any split of the chunks over the sequences."""
    out = run(tmp_path, '''
        long long cut = 0;
        for (int seqs = 1; seqs <= 64; ++seqs)
            for (int vh : {1, 2, 3, 4, 7, 8, 16, 32, 48, 49, 64})
                for (int chunks = 0; chunks <= 640; ++chunks)
                    for (bool packed : {false, true})
                        for (long long limit : {plan_detail::kNoLimit, 0ll, 5ll * vh, 40ll}) {
                            if (seqs * vh > 64) continue;
                            const long long total = packed && chunks ? chunks * (long long)seqs - seqs / 2 : chunks * (long long)seqs;
                            const SegmentPlan p = prefill_segments_short(seqs, vh, chunks, total, packed, limit);
                            if (p.num_segments == 1) continue;
                            ++cut;
                            const long long slots = packed ? total / p.seg_chunks + seqs : seqs * (long long)p.num_segments;
                            const bool ok = p.first_apart == 1 && p.seg_chunks >= 5 && (long long)(p.num_segments - 1) * p.seg_chunks < chunks &&
                                            (long long)p.num_segments * p.seg_chunks >= chunks && p.slots == slots && slots * vh <= limit &&
                                            (packed || (slots - seqs) * vh <= 148) && seqs * vh <= kManyChains;
                            if (!ok) std::printf("%d x %d, %d chunks, packed %d, limit %lld: %d segments of %d, %d slots\\n", seqs, vh, chunks, packed, limit, p.num_segments, p.seg_chunks, p.slots);
                        }
        // slots of a packed plan: any lengths whose chunks add up
        unsigned x = 1;
        for (int i = 0; i < 200000; ++i) {
            int n[48], seqs = 1 + (x = x * 1664525u + 1013904223u) % 48;
            long long total = 0;
            for (int s = 0; s < seqs; ++s) total += n[s] = ((x = x * 1664525u + 1013904223u) >> 8) % ((x & 64) ? 2000 : 20);
            const SegmentPlan p = prefill_segments_short(seqs, 1, (total + seqs - 1) / seqs, total, true);
            if (p.num_segments == 1) continue;
            long long used = 0;
            for (int s = 0; s < seqs; ++s) used += n[s] ? (n[s] + p.seg_chunks - 1) / p.seg_chunks : 1;
            if (used > p.slots) std::printf("%lld of %d slots used\\n", used, p.slots);
        }
        std::printf("%s\\n", cut > 100000 ? "done" : "hardly any plan cuts");
    ''')
    assert out == ["done"], out[:10]


def test_groups_of_token_block_rows(tmp_path):
    """block_groups at the measured shapes: tiles of 16 rows, 148 SMs"""
    out = run(tmp_path, '''
        for (long long tiles : {256, 512, 384, 1024, 64, 192, 576, 2048}) std::printf("%d ", block_groups(tiles, 148));
    ''')
    # d=256, 8 v-heads B=2, 4, 3, 8, 4 v-heads B=1; d=192 8 v-heads B=2, 6; 16 packed sequences, d=256
    assert out[0].split() == ["2", "2", "1", "1", "1", "2", "2", "2"]
