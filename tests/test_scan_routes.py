"""Which launches a recurrence takes (csrc/scan_routes.h), against what was measured: every line was at least a tenth faster that way than the next
(B200, 148 SMs; the best in us, and the others)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ONES = {n: [(1, n)] for n in (1, 15, 63)}
MEASURED = [
    ("scan", 8192, [(2048, 1)], "stream"),                 # 177; chunks 228, tile 433
    ("scan", 8192, [(300, 1)], "stream"),                  # 28; chunks 44
    ("scan", 8192, [(1000, 3)], "stream"),                 # 262; chunks 311
    ("scan", 4096, [(300, 1)], "stream"),                  # 19; chunks 32
    ("scan", 4096, [(1000, 1)], "stream"),                 # 55; chunks 63
    ("scan", 4096, [(300, 4)], "stream"),                  # 55; chunks 78
    ("scan", 2048, [(300, 4)], "stream"),                  # 28; chunks 43
    ("scan", 4096, [(2000, 4)], "stream"),                 # 348; tile 472
    ("scan", 10240, [(100, 1)], "stream"),                 # 21; chunks 34
    ("scan", 10240, [(2048, 1)], "chunks"),                # 285; stream 351: two rounds of CTAs
    ("scan", 10240, [(1000, 1)], "chunks"),                # 141; stream 175
    ("scan", 12288, [(4000, 1)], "chunks"),                # 617; stream 678
    ("scan", 3072, [(4000, 1)], "chunks"),                 # 177; stream about 210
    ("scan", 2048, [(2048, 1)], "chunks"),                 # 64; stream 111
    ("scan", 2048, ONES[15] + [(2048, 1)], "chunks"),      # 67; stream 181, apart 118
    ("scan", 2048, [(65, 10), (2000, 1)], "chunks"),       # 75; stream 188
    ("scan", 4096, ONES[15] + [(300, 1)], "apart"),        # 24; chunks 37, stream 39
    ("scan", 4096, ONES[63] + [(300, 1)], "apart"),        # 33; chunks 63, stream 76
    ("scan", 8192, ONES[63] + [(300, 1)], "apart"),        # 54; chunks 109, stream 129
    ("scan", 8192, ONES[63] + [(2048, 1)], "apart"),       # 208; chunks 289, stream 292
    ("scan", 8192, [(40, 8), (500, 1)], "apart"),          # 73; chunks 97, stream 83
    ("scan", 8192, [(1000, 8)], "tile"),                   # 506; stream 617
    ("scan", 8192, [(300, 8)], "tile"),                    # 156; stream 197
    ("scan", 2048, [(70, 63)], "tile"),                    # 70; stream 115
    ("scan", 4096, [(100, 16)], "tile"),                   # 55; stream 73
    ("scan", 8192, [(100, 16)], "tile"),                   # 97; stream 147
    ("scan", 4096, [(45, 1)], "tile"),                     # 10; chunks 18
    ("scan", 8192, ONES[63] + [(64, 1)], "tile"),          # 41; chunks 93
    ("scan", 2048, [(64, 16)], "tile"),                    # 27; chunks 44
    ("gated", 4096, [(45, 1)], "tile"),                    # 13; chunks 18
    ("gated", 4096, [(4000, 1)], "stream"),                # 107; chunks 162
    ("gated", 4096, [(300, 1)], "stream"),                 # 15; chunks 29
    ("gated", 8192, [(2048, 1)], "stream"),                # 111; chunks 179
    ("gated", 2048, [(300, 4)], "stream"),                 # 29; chunks 38
    ("gated", 8192, [(1000, 8)], "stream"),                # 425; tile 510
    ("gated", 1024, [(2048, 1)], "chunks"),                # 30; stream 56
    ("gated", 2048, ONES[63] + [(2048, 1)], "chunks"),     # 54; stream 150, apart 63
    ("gated", 4096, ONES[15] + [(300, 1)], "apart"),       # 18; chunks 29, tile 77
    ("gated", 4096, ONES[63] + [(300, 1)], "apart"),       # 22; chunks 32, tile 77
    ("gated", 8192, ONES[63] + [(2048, 1)], "apart"),      # 125; chunks 194
    ("gated", 8192, [(300, 16)], "tile"),                  # 242; stream 342
    ("gated", 4096, [(100, 16)], "tile"),                  # 56; stream 97
    ("gated", 8192, [(100, 16)], "tile"),                  # 84; stream 188
]


def chunk_tokens(lens, threads, sms=148, per_sm=1024):
    """Tokens of a chunk as the planner of steps has it: as few chunks as fill the GPU."""
    tokens, chunks = sum(n * c for n, c in lens), max(1, sms * per_sm // threads)
    even = max(32, (-(-tokens // chunks) + 15) // 16 * 16)
    for length in range(even, 2 * even, max(16, even // 256 * 16)):
        if sum(-(-n // length) * c for n, c in lens if n > 32) <= chunks:
            return length
    return even


@pytest.fixture(scope="module")
def ways(tmp_path_factory):
    """[(kind, channels, states, chunk, [(tokens, sequences), ...])] -> what such steps do."""
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("routes") / "routes")
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-fsanitize=address,undefined", "-I", os.path.join(ROOT, "inference-agent_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "scan_routes.cpp"), "-o", exe], check=True, timeout=120)

    def of(steps):
        lines = "".join(f"{kind} {channels} {states} 148 {chunk} " + " ".join(f"{n} {count}" for n, count in lens) + "\n" for kind, channels, states, chunk, lens in steps)
        return subprocess.run([exe], input=lines, capture_output=True, text=True, check=True, timeout=60).stdout.split()
    return of


def test_ways_that_were_measured(ways):
    got = ways([(kind, channels, 16 if kind == "scan" else 1, chunk_tokens(lens, channels * (2 if kind == "scan" else 1)), lens) for kind, channels, lens, _ in MEASURED])
    assert [(m[:3], m[3], g) for m, g in zip(MEASURED, got) if m[3] != g] == [] and len(got) == len(MEASURED)


def test_shapes_of_the_comparison_of_bits(ways):
    """test_gpu_scan_bits.py compares chunks with streams."""
    import test_gpu_scan_bits as B
    for kind, shapes in (("scan", [(c, B.lib().ingot_scan_state_pad(n), m) for c, n, m in B.SCANS]), ("gated", [(c, 1, m) for c, _, m in B.UNITS])):
        steps = [(kind, c, states, chunk, [(n, m)]) for c, states, copies in shapes for n, chunk in B.CUTS for m in (1, copies)]
        got = ways(steps)
        wrong = [(s, g) for s, g, want in zip(steps, got, ["chunks", "stream"] * len(steps)) if g != want and (g, want, s[3]) != ("tile", "chunks", 260)]
        assert wrong == [], wrong
