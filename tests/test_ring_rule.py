"""Which kernel a decode-only format's matvec takes, on the host (no GPU): the header that the launch code asks, compiled with g++ and asked about
weights whose two kernels were timed, and about the ones that tests/test_gpu_generic_ring.py runs."""
import subprocess
from pathlib import Path

import pytest

from tests import oracle_lib as ol

ROOT = Path(__file__).resolve().parent.parent
SHARE = 148 * 2 * 8  # rows at one a warp, two CTAs of eight warps on each of 148 SMs

# (type, rows, inputs) with the ring: every format that has one; its first row count; shares of four, five, six and seven rows; part-filled last
# rounds of 32 groups, whole units and not; one round and several; the fewest slots
RING = [(ol.Q5_K, 4 * SHARE + 1, 512), (ol.Q8_1, 4 * SHARE + 1, 384), (ol.Q8_K, 4 * SHARE + 1, 1024), (ol.IQ4_XS, 14336, 1536), (ol.Q4_1, 6 * SHARE + 1, 2176), (ol.Q2_K, 6 * SHARE + 1, 3072),
        (ol.Q5_0, 14337, 3072), (ol.Q5_1, 14336, 3584), (ol.IQ4_NL, 15000, 4096), (ol.Q4_1, 4 * SHARE, 4096), (ol.Q5_0, 4 * SHARE, 8192), (ol.Q8_1, 12000, 1152), (ol.Q5_K, 12000, 8192), (ol.Q8_K, 10000, 2048),
        (ol.Q4_1, 14336, 8192), (ol.Q2_K, 14500, 8192), (ol.IQ4_XS, 24000, 512), (ol.Q8_1, 14336, 8192), (ol.Q8_K, 9999, 8192), (ol.Q5_1, 10000, 4608)]
# without: Q3_K; one row too few; rows that are not whole lines; inputs past shared memory; where the ring was measured slower
PLAIN = [(ol.Q3_K, 14336, 4096), (ol.Q5_K, 4 * SHARE, 2048), (ol.Q4_1, 4 * SHARE - 1, 4096), (ol.Q8_K, 14336, 512), (ol.Q4_1, 14336, 2080), (ol.Q8_1, 14336, 8448), (ol.Q4_1, 12000, 2048), (ol.Q4_1, 40000, 1024), (ol.Q5_0, 12000, 2048),
         (ol.IQ4_NL, 9472, 4096), (ol.IQ4_NL, 20000, 4096), (ol.IQ4_XS, 13000, 1024), (ol.Q2_K, 12000, 2048), (ol.Q5_1, 28416, 4096)]


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    exe = tmp_path_factory.mktemp("ring") / "ring_rule_test"
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{ROOT / 'include'}", f"-I{ROOT / 'recipe_dev_b200' / 'csrc'}", str(ROOT / "tests/cpp/ring_rule_test.cpp"), "-o", str(exe)], check=True)

    def run(calls):
        text = "\n".join(" ".join(map(str, c)) for c in calls)
        out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True, timeout=60).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]

    return run


def test_the_measured_side_is_taken(ask):
    for (stages, _, _), call in zip(ask([(t, 148, r, c, 1) for t, r, c in RING]), RING):
        assert 2 <= stages <= 4, call
    for (stages, _, _), call in zip(ask([(t, 148, r, c, 1) for t, r, c in PLAIN]), PLAIN):
        assert stages == 0, call
    assert all(s == 0 for s, _, _ in ask([(t, 148, r, c, n) for t, r, c in RING for n in (2, 5)]))


def test_every_ring_fits_and_copies_whole_lines(ask):
    calls = [(t, sms, r, c, 1) for t in ol.STORED_ONLY for sms in (1, 132, 148) for r in (1, 64, 5000, 9473, 14336, 152064) for c in range(256, 9000, 256 if ol.GEOMETRY[t][0] == 256 else 32)]
    seen = set()
    for (stages, values, size), (t, _, _, c, _) in zip(ask(calls), calls):
        assert (values, size) == ol.GEOMETRY[t]
        if stages:
            seen.add(t)
            chunk = 1024 // values * size
            assert chunk % 16 == 0 and (c // values * size) % 16 == 0 and c <= 8192
            assert (c // 32 * 144 + 127) // 128 * 128 + stages * 8 * 4 * chunk <= 112 * 1024
    assert seen == set(ol.STORED_ONLY) - {ol.Q3_K}
