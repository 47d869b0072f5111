"""CPU test of the steps that SLRIter's level schedule runs in
(muontomography_gb300/csrc/slr_levels.h, slr_steps): every level in order, cut at a
number of muons and at a number of pairs, also where the pairs' offsets are beyond
2^32 (the device numbers a step's pairs in 32 bits from the step's first one)."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
HEADER = ROOT / "muontomography_gb300" / "csrc" / "slr_levels.h"

HARNESS = r"""
#include <cstdio>
#include <vector>
#include "slr_levels.h"
int main() {
    unsigned levels = 0, muons = 0;
    unsigned long long pairs = 0, nt = 0;
    if (std::scanf("%u %llu %u %llu", &levels, &nt, &muons, &pairs) != 4) return 2;
    std::vector<uint32_t> start(levels + 2), sstart;
    std::vector<uint64_t> fo(nt + 1);
    std::vector<uint8_t> place;
    for (auto& s : start) { unsigned x; if (std::scanf("%u", &x) != 1) return 2; s = x; }
    for (auto& o : fo) { unsigned long long x; if (std::scanf("%llu", &x) != 1) return 2; o = x; }
    const uint32_t n = muto::slr_steps(start, levels, fo.data(), muons, pairs, sstart, place);
    std::printf("%u\n", n);
    for (auto s : sstart) std::printf("%u\n", s);
    for (auto p : place) std::printf("%u\n", static_cast<unsigned>(p));
    return 0;
}
"""


@pytest.fixture(scope="module")
def steps_exe(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("slr_steps")
    (d / "main.cpp").write_text(HARNESS)
    exe = d / "steps"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{HEADER.parent}", str(d / "main.cpp"), "-o", str(exe)], check=True)
    return exe


# (muons of each level, pairs of a muon, most muons, most pairs); the third holds 2^33
# pairs in paths of 2^27, the fourth paths longer than a step's pairs
@pytest.mark.parametrize("per_level,longest,muons,pairs", [
    ([1, 24, 25, 48, 49, 3, 1], 40, 24, 1 << 31),
    ([7] * 30, 40, 24, 100),
    ([20, 44], 1 << 27, 24, 1 << 31),
    ([5, 9], 64, 24, 32),
    ([300], 0, 24, 1 << 31)])
def test_steps(steps_exe, per_level, longest, muons, pairs):
    rng = np.random.default_rng(len(per_level))
    nt, levels = sum(per_level), len(per_level)
    n = np.full(nt, longest) if longest > 1000 else rng.integers(0, longest + 1, nt)
    start = np.concatenate([[0], np.cumsum([0] + per_level)])
    fo = np.concatenate([[0], np.cumsum(n)])
    text = f"{levels} {nt} {muons} {pairs}\n" + " ".join(map(str, start)) + "\n" + " ".join(map(str, fo)) + "\n"
    out = [int(x) for x in subprocess.run([str(steps_exe)], input=text, capture_output=True, text=True,
                                          check=True).stdout.split()]
    steps = out[0]
    sstart, place = np.array(out[1:steps + 2]), np.array(out[steps + 2:])
    assert len(place) == nt and sstart[0] == 0 and sstart[-1] == nt and (np.diff(sstart) > 0).all()
    assert set(start[1:]) <= set(sstart)  # a step holds muons of one level alone
    for a, b in zip(sstart[:-1], sstart[1:]):
        assert b - a <= muons and (b - a == 1 or fo[b] - fo[a] <= pairs)
        assert (place[a:b] == np.arange(b - a)).all()
        # as long as it may be
        assert b in start or b - a == muons or fo[b + 1] - fo[a] > pairs
