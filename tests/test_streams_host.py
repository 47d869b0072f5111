"""CPU test of the stream pool and of forked work (muontomography_gb300/csrc/streams.h)
against a fake of the CUDA runtime's stream calls: a set goes back to the pool with
every one of its streams waited for, one whose side stream's work failed is destroyed,
the pool stays bounded, a set that cannot be made whole is given up, and a fork that is
left before its join waits for its side streams."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
HEADER = ROOT / "muontomography_gb300" / "csrc" / "streams.h"

FAKE = r"""
#pragma once
#include <set>
#include <vector>
typedef int cudaError_t;
typedef long* cudaStream_t;
typedef long* cudaEvent_t;
enum { cudaSuccess = 0, cudaErrorNotReady = 600, cudaErrorUnknown = 999, cudaStreamNonBlocking = 1, cudaEventDisableTiming = 2 };
struct Fake {
    std::set<long*> live, bad, busy;      // handles alive; streams whose work failed, or still runs
    std::vector<cudaStream_t> synced;     // in order
    int make_until = 1 << 30;             // creations that succeed
};
inline Fake& fake() { static Fake f; return f; }
inline cudaError_t fake_make(long** p) {
    if (fake().make_until-- <= 0) return cudaErrorUnknown;
    *p = new long(0);
    fake().live.insert(*p);
    return cudaSuccess;
}
inline cudaError_t fake_drop(long* p) { return fake().live.erase(p) ? cudaSuccess : cudaErrorUnknown; }
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, int) { return fake_make(s); }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) { return fake_make(e); }
inline cudaError_t cudaStreamDestroy(cudaStream_t s) { return fake_drop(s); }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { return fake_drop(e); }
inline cudaError_t cudaStreamQuery(cudaStream_t s) {
    return fake().busy.count(s) ? cudaErrorNotReady : fake().bad.count(s) ? cudaErrorUnknown : cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    fake().synced.push_back(s);
    fake().busy.erase(s);
    return fake().bad.count(s) ? cudaErrorUnknown : cudaSuccess;
}
"""

MAIN = r"""
#include <algorithm>
#include <cstdio>
#include <stdexcept>
#include "streams.h"
using muto::ClassFan; using muto::Forked; using muto::HandleStreams;
static int bad = 0;
#define EXPECT(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); ++bad; } } while (0)
static bool synced(cudaStream_t s) { auto& v = fake().synced; return std::count(v.begin(), v.end(), s) > 0; }
int main() {
    HandleStreams a;
    EXPECT(HandleStreams::take(0, &a) == cudaSuccess && a.fan.n == ClassFan::kSide);
    const size_t whole = fake().live.size();
    EXPECT(whole == 2 + 2 * ClassFan::kSide + HandleStreams::kOverlap);
    const HandleStreams was = a;
    fake().busy = {was.stream, was.fan.side[0], was.fan.side[ClassFan::kSide - 1]};
    a.give();  // every stream that runs waited for, then kept
    EXPECT(!a.stream && synced(was.stream) && fake().busy.empty() && fake().live.size() == whole);
    a.give();  // nothing left to give
    EXPECT(HandleStreams::take(0, &a) == cudaSuccess && a.stream == was.stream && fake().live.size() == whole);
    for (int k = 0; k <= ClassFan::kSide; ++k) {  // the work of one stream failed: not kept
        HandleStreams b;
        EXPECT(HandleStreams::take(0, &b) == cudaSuccess && b.stream != a.stream);
        fake().bad = {k < ClassFan::kSide ? b.fan.side[k] : b.stream};
        if (k % 2) fake().busy = fake().bad;
        b.give();
        EXPECT(!b.stream && fake().live.size() == whole);
        fake().bad.clear();
    }
    HandleStreams c;
    EXPECT(HandleStreams::take(1, &c) == cudaSuccess && c.device == 1);  // sets of a device stay there
    c.give();
    EXPECT(HandleStreams::take(0, &c) == cudaSuccess && c.device == 0);
    c.give();
    std::vector<HandleStreams> many(HandleStreams::kKept + 3);
    for (auto& m : many) EXPECT(HandleStreams::take(0, &m) == cudaSuccess);
    for (auto& m : many) m.give();
    EXPECT(HandleStreams::kept()[0].size() == HandleStreams::kKept);
    EXPECT(fake().live.size() == whole * (HandleStreams::kKept + 2));  // a, those kept here and on device 1
    for (int n = 0; n < static_cast<int>(whole); ++n) {  // a creation fails: nothing of the set is left
        fake().make_until = n;
        HandleStreams d;
        const size_t before = fake().live.size();
        EXPECT(HandleStreams::take(2, &d) != cudaSuccess && !d.stream && fake().live.size() == before);
    }
    for (int n = 0; n <= ClassFan::kSide; ++n) {  // left by an exception; joined
        fake().synced.clear();
        try {
            Forked f(a.fan, n);
            throw std::runtime_error("between fork and join");
        } catch (const std::exception&) {
        }
        EXPECT(fake().synced.size() == static_cast<size_t>(n) && (n == 0 || synced(a.fan.side[n - 1])));
        fake().synced.clear();
        {
            Forked f(a.fan, n);
            f.joined = true;
        }
        EXPECT(fake().synced.empty());
    }
    std::printf(bad ? "failed\n" : "ok\n");
    return bad;
}
"""


def test_pool_and_forks(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "main.cpp").write_text(MAIN)
    (tmp_path / "streams.h").write_text(HEADER.read_text())
    exe = tmp_path / "streams"
    subprocess.run(["g++", "-std=c++17", f"-I{tmp_path}", str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
