"""CPU test of the host entry points' copies (ffg_slots.h) against a fake of the
runtime's calls, whose copies from and to pinned memory happen only when an event or
the stream is waited for: sizes around a slot and around all four, the source
overwritten as soon as up() returns; and without pinned memory (the allocation or an
event refused) the same bytes by the driver's own copies, with nothing left allocated
and no error left behind for the next launch to find."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fastfib_b200" / "csrc"

SOURCE = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <set>
#include <vector>
#include "ffg_slots.h"
using namespace ffg;
static bool no_memory = false;
static int events_left = 1000, events = 0, pending_copies = 0;
static cudaError_t last = cudaSuccess;
static char *pin = nullptr;
static size_t pin_n = 0;
struct Op { std::function<void()> run; cudaEvent_t mark; };
static std::vector<Op> queue_;
static void flush(cudaEvent_t until) {
    size_t stop = queue_.size();
    if (until) {
        stop = 0;
        for (size_t i = 0; i < queue_.size(); i++) if (queue_[i].mark == until) stop = i + 1;
    }
    for (size_t i = 0; i < stop; i++) if (queue_[i].run) queue_[i].run();
    queue_.erase(queue_.begin(), queue_.begin() + stop);
}
static bool pinned(const void *p) { return pin && (char *)p >= pin && (char *)p < pin + pin_n; }
extern "C" {
cudaError_t cudaMallocHost(void **p, size_t n) {
    if (no_memory) return last = cudaErrorMemoryAllocation;
    *p = pin = (char *)malloc(n);
    pin_n = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { free(p); pin = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    if (events_left-- <= 0) return last = cudaErrorMemoryAllocation;
    *e = (cudaEvent_t)malloc(1);
    events++;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { free((void *)e); events--; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { queue_.push_back({nullptr, e}); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { flush(e); return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind, cudaStream_t) {
    if (pinned(d) || pinned(s)) {
        queue_.push_back({[=] { memcpy(d, s, n); }, nullptr});
    } else { // pageable: staged before the call returns
        flush(nullptr);
        memcpy(d, s, n);
    }
    return cudaSuccess;
}
}
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); exit(1); } } while (0)
static std::vector<char> bytes(size_t n, int seed) {
    std::vector<char> v(n);
    uint32_t x = 12345u + seed;
    for (auto &c : v) c = (char)((x = x * 1664525u + 1013904223u) >> 24);
    return v;
}
static void round_trip(HostSlots &s) {
    const size_t K = HostSlots::kBytes;
    const size_t sizes[] = {0, 1, 8, K - 1, K, K + 1, 3 * K, 4 * K, 4 * K + 1, 5 * K, 9 * K + K / 3};
    for (size_t na : sizes)
        for (size_t nb : sizes) {
            s.ready();
            std::vector<char> a = bytes(na, 1), b = bytes(nb, 2), da(na), db(nb), src = a;
            CHECK(!s.up(da.data(), src.data(), na, nullptr));
            std::fill(src.begin(), src.end(), 0);
            src = b;
            CHECK(!s.up(db.data(), src.data(), nb, nullptr));
            std::fill(src.begin(), src.end(), 0);
            std::vector<char> out(na + 1, 'x'); // down waits for all that is queued
            CHECK(!s.down(out.data(), da.data(), na, nullptr));
            flush(nullptr);
            CHECK(da == a && db == b);
            CHECK(std::vector<char>(out.begin(), out.end() - 1) == a && out[na] == 'x');
        }
}
int main() {
    HostSlots s;
    CHECK(s.ready() && s.mem);
    round_trip(s);
    s.release();
    CHECK(!pin && events == 0 && !s.mem);
    for (int c = 0; c < 2; c++) { // no pinned memory; no third event
        no_memory = c == 0;
        events_left = c == 0 ? 1000 : 2;
        CHECK(!s.ready() && !s.mem && !pin && events == 0 && last == cudaSuccess);
        events_left = c == 0 ? 1000 : 0;
        round_trip(s);
        CHECK(last == cudaSuccess);
    }
    no_memory = false;
    events_left = 1000;
    CHECK(s.ready()); // and the slots again once they can be had
    round_trip(s);
    s.release();
    puts("ok");
}
"""


def test_copies_with_and_without_pinned_memory(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not shutil.which("g++") or not os.path.exists(os.path.join(inc, "cuda_runtime_api.h")):
        pytest.skip("needs g++ and the CUDA headers")
    (tmp_path / "t.cpp").write_text(SOURCE)
    exe = tmp_path / "t"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address,undefined", f"-I{CSRC}", f"-I{inc}",
                        str(tmp_path / "t.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr[-3000:]


def test_entry_points_take_the_copies_that_there_are():
    """ready() answering no is not an error of the entry points."""
    text = (CSRC / "ffg_host.cu").read_text()
    assert "pinned host slots" not in text
    assert text.count("g_slots.ready()") == 2 and "g_slots.up(" in text and "g_slots.down(" in text
