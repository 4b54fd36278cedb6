"""The copy threads of the host-pointer products (csrc/host_copy.cuh) against a stand-in for the CUDA runtime, on the CPU: every
byte of every piece arrives, a failing transfer is reported and ends the call, and nobody burns a core while a long product
runs or no segment is there. Compiled with the host compiler, the thread sanitizer where it is available."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUNTIME = r"""
#pragma once
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <thread>
// Device memory is host memory, copies happen at once, and a product is a time before which nothing recorded after it is over.
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorOperatingSystem = 304, cudaErrorNotReady = 600, cudaErrorUnknown = 999 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost };
enum cudaMemoryType { cudaMemoryTypeUnregistered };
struct cudaPointerAttributes { cudaMemoryType type; };
struct FakeEvent { bool blocking; std::chrono::steady_clock::time_point over; }; // when what was recorded is over
using cudaEvent_t = FakeEvent *;
using cudaStream_t = void *;
constexpr unsigned cudaEventDisableTiming = 2, cudaEventBlockingSync = 1, cudaHostAllocDefault = 0;
extern std::chrono::steady_clock::time_point fake_busy_until;
extern std::atomic<int> fake_copies_left;
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
inline cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = std::malloc(n); return *p ? cudaSuccess : cudaErrorUnknown; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned flags) { *e = new FakeEvent{(flags & cudaEventBlockingSync) != 0, {}}; return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { e->over = fake_busy_until; return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    if (e->blocking) std::this_thread::sleep_until(e->over);
    else while (std::chrono::steady_clock::now() < e->over) {}
    return cudaSuccess;
}
inline cudaError_t cudaEventQuery(cudaEvent_t e) { return std::chrono::steady_clock::now() < e->over ? cudaErrorNotReady : cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (fake_copies_left.fetch_sub(1) <= 0) return cudaErrorUnknown;
    std::memcpy(dst, src, n);
    return cudaSuccess;
}
"""

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <ctime>
#include <vector>
#include "cuda_runtime.h"
#include "host_copy.cuh"
std::chrono::steady_clock::time_point fake_busy_until;
std::atomic<int> fake_copies_left{1 << 30};
using namespace b200i;
static double cpu_seconds() {
    timespec t;
    clock_gettime(CLOCK_PROCESS_CPUTIME_ID, &t);
    return t.tv_sec + t.tv_nsec * 1e-9;
}
int main() {
    HostStage stage;
    if (host_stage_prepare(stage) != cudaSuccess) return 2;
    const size_t shapes[][3] = {{1, 1, 1}, {1000, 1000, 7}, {4, 64, 3000}, {3 << 20, 3 << 20, 1}, {(1 << 20) + 5, (1 << 20) + 9, 5}, {300, 4096, 5000}, {1 << 20, 1 << 21, 3}};
    for (const auto &s : shapes) { // width, pitch, rows
        std::vector<unsigned char> host(s[1] * s[2]), device(s[0] * s[2]), back(s[1] * s[2], 0xEE);
        const std::vector<unsigned char> untouched(s[1] - s[0], 0xEE);
        for (size_t i = 0; i < host.size(); i += 61) host[i] = (unsigned char)(i * 2654435761u >> 13);
        {
            HostCopier c(stage, 0, host.size());
            c.wait(c.add(true, device.data(), host.data(), s[0], s[1], s[2], nullptr));
            c.add(false, device.data(), back.data(), s[0], s[1], s[2], nullptr);
            if (!c.ok() || c.finish() != cudaSuccess) return 3;
        }
        for (size_t r = 0; r < s[2]; r++) {
            const size_t at = r * s[1];
            if (std::memcmp(&back[at], &host[at], s[0]) != 0 || std::memcmp(back.data() + at + s[0], untouched.data(), untouched.size()) != 0) return 4;
        }
    }
    { // a transfer fails in the middle: reported, and neither the waiting caller nor a worker stays behind
        std::vector<unsigned char> host(8 << 20), device(8 << 20);
        fake_copies_left = 3;
        HostCopier c(stage, 0, host.size());
        c.wait(c.add(true, device.data(), host.data(), host.size(), host.size(), 1, nullptr));
        c.add(false, device.data(), host.data(), host.size(), host.size(), 1, nullptr);
        if (c.finish() != cudaErrorUnknown) return 5;
        fake_copies_left = 1 << 30;
    }
    std::vector<unsigned char> host(8 << 20, 1), device(8 << 20);
    const double before = cpu_seconds();
    {
        HostCopier c(stage, 0, host.size());
        std::this_thread::sleep_for(std::chrono::milliseconds(300)); // nothing to do yet
        c.wait(c.add(true, device.data(), host.data(), host.size(), host.size(), 1, nullptr));
        fake_busy_until = std::chrono::steady_clock::now() + std::chrono::milliseconds(300); // the product
        c.add(false, device.data(), host.data(), host.size(), host.size(), 1, nullptr);
        if (c.finish() != cudaSuccess) return 6;
    }
    std::printf("%.3f\n", cpu_seconds() - before);
    return 0;
}
"""


def _run(tmp_path, flags):
    (tmp_path / "cuda_runtime.h").write_text("#include <atomic>\n" + RUNTIME)
    (tmp_path / "main.cpp").write_text(PROGRAM)
    exe = tmp_path / "copier"
    built = subprocess.run(["g++", "-std=c++17", "-pthread", *flags, "-I", str(tmp_path), "-I", os.path.join(ROOT, "mojolearn_b200", "csrc"), str(tmp_path / "main.cpp"),
                            "-o", str(exe)], capture_output=True, text=True)
    if built.returncode != 0 and "-fsanitize=thread" in flags:
        pytest.skip("no thread sanitizer: " + built.stderr[-200:])
    assert built.returncode == 0, built.stderr
    return subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_copies_are_whole_and_nobody_spins(tmp_path):
    ran = _run(tmp_path, ["-O2"])
    assert ran.returncode == 0, (ran.returncode, ran.stderr)
    assert float(ran.stdout) < 0.1, "CPU seconds in 0.6 s of waiting for work and for a product"


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_copies_under_the_thread_sanitizer(tmp_path):
    ran = _run(tmp_path, ["-O1", "-g", "-fsanitize=thread"])
    if "unexpected memory mapping" in ran.stderr:
        pytest.skip("the thread sanitizer does not run on this kernel")
    assert ran.returncode == 0 and "data race" not in ran.stderr, (ran.returncode, ran.stderr[-2000:])
