"""The host side of state and row copies (autan_b200/csrc/host_stage.hpp) compiled for the host against
a stand-in of the runtime's calls: what comes back is what went in with the slots, without pinned memory
and with the slots taken by another copy."""

import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parent.parent

RUNTIME = r"""
#pragma once
#include <atomic>
#include <cstdlib>
#include <cstring>
typedef int cudaError_t;
typedef void* cudaStream_t;
typedef void* cudaEvent_t;
constexpr int cudaSuccess = 0, cudaErrorMemoryAllocation = 2;
enum cudaMemcpyKind { cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost };
enum { cudaHostAllocDefault = 0, cudaEventDisableTiming = 2 };
enum { cudaMemoryTypeUnregistered, cudaMemoryTypeHost, cudaMemoryTypeDevice, cudaMemoryTypeManaged };
struct cudaPointerAttributes { int type; };
inline bool pinned_memory_there = true;
inline std::atomic<int> pinned_calls{0}, copies{0};
inline cudaError_t cudaGetDevice(int* d) { *d = 0; return 0; }
inline cudaError_t cudaSetDevice(int) { return 0; }
inline cudaError_t cudaGetLastError() { return 0; }
inline cudaError_t cudaHostAlloc(void** p, size_t n, int) {
  ++pinned_calls;
  if (!pinned_memory_there) return cudaErrorMemoryAllocation;
  *p = std::malloc(n);
  return 0;
}
inline cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
inline cudaError_t cudaFreeHost(void* p) { std::free(p); return 0; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) { *e = std::malloc(1); return 0; }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return 0; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return 0; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return 0; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = 0; return 0; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  ++copies;
  std::memcpy(d, s, n);
  return 0;
}
"""

PROGRAM = r"""
#include "host_stage.hpp"
#include <cstdio>
#include <cstdlib>
using namespace autan_b200;
int main(int, char** argv) {
  const size_t bytes = std::strtoull(argv[1], nullptr, 10);
  pinned_memory_there = argv[2][0] == '1';
  const bool may_pin = argv[3][0] == '1';
  const int callers = std::atoi(argv[4]);
  auto in = HostStage::of_device(0), out = HostStage::of_device(1);
  std::atomic<int> errors{0}, wrong{0};
  auto caller = [&](unsigned seed) {
    std::vector<unsigned char> a(bytes), dev(bytes), b(bytes, 0);
    for (size_t i = 0; i < bytes; ++i) a[i] = static_cast<unsigned char>((i + seed) * 2654435761u >> 13);
    if (in->to_device(dev.data(), a.data(), bytes, nullptr, may_pin) != cudaSuccess) ++errors;
    if (out->to_host(b.data(), dev.data(), bytes, nullptr, may_pin) != cudaSuccess) ++errors;
    if (a != b) ++wrong;
  };
  std::vector<std::thread> team;
  for (int c = 1; c < callers; ++c) team.emplace_back(caller, 77u * static_cast<unsigned>(c));
  caller(0);
  for (std::thread& t : team) t.join();
  const int made = copies.load();
  HostRows rows;
  const bool first = rows.get(4096) != nullptr;
  const int asked = pinned_calls;
  const bool again = rows.get(4096) != nullptr;
  std::printf("%d %d %d %d %d %d\n", errors.load(), wrong.load(), made, first ? 1 : 0, again ? 1 : 0,
              pinned_calls.load() - asked);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("stage")
    (d / "cuda_runtime.h").write_text(RUNTIME)
    (d / "stage.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{d}", f"-I{REPO / 'autan_b200' / 'csrc'}",
                    str(d / "stage.cpp"), "-o", str(d / "stage")], check=True)  # fmt: skip

    def run(*args):
        r = subprocess.run([str(d / "stage"), *map(str, args)], check=True, capture_output=True, text=True,
                           timeout=60)  # fmt: skip
        return [int(v) for v in r.stdout.split()]

    return run


@pytest.mark.parametrize("size", [1, 4096, (1 << 20) - 1, 1 << 20, (1 << 20) + 12345, 5 << 20, (9 << 20) + 7])
@pytest.mark.parametrize("there", [1, 0])
@pytest.mark.parametrize("may_pin", [1, 0])
def test_copies_come_back(program, size, there, may_pin):
    errors, wrong, copies, first, again, asked = program(size, there, may_pin, 1)
    assert errors == 0 and wrong == 0
    assert (copies > 2) == bool(there and may_pin and size >= 1 << 20)  # through the slots, or one a way
    # rows of a handle's own: got once, or done without after one refusal
    assert (first, again, asked) == ((1, 1, 0) if there else (0, 0, 0))


@pytest.mark.parametrize("size", [(1 << 20) + 12345, (9 << 20) + 7])
def test_copies_of_several_threads(program, size):
    """The slots serve one copy at a time and direction; the others go the driver's way."""
    for _ in range(5):
        errors, wrong, copies, *_ = program(size, 1, 1, 6)
        assert errors == 0 and wrong == 0 and copies > 12
