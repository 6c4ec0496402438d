"""Parts of the kernels that are plain C++ (`csrc/*.cuh`), compiled for the host and run here."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "slopllm_b200", "csrc")


def run(tmp_path, source: str, *flags: str) -> None:
    """Compiles a program that returns the line of its first failing check."""
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    (tmp_path / "t.cpp").write_text("#define CHECK(x) do { if (!(x)) return __LINE__; } while (0)\n#line 1\n" + source)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, *flags, "-o", exe, str(tmp_path / "t.cpp")], check=True)
    r = subprocess.run([exe], timeout=60)
    assert r.returncode == 0, f"line {r.returncode}: {source.splitlines()[r.returncode - 1]}"


def test_bounded_waits_end_once_one_has_run_out(tmp_path):
    """A phase that never comes ends the wait by the clock; behind it no wait and no poll of this thread looks at a barrier again, and those of
    other threads of the block end within 256 looks."""
    run(tmp_path, """
#include "bounded_waits.cuh"
struct Dev {
    using Bar = int;                       // phases that have passed
    static inline int looks = 0, reported = 0;
    static inline uint64_t clock = 1;
    static bool try_wait(Bar* b, uint32_t parity) { ++looks; return *b > 0 && ((*b - 1) & 1) == (int)parity; }
    static bool test(Bar* b, uint32_t parity) { return try_wait(b, parity); }
    static uint64_t now_ns() { return clock += 1000000; }
    static bool any(bool f) { return f; }
    static void report(int* err, int code) { *err = code; ++reported; }
};
int main() {
    volatile int failed = 0;
    int err = 0, never = 0, passed = 1;
    BoundedWaits<Dev> a{&failed, &err, 34}, b{&failed, &err, 34};
    CHECK(a(&passed, 0) && Dev::looks == 1);
    CHECK(a.second_of(&never, 0, &passed, 0) && !a.second_of(&passed, 0, &passed, 0) && a.alive);
    Dev::looks = 0;
    CHECK(!a.second_of(&never, 0, &never, 0) && a.alive && failed == 0);
    CHECK(Dev::looks == 2 * (int)BoundedWaits<Dev>::POLLS);
    Dev::looks = 0;
    CHECK(!a(&never, 0) && !a.alive && failed == 1 && err == 34 && Dev::reported == 1);
    CHECK(Dev::looks > 256 && Dev::looks < 256 * 2010);
    Dev::looks = 0;
    CHECK(!a(&passed, 0) && !a.second_of(&never, 0, &never, 0) && !a.second_of(&never, 0, &passed, 0) && Dev::looks == 0);
    CHECK(!b.second_of(&never, 0, &never, 0) && Dev::looks <= 2 * 256 && b.alive);
    Dev::looks = 0;
    CHECK(!b(&never, 0) && !b.alive && Dev::looks <= 257 + 256);
    return 0;
}
""")


def test_shared_memory_opt_in_is_per_device_and_after_success(tmp_path):
    """Attributes are set once on each device, again where they failed (and the call's error returned, and cleared), and for one kernel only."""
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))), "include")
    if not os.path.exists(os.path.join(inc, "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    run(tmp_path, """
#include "smem_optin.h"
static int device = 0, sets = 0, clears = 0, fail = 0, last_value = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int v) { ++sets; last_value = v; return fail ? cudaErrorInvalidValue : cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { ++clears; return cudaSuccess; }
int main() {
    SmemOptIn a, b;
    fail = 1;
    CHECK(a(0, 100) == cudaErrorInvalidValue && sets == 1 && clears == 1);
    fail = 0;
    CHECK(a(0, 100) == 0 && sets == 2 && last_value == 100 && a(0, 100) == 0 && sets == 2);
    device = 1;
    CHECK(a(0, 100) == 0 && sets == 3 && a(0, 100) == 0 && sets == 3);
    device = 0;
    CHECK(a(0, 100) == 0 && sets == 3 && b(0, 100, 40) == 0 && sets == 5 && last_value == 40 && b(0, 100, 40) == 0 && sets == 5);
    device = 70;
    CHECK(a(0, 100) == 0 && a(0, 100) == 0 && sets == 7);
    return 0;
}
""", "-I", inc)
