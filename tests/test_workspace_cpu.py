"""The store of kept blocks (csrc/workspace.cu) over a CUDA runtime that only keeps books:
what it asks the driver for, what it keeps and what it gives back."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MiB = 1 << 20
HELD = 512 * MiB  # kept at most, per device

FAKE_RUNTIME = r"""
#include <cuda_runtime.h>
#include <cstdarg>
#include <map>
#include "internal.h"

static std::map<void *, size_t> g_device, g_host;
static size_t g_used, g_total = ~0ull, g_calls;
static uintptr_t g_next = 1u << 20;

static cudaError_t take(std::map<void *, size_t> &m, void **p, size_t n, bool counts) {
    if (counts && g_used + n > g_total) return cudaErrorMemoryAllocation;
    g_calls += 1;
    *p = (void *)g_next;
    g_next += n + 512;
    m[*p] = n;
    if (counts) g_used += n;
    return cudaSuccess;
}
extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) { return take(g_device, p, n, true); }
cudaError_t cudaFree(void *p) { g_used -= g_device.at(p); g_device.erase(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return take(g_host, p, n, false); }
cudaError_t cudaFreeHost(void *p) { g_host.erase(p); return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { *s = (cudaStream_t)g_next++; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }

void *t_alloc(size_t n) { void *p = nullptr; return ag::workspace_alloc(&p, n) == cudaSuccess ? p : nullptr; }
void t_free(void *p) { ag::workspace_free(p); }
void *t_user() { return new ag::WorkspaceUser(); }
void t_user_gone(void *u) { delete (ag::WorkspaceUser *)u; }
size_t t_used() { return g_used; }
size_t t_calls() { return g_calls; }
void t_total(size_t n) { g_total = n; }
}
namespace ag { void set_error(const char *, ...) {} }
"""


@pytest.fixture(scope="module")
def build(tmp_path_factory):
    cuda = os.environ.get("CUDA_HOME") or "/usr/local/cuda"
    if not shutil.which("g++") or not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("workspace")
    (d / "fake.cpp").write_text(FAKE_RUNTIME)
    csrc = os.path.join(ROOT, "aethergraph_b200", "csrc")
    # -Bsymbolic: the fake runtime, whatever other one the process has loaded
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I" + os.path.join(cuda, "include"), "-I" + csrc, "-x", "c++",
                    os.path.join(csrc, "workspace.cu"), str(d / "fake.cpp"), "-o", str(d / "ws.so")], check=True)
    return d


@pytest.fixture
def ws(build, tmp_path):
    """A library of its own for every test: the store is never destroyed."""
    so = shutil.copy(build / "ws.so", tmp_path / "ws.so")
    lib = C.CDLL(so)
    lib.t_alloc.restype = lib.t_user.restype = C.c_void_p
    lib.t_used.restype = lib.t_calls.restype = C.c_size_t
    lib.t_alloc.argtypes = lib.t_total.argtypes = [C.c_size_t]
    lib.t_free.argtypes = lib.t_user_gone.argtypes = [C.c_void_p]
    lib.first_user = lib.t_user()
    return lib


@pytest.mark.parametrize("mib", [2.0, 2.1, 9.3, 290, 511, 513, 7000.7])
def test_large_blocks_take_no_more_than_the_driver_maps(ws, mib):
    """The driver maps 2 MiB at a time; anything above that is memory a program can miss."""
    want = int(mib * MiB)
    a, b = ws.t_alloc(want), ws.t_alloc(want)
    assert a and b and ws.t_used() <= 2 * -(-want // (2 * MiB)) * 2 * MiB


def test_a_program_that_just_fits(ws):
    ws.t_total(4000 * MiB)
    blocks = [ws.t_alloc(290 * MiB) for _ in range(13)]
    assert all(blocks)


def test_kept_blocks_serve_equal_and_somewhat_smaller_requests(ws):
    for want, smaller, much_smaller in ((4000, 3900, 2000), (3 * MiB, 3 * MiB - 100, MiB), (290 * MiB, 270 * MiB, 200 * MiB)):
        p = ws.t_alloc(want)
        ws.t_free(p)
        assert ws.t_alloc(want) == p
        ws.t_free(p)
        assert ws.t_alloc(smaller) == p
        ws.t_free(p)
        calls = ws.t_calls()
        ws.t_free(ws.t_alloc(much_smaller))
        assert ws.t_calls() == calls + 1


def test_kept_memory_is_bounded(ws):
    blocks = [ws.t_alloc(s * MiB) for s in (100, 200, 300, 50, 513)]
    for p in blocks:
        ws.t_free(p)
        assert ws.t_used() <= HELD + sum((100, 200, 300, 50, 513)) * MiB
    assert ws.t_used() <= HELD


def test_a_failed_request_is_tried_again_without_the_kept_blocks(ws):
    ws.t_total(600 * MiB)
    ws.t_free(ws.t_alloc(400 * MiB))
    assert ws.t_alloc(500 * MiB)


def test_kept_memory_can_be_asked_back(ws):
    held = ws.t_alloc(10 * MiB)
    ws.t_free(ws.t_alloc(100 * MiB))
    ws.ag_release_kept_memory()
    assert ws.t_used() == 10 * MiB
    ws.t_free(held)
    assert ws.t_alloc(10 * MiB) == held


def test_the_last_user_gives_everything_back(ws):
    second = ws.t_user()
    ws.t_free(ws.t_alloc(100 * MiB))
    ws.t_user_gone(second)
    assert ws.t_used() > 0
    ws.t_user_gone(ws.first_user)
    assert ws.t_used() == 0
    ws.t_free(ws.t_alloc(100 * MiB))  # nobody left to keep it for
    assert ws.t_used() == 0
