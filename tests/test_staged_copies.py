"""The staged host copies (staging.cu) against a fake CUDA runtime on the CPU:
every byte arrives in both directions whatever the runtime refuses, the
page-locked slots, the event, or all but some of the streams.  Host memory that
is page-locked itself goes without slots.  A refused copy itself is an error."""

from __future__ import annotations

import ctypes
import subprocess

import numpy as np
import pytest

from conftest import ROOT

FAKE = r"""
#include <atomic>
#include <cstdlib>
#include "staging.cuh"

static int g_alloc = 1, g_event = 1, g_copy = 1;
static cudaMemoryType g_host = cudaMemoryTypeUnregistered;
static std::atomic<int> g_streams{0};
static std::atomic<int> g_made{0}, g_plain{0}, g_live{0};
static char g_stream_tags[64];

extern "C" {
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    a->type = g_host;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    if (!g_alloc) return cudaErrorMemoryAllocation;
    *p = std::malloc(n);
    ++g_live;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { std::free(p); --g_live; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    if (g_made >= g_streams) return cudaErrorMemoryAllocation;
    *s = reinterpret_cast<cudaStream_t>(&g_stream_tags[g_made++]);
    ++g_live;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { --g_live; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    if (!g_event) return cudaErrorMemoryAllocation;
    *e = reinterpret_cast<cudaEvent_t>(&g_event);
    ++g_live;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { --g_live; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t n, cudaMemcpyKind,
                            cudaStream_t stream) {
    if (!g_copy) return cudaErrorInvalidValue;
    if (!stream) ++g_plain;  // the caller's own stream
    std::memcpy(to, from, n);
    return cudaSuccess;
}

// 0 and the count of plain copies in *plain, or 1 for an error, 2 for a leak.
int staged_copy(int alloc, int event, int streams, int copy, int locked, int to_host,
                char *host, char *gpu, size_t bytes, int *plain) {
    g_host = locked ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    g_alloc = alloc, g_event = event, g_streams = streams, g_copy = copy;
    g_made = 0, g_plain = 0;
    int status = 0;
    try {
        ls200::StagedCopies copies;
        for (int again = 0; again < 2; ++again) {
            if (to_host) copies.to_host(0, host, gpu, bytes, nullptr);
            else copies.to_device(0, gpu, host, bytes, nullptr);
        }
    } catch (const ls200::Error &) {
        status = 1;
    }
    *plain = g_plain;
    return g_live ? 2 : status;
}
}
"""


@pytest.fixture(scope="module")
def copy(tmp_path_factory):
    folder = tmp_path_factory.mktemp("staging")
    (folder / "fake.cpp").write_text(FAKE)
    csrc = ROOT / "lunarscout_b200" / "csrc"
    library = folder / "libstaging.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic",
                    f"-I{csrc}", "-I/usr/local/cuda/include", "-x", "c++",
                    str(csrc / "staging.cu"), str(folder / "fake.cpp"), "-o", str(library),
                    "-lpthread"], check=True)
    function = ctypes.CDLL(str(library)).staged_copy
    function.argtypes = [ctypes.c_int] * 6 + [ctypes.c_void_p] * 2 + [ctypes.c_size_t,
                                                                      ctypes.c_void_p]
    return function


def _run(copy, to_host, size, *, alloc=1, event=1, streams=10, works=1, locked=0):
    rng = np.random.default_rng(size)
    source = rng.integers(0, 256, size, dtype=np.uint8)
    target = np.zeros(size, np.uint8)
    host, gpu = (target, source) if to_host else (source, target)
    plain = ctypes.c_int()
    status = copy(alloc, event, streams, works, locked, to_host, host.ctypes.data,
                  gpu.ctypes.data, size, ctypes.byref(plain))
    return status, bool((source == target).all()), plain.value


@pytest.mark.parametrize("to_host", [0, 1])
@pytest.mark.parametrize("size", [1, (1 << 20) - 1, 1 << 20, (1 << 20) + 1, 13_000_003])
def test_every_byte_arrives(copy, to_host, size):
    assert _run(copy, to_host, size) == (0, True, 0)
    for streams in (1, 2, 9):
        assert _run(copy, to_host, size, streams=streams) == (0, True, 0)


@pytest.mark.parametrize("to_host", [0, 1])
@pytest.mark.parametrize("refused", [dict(alloc=0), dict(event=0), dict(streams=0),
                                     dict(alloc=0, event=0, streams=0)])
def test_a_refused_slot_event_or_stream_leaves_the_plain_copy(copy, to_host, refused):
    assert _run(copy, to_host, 3_000_001, **refused) == (0, True, 2)


@pytest.mark.parametrize("to_host", [0, 1])
def test_page_locked_memory_takes_the_plain_copy(copy, to_host):
    assert _run(copy, to_host, 3_000_001, locked=1) == (0, True, 2)


@pytest.mark.parametrize("to_host", [0, 1])
@pytest.mark.parametrize("options", [{}, dict(alloc=0)])
def test_a_failed_copy_is_an_error(copy, to_host, options):
    assert _run(copy, to_host, 3_000_001, works=0, **options)[0] == 1
