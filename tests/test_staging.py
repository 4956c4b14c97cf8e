"""The staged host copies (wr_staging.cpp) against a CUDA runtime made for the test: copies between its
pinned buffers and its device memory stay in flight until something waits for them, and single calls can
be made to fail. No GPU is involved."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "wurstrenderer_b200", "csrc")

RUNTIME = r"""
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <vector>

#include "wr_staging.h"

namespace {
struct Copy { void *to; const void *from; size_t bytes; };
std::mutex m;
std::deque<Copy> pending;              // in stream order
size_t issued = 0, done = 0;           // copies handed to the stream, and completed
std::map<char *, size_t> pinned;       // live pinned allocations
int host_allocs = 0, records = 0, fail_record = -1, early_frees = 0;

void run_to(size_t count) {
    while (done < count) {
        memcpy(pending.front().to, pending.front().from, pending.front().bytes);
        pending.pop_front();
        ++done;
    }
}
bool is_pinned(const void *p) {
    auto it = pinned.upper_bound(static_cast<char *>(const_cast<void *>(p)));
    return it != pinned.begin() && static_cast<const char *>(p) < (--it)->first + it->second;
}
}  // namespace

extern "C" {
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned int) {
    std::lock_guard<std::mutex> l(m);
    *p = malloc(bytes);
    pinned[static_cast<char *>(*p)] = bytes;
    ++host_allocs;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    std::lock_guard<std::mutex> l(m);
    for (const Copy &c : pending)
        if (is_pinned(c.to) || is_pinned(c.from)) ++early_frees;
    pinned.erase(static_cast<char *>(p));
    free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    std::lock_guard<std::mutex> l(m);
    a->type = is_pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned int) {
    *e = reinterpret_cast<cudaEvent_t>(new size_t(0));
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<size_t *>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
    std::lock_guard<std::mutex> l(m);
    if (records++ >= fail_record && fail_record >= 0) return cudaErrorUnknown;
    *reinterpret_cast<size_t *>(e) = issued;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::lock_guard<std::mutex> l(m);
    run_to(*reinterpret_cast<size_t *>(e));
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    std::lock_guard<std::mutex> l(m);
    run_to(issued);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t bytes, cudaMemcpyKind, cudaStream_t) {
    std::lock_guard<std::mutex> l(m);
    pending.push_back({to, from, bytes});
    ++issued;
    if (!is_pinned(to) && !is_pinned(from)) run_to(issued);   // pageable: the driver waits
    return cudaSuccess;
}
}

std::vector<unsigned char> bytes_of(size_t n, unsigned seed) {
    std::vector<unsigned char> v(n);
    for (size_t i = 0; i < n; ++i) v[i] = static_cast<unsigned char>((i * 2654435761u + seed) >> 7);
    return v;
}
#define CHECK(x) do { if (!(x)) { std::fprintf(stderr, "failed: %s (line %d)\n", #x, __LINE__); std::exit(1); } } while (0)
"""


def run_program(tmp_path, body):
    src, exe = tmp_path / "staging.cpp", tmp_path / "staging"
    src.write_text(RUNTIME + body)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", "/usr/local/cuda/include", str(src),
                    os.path.join(CSRC, "wr_staging.cpp"), "-o", str(exe), "-lpthread"], check=True)
    r = subprocess.run([str(exe)], timeout=120, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("fail", [0, 5, 38])
@pytest.mark.parametrize("way", ["to_host", "to_device"])
def test_a_failed_copy_leaves_nothing_in_flight(tmp_path, way, fail):
    """Events that cannot be recorded end the copy with an error, and no piece of it is on the bus
    over a staging buffer when the call returns; the copies after that are whole."""
    run_program(tmp_path, r"""
int main() {
    auto s = wr::Staging::shared();
    const size_t n = (size_t(100) << 20) + 12345;   // large enough to be staged, in 101 pieces
    auto a = bytes_of(n, 1), b = bytes_of(n, 2);
    std::vector<unsigned char> dev(n), host(n);
    CHECK(s->to_device(dev.data(), a.data(), n, nullptr) == cudaSuccess && dev == a);
    CHECK(host_allocs == 1);
    records = 0;
    fail_record = %d;
    CHECK(s->%s(%s) != cudaSuccess);
    CHECK(pending.empty());
    fail_record = -1;
    CHECK(s->to_device(dev.data(), b.data(), n, nullptr) == cudaSuccess && dev == b);
    CHECK(s->to_host(host.data(), dev.data(), n, nullptr) == cudaSuccess && host == b);
    CHECK(pending.empty());
    s.reset();
    CHECK(pinned.empty() && early_frees == 0);
}
""" % (fail, way, "host.data(), dev.data(), n, nullptr" if way == "to_host" else "dev.data(), a.data(), n, nullptr"))


def test_few_large_copies_need_no_buffers(tmp_path):
    """A program that copies little never pays for the staging buffers; one that goes on, or copies much
    at once, gets them, and they are given back with the last holder."""
    run_program(tmp_path, r"""
int main() {
    for (size_t mb : {3, 20, 64, 65}) {
        host_allocs = 0;
        auto s = wr::Staging::shared();
        const size_t n = mb << 20;
        auto a = bytes_of(n, unsigned(mb));
        std::vector<unsigned char> dev(n), host(n);
        size_t copied = 0;
        for (int k = 0; k < 30 && copied < (size_t(200) << 20); ++k) {
            const bool up = k % 2 == 0;
            CHECK((up ? s->to_device(dev.data(), a.data(), n, nullptr) : s->to_host(host.data(), dev.data(), n, nullptr)) == cudaSuccess);
            CHECK(up ? dev == a : host == a);
            copied += n;
            CHECK(host_allocs == (copied > (size_t(64) << 20) ? 1 : 0));
        }
        s.reset();
        CHECK(pinned.empty() && early_frees == 0);
    }
}
""")
