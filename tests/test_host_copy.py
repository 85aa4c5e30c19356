"""The host-side copier: shared copies, streams through a ring, and the errors that end them (CPU only)."""
import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include "host_copy.h"
#include <new>
#include <stdio.h>
#include <stdlib.h>

static bool full = false;   // memory has run out
void *operator new(size_t n) {
    if (full) throw std::bad_alloc();
    return malloc(n);
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    HostCopier copier;
    const size_t chunk = HostCopier::kChunk, ring_bytes = 8 * chunk;
    std::vector<unsigned char> src(23 * 1024 * 1024 + 17), dst(src.size()), ring(ring_bytes);
    for (size_t i = 0; i < src.size(); ++i) src[i] = (unsigned char)(i * 2654435761u >> 13);
    const size_t sizes[] = {0, 1, 100, HostCopier::kParallelFrom - 1, HostCopier::kParallelFrom, HostCopier::kWakeFrom + 3, ring_bytes, src.size()};
    for (int round = 0; round < 3; ++round)
        for (size_t n : sizes) {
            std::fill(dst.begin(), dst.end(), 0);
            copier.copy(dst.data(), src.data(), n);
            CHECK(memcmp(dst.data(), src.data(), n) == 0 && (n == dst.size() || dst[n] == 0));
            if (n == 0) continue;
            // pieces in order, none wraps, each consumed two calls after it was sent
            std::fill(dst.begin(), dst.end(), 0);
            size_t sent = 0, before = 0, freed = 0;
            int rc = copier.stream(ring.data(), ring_bytes, src.data(), n,
                [&](size_t at, size_t lo, size_t len) -> int {
                    if (lo != sent || at + len > ring_bytes) return -9;
                    memcpy(dst.data() + lo, ring.data() + at, len);
                    before = sent;
                    sent += len;
                    return 0;
                },
                [&]() -> long long {
                    const size_t f = freed;
                    freed = before == f ? sent : before;
                    return (long long)f;
                }, -7);
            CHECK(rc == 0 && sent == n && memcmp(dst.data(), src.data(), n) == 0);
        }
    // a consumer that fails: the copy ends with its code, whoever finds out
    int calls = 0;
    CHECK(copier.stream(ring.data(), ring_bytes, src.data(), src.size(), [&](size_t, size_t, size_t) { return 0; },
                        [&]() -> long long { return ++calls > 5 ? -2 : 0; }, -7) == -2);
    size_t gone = 0;
    CHECK(copier.stream(ring.data(), ring_bytes, src.data(), src.size(), [&](size_t, size_t lo, size_t len) { gone = lo + len; return lo > 0 ? -3 : 0; },
                        [&]() -> long long { return (long long)gone; }, -7) == -3);
    copier.copy(dst.data(), src.data(), src.size());
    CHECK(memcmp(dst.data(), src.data(), src.size()) == 0);
    // without memory for its marks a copy is made alone, and a stream is refused before anything was sent
    HostCopier fresh;
    std::fill(dst.begin(), dst.end(), 0);
    full = true;
    fresh.copy(dst.data(), src.data(), src.size());
    const int rc = fresh.stream(ring.data(), ring_bytes, src.data(), src.size(), [&](size_t, size_t, size_t) { return -9; }, [&]() -> long long { return 0; }, -7);
    full = false;
    CHECK(rc == -7 && memcmp(dst.data(), src.data(), src.size()) == 0);
    return 0;
}
"""


def test_host_copier(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", os.path.join(ROOT, "aet-cnn_b200", "csrc"), str(tmp_path / "t.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
