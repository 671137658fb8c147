"""Host copies shared out over helper threads (csrc/host_copy.cpp), compiled into a small program of their own: no GPU."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kyanite_b200", "csrc")

HEAD = r"""
#include "host_copy.cpp"
#include <cstdio>
#include <cstdlib>
#include <stdexcept>
#include <sys/mman.h>
#define REQUIRE(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); std::exit(1); } } while (0)
static uint8_t* pages(size_t n) {
    void* p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    REQUIRE(p != MAP_FAILED);
    return (uint8_t*)p;
}
static void fill(uint8_t* p, size_t n, unsigned seed) { for (size_t i = 0; i < n; i++) p[i] = (uint8_t)(i * 31 + (i >> 8) * 7 + seed); }
"""

# An upload of a finished range fails: the exception leaves `copy` only when no helper touches either buffer any more.
THROWING = r"""
int main() {
    auto pool = kn::CopyPool::shared();
    for (int turn = 0; turn < 20; turn++) {
        const size_t n = 64u << 20;
        uint8_t *src = pages(n), *dst = pages(n);
        fill(src, n, turn);
        bool thrown = false;
        try {
            pool->copy(dst, src, n, true, [](size_t, size_t) { throw std::runtime_error("upload"); });
        } catch (const std::runtime_error&) {
            thrown = true;
        }
        REQUIRE(thrown);
        munmap(src, n);   // a helper that goes on faults here
        munmap(dst, n);
    }
}
"""

# The process may start no more threads: the copy is made all the same.
NO_THREADS = r"""
extern "C" int pthread_create(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*) { return EAGAIN; }
int main() {
    const size_t n = (5u << 20) + 77;
    uint8_t *src = pages(n), *dst = pages(n);
    fill(src, n, 3);
    size_t next = 0;
    kn::CopyPool::shared()->copy(dst, src, n, true, [&](size_t from, size_t to) { REQUIRE(from == next); next = to; });
    REQUIRE(next == n && memcmp(src, dst, n) == 0);
}
"""

# Several threads at once: one has the helpers, the others copy alone; buffers that start at any byte.
SEVERAL = r"""
int main() {
    auto pool = kn::CopyPool::shared();
    std::vector<std::thread> users;
    for (int t = 0; t < 4; t++)
        users.emplace_back([&, t] {
            const size_t n = (3u << 20) + 1000 * t + 13;
            uint8_t *src = pages(n + 16), *dst = pages(n + 16);
            for (int turn = 0; turn < 30; turn++) {
                fill(src, n, turn + 100 * t);
                size_t next = 0;
                pool->copy(dst + t, src, n, turn % 2 == 0, [&](size_t from, size_t to) { REQUIRE(from == next && to > from); next = to; });
                REQUIRE(next == n && memcmp(src, dst + t, n) == 0);
            }
        });
    for (auto& u : users) u.join();
}
"""


def run(tmp_path, body, *flags):
    compiler = shutil.which("g++")
    if compiler is None:
        pytest.skip("no g++")
    source, program = tmp_path / "program.cpp", tmp_path / "program"
    source.write_text(HEAD + body)
    subprocess.run([compiler, "-std=c++17", "-O2", "-I", CSRC, str(source), "-o", str(program), "-lpthread", *flags], check=True)
    done = subprocess.run([str(program)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, (done.returncode, done.stdout)


def test_failing_upload(tmp_path):
    run(tmp_path, THROWING)


def test_no_threads(tmp_path):
    run(tmp_path, NO_THREADS)


def test_several_users(tmp_path):
    run(tmp_path, SEVERAL)
