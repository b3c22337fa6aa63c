"""The cached scratch buffers (mimir_b200/csrc/scratch_pool.h) under several host threads, on the CPU: a buffer belongs to one call at a time, is
neither freed nor grown under it, and a failed allocation leaves the pool usable."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include <thread>
#include <vector>
#include "scratch_pool.h"

std::mutex m;
std::map<void*, size_t> live;   // what is allocated
std::map<void*, int> holders;   // who has it
std::atomic<int> fail{0}, waits{0}, bad{0};
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); ++bad; } } while (0)

struct Memory {
    static int alloc(void** p, size_t n) {
        if (fail) return 7;
        std::lock_guard<std::mutex> l(m);
        *p = std::malloc(1);
        live[*p] = n;
        return 0;
    }
    static int free(void* p) {
        std::lock_guard<std::mutex> l(m);
        CHECK(live.erase(p) == 1);
        CHECK(holders[p] == 0);
        std::free(p);
        return 0;
    }
    static int wait() { ++waits; return 0; }
};
using Pool = mimk::ScratchPool<Memory, 8>;

void calls(Pool& pool, int streams, int seed, int n) {
    std::mt19937 r(seed);
    for (int i = 0; i < n; ++i) {
        const size_t bytes = size_t(1) << (18 + r() % 6);
        Pool::Slot* s = nullptr;
        CHECK(pool.acquire(bytes, reinterpret_cast<void*>(size_t(r() % streams)), &s) == 0);
        void* p = s->ptr;
        {
            std::lock_guard<std::mutex> l(m);
            CHECK(live.count(p) && live[p] >= bytes && ++holders[p] == 1);
        }
        std::this_thread::yield();   // the call's launches
        {
            std::lock_guard<std::mutex> l(m);
            CHECK(live.count(p) && s->ptr == p && --holders[p] == 0);
        }
        pool.release(s);
    }
}

int main() {
    for (int streams : {1, 3, 8, 20}) {
        Pool pool;
        std::vector<std::thread> t;
        for (int i = 0; i < 10; ++i) t.emplace_back(calls, std::ref(pool), streams, i, 500);
        for (auto& x : t) x.join();
        std::lock_guard<std::mutex> l(m);
        CHECK(live.size() <= 8);
        live.clear(), holders.clear();
    }
    Pool pool;
    Pool::Slot *a = nullptr, *b = nullptr;
    void *one = reinterpret_cast<void*>(1), *two = reinterpret_cast<void*>(2);
    CHECK(pool.acquire(100, one, &a) == 0);
    void* p = a->ptr;
    CHECK(pool.acquire(100, two, &b) == 0 && b->ptr != p);   // another stream does not wait
    pool.release(a), pool.release(b);
    waits = 0;
    CHECK(pool.acquire(200, one, &a) == 0 && a->ptr == p && waits == 0);   // large enough: the same one, at once
    pool.release(a);
    fail = 1;
    CHECK(pool.acquire(size_t(1) << 30, one, &a) == 7 && waits == 1);
    CHECK(pool.acquire(100, reinterpret_cast<void*>(3), &a) == 7);
    fail = 0;
    CHECK(pool.acquire(100, one, &a) == 0 && live.count(a->ptr));
    pool.release(a);
    if (!bad) std::puts("ok");
    return bad != 0;
}
"""


def test_a_buffer_belongs_to_one_call_at_a_time(tmp_path):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM)
    build = subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "mimir_b200", "csrc"), str(src), "-o", str(exe)],
                           capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=240)
    assert run.returncode == 0 and run.stdout == "ok\n", run.stdout + run.stderr
