"""The list of work memory that gradients leave for the next ones (csrc/bfx_work_pool.h, host-only),
compiled with g++ over a stand-in allocator of a given capacity.  CPU only."""
from __future__ import annotations

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "numi-gpu-physics_b200", "csrc")

FAKE = r'''
#include <cstdio>
#include <map>
#include <mutex>
#include <thread>
#include <vector>
#include "bfx_work_pool.h"
using namespace bfx;
// a device of `room` bytes
static std::mutex fm;
static std::map<void*, size_t> live;
static size_t room = 0, used = 0;
static int allocations = 0;
static char* next_address = (char*)4096;
enum { kOk = 0, kBroken = 1, kOutOfMemory = 2 };
static int broken = 0;
static int fake_allocate(void** p, size_t n) {
    std::lock_guard<std::mutex> l(fm);
    if (broken) return kBroken;
    if (n > room - used) return kOutOfMemory;
    *p = next_address;
    next_address += n + 4096;
    live[*p] = n;
    used += n;
    ++allocations;
    return kOk;
}
static int bad_release = 0;
static void fake_release(void* p) {
    std::lock_guard<std::mutex> l(fm);
    auto it = live.find(p);
    if (it == live.end()) { ++bad_release; return; }
    used -= it->second;
    live.erase(it);
}
#define CHECK(c) do { if (!(c)) { std::printf("FAIL %s:%d %s\n", __FILE__, __LINE__, #c); return 1; } } while (0)
static int A, B;  // owners
'''

DRIVER = FAKE + r'''
static WorkPool pool({fake_allocate, fake_release, kOutOfMemory});
static void reset(size_t r) { pool.drain(0); pool.drain(1); room = r; allocations = 0; broken = 0; }

static int a_call_finds_the_blocks_of_the_last() {
    reset(1 << 30);
    void *p = nullptr, *q = nullptr, *first[2];
    { WorkCall c(pool, 0, &A); CHECK(c.get(&p, 1000000) == 0 && c.get(&q, 0) == 0 && c.bytes() == 1000016);
      first[0] = p; first[1] = q; c.keep(1 << 30); }
    CHECK(used == 1000016 && pool.held(&A) == 1000016 && pool.held(&B) == 0);
    { WorkCall c(pool, 0, &B); CHECK(c.get(&p, 900000) == 0 && p == first[0] && allocations == 2 && !c.allocated());
      CHECK(pool.held(&A) == 16); c.keep(1 << 30); }
    CHECK(pool.held(&B) == 1000000 && pool.held(&A) == 16);
    { WorkCall c(pool, 0, &A); CHECK(c.get(&p, 700000) == 0 && p != first[0]);    // a quarter wasted: not taken
      void* r = nullptr; CHECK(c.get(&r, 1000001) == 0 && r != first[0] && c.allocated()); c.keep(1 << 30); }
    CHECK(pool.held(&A) == 1700001);                  // its 16 bytes, not used again, were freed
    WorkCall other(pool, 1, &A);                      // another device's blocks are no use
    CHECK(other.get(&p, 1000000) == 0 && p != first[0] && pool.held(&B) == 1000000);
    return 0;
}
static int a_failed_call_frees_all_it_had() {
    reset(1000);
    void *p = nullptr, *q = nullptr;
    { WorkCall c(pool, 0, &A); CHECK(c.get(&p, 600) == 0); c.keep(1000); }
    CHECK(used == 600);
    { WorkCall c(pool, 0, &B); CHECK(c.get(&p, 600) == 0 && c.get(&q, 500) == kOutOfMemory); }
    CHECK(used == 0 && pool.held(&A) == 0 && pool.held(&B) == 0);
    return 0;
}
static int an_allocation_that_fails_gets_the_list() {
    reset(1000);
    void *p = nullptr, *q = nullptr;
    { WorkCall c(pool, 0, &A); CHECK(c.get(&p, 300) == 0 && c.get(&q, 300) == 0); c.keep(1000); }
    void* r = nullptr;
    CHECK(pool.allocate(0, &r, 900) == 0 && used == 900 && pool.held(&A) == 0);   // any handle's allocation
    CHECK(pool.allocate(0, &q, 200) == kOutOfMemory);                             // nothing left to give
    pool.release(r);
    { WorkCall c(pool, 1, &A); CHECK(c.get(&p, 600) == 0); c.keep(1000); }
    CHECK(pool.allocate(0, &r, 900) == kOutOfMemory && pool.held(&A) == 600);     // the other device keeps its own
    broken = 1;                                                                   // not a lack of memory
    CHECK(pool.allocate(1, &r, 900) == kBroken && pool.held(&A) == 600);
    return 0;
}
static int the_list_is_bounded() {
    reset(1 << 30);
    void* p = nullptr;
    { WorkCall c(pool, 0, &A); for (int i = 0; i < 4; ++i) CHECK(c.get(&p, 100000 * (i + 1)) == 0); c.keep(350000); }
    CHECK(pool.held(&A) == 300000 && used == 300000);         // 100 + 200; 300 and 400 do not fit
    { WorkCall c(pool, 0, &B); CHECK(c.get(&p, 350000) == 0); c.keep(350000); }
    CHECK(pool.held(&B) == 350000 && pool.held(&A) == 0 && used == 350000);       // the oldest went
    { WorkCall c(pool, 0, &A); CHECK(c.get(&p, 10000) == 0); c.keep(0); }
    CHECK(pool.held(&A) == 0 && used == 350000);              // nothing is kept when nothing may be
    { WorkCall c(pool, 0, &A); int got = 0; while (c.get(&p, 5000000) == 0) ++got;
      CHECK(got == WorkPool::kMaxBlocks); c.keep((size_t)1 << 30); }
    CHECK(pool.held(&A) == (size_t)5000000 * WorkPool::kMaxBlocks && pool.held(&B) == 0);
    CHECK(pool.drop(&A) == (size_t)5000000 * WorkPool::kMaxBlocks && used == 0);  // and goes with its handle
    return 0;
}
int main() {
    if (a_call_finds_the_blocks_of_the_last() || a_failed_call_frees_all_it_had() ||
        an_allocation_that_fails_gets_the_list() || the_list_is_bounded()) return 1;
    CHECK(bad_release == 0);
    std::printf("OK\n");
    return 0;
}
'''

THREADS = FAKE + r'''
static WorkPool pool({fake_allocate, fake_release, kOutOfMemory});
int main() {
    room = 40000;
    std::mutex bm;
    int bad = 0;
    auto worker = [&](int id) {
        int me;  // an owner of its own
        for (int i = 0; i < 4000; ++i) {
            WorkCall c(pool, id & 1, &me);
            std::vector<void*> mine;
            for (int k = 0; k < 3; ++k) {
                void* p = nullptr;
                if (c.get(&p, 100 + 37 * ((i + k + id) % 90)) == 0) mine.push_back(p);
            }
            {   // every block is live and belongs to this call alone
                std::lock_guard<std::mutex> l(fm);
                for (void* p : mine) if (!live.count(p)) { std::lock_guard<std::mutex> b(bm); ++bad; }
            }
            if (i % 5) c.keep(9000);
            if (i % 97 == 0) pool.drain(id & 1);
            if (i % 31 == 0) pool.drop(&me);
        }
        pool.drop(&me);
    };
    std::vector<std::thread> t;
    for (int i = 0; i < 4; ++i) t.emplace_back(worker, i);
    for (auto& x : t) x.join();
    std::printf("%s\n", bad || bad_release || used ? "BAD" : "OK");
    return 0;
}
'''


def run(tmp_path, source, tsan=False):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(source)
    base = ["g++", "-std=c++17", "-O1", "-g", "-pthread", "-I", CSRC, str(src), "-o", str(exe)]
    if not tsan or subprocess.run(base + ["-fsanitize=thread"], capture_output=True).returncode != 0:
        subprocess.run(base, check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout + out.stderr[:2000]
    assert "WARNING: ThreadSanitizer" not in out.stderr, out.stderr[:2000]


def test_work_memory_is_reused_bounded_and_given_back(tmp_path):
    run(tmp_path, DRIVER)


def test_work_memory_with_concurrent_calls(tmp_path):
    run(tmp_path, THREADS, tsan=True)
