"""Results on their way to the caller's arrays: host logic, compiled with a runtime that copies when it is waited for."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gw_fopt_b200", "csrc")

PROLOGUE = r"""
#include "readback.h"
#include <cstdio>
#include <cstdlib>
#include <stdexcept>
#include <vector>
#define EXPECT(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); std::exit(1); } } while (0)
struct Queue {
    struct Copy { void* dst; const void* src; size_t bytes; };
    std::vector<Copy> queued;
    int waits = 0;
    bool fail = false;
};
struct Rt {
    Queue* q;
    void* block;
    void* take() { return block; }
    void give(void*) {}
    void copy(void* dst, const void* src, size_t bytes) { q->queued.push_back({dst, src, bytes}); }
    void wait() {
        ++q->waits;
        if (q->fail) throw std::runtime_error("lost");
        for (auto& c : q->queued) std::memcpy(c.dst, c.src, c.bytes);
        q->queued.clear();
    }
};
using R = bgw::Readback<Rt>;
const size_t kLarge = R::kBytes + 8;
"""


def run(tmp_path, body):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.fail("no C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROLOGUE + body)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)],
                   check=True)
    got = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert got.returncode == 0, got.stdout + got.stderr


# A call whose status is bad, or whose work is lost, leaves the caller's arrays alone: results that pass through
# the staging block and results that are copied directly.
def test_a_failed_call_leaves_the_outputs_alone(tmp_path):
    run(tmp_path, r"""
int main() {
    std::vector<char> block(R::kBytes), large(kLarge, 'x'), small(16, 'x'), dev(kLarge, 'd');
    const std::vector<char> large0 = large, small0 = small;
    for (int lost = 0; lost < 2; ++lost) {
        Queue q;
        q.fail = lost;
        unsigned status = 0;
        const unsigned bad = 7;
        R r(Rt{&q, block.data()});
        r.status(&status, &bad, sizeof bad);
        r.add(small.data(), dev.data(), small.size());
        r.add(large.data(), dev.data(), large.size());
        bool thrown = false;
        try {
            r.wait([&] { if (status) throw std::runtime_error("bad"); });
        } catch (const std::runtime_error&) {
            thrown = true;
        }
        EXPECT(thrown && status == (lost ? 0u : 7u));
        EXPECT(small == small0 && large == large0);
        for (auto& c : q.queued) EXPECT(c.dst >= block.data() && c.dst < block.data() + block.size());
    }
}
""")


# Everything arrives, in one wait without a large result under a status, and the block serves the next call.
def test_results_arrive(tmp_path):
    run(tmp_path, r"""
int main() {
    std::vector<char> block(R::kBytes), dev(kLarge);
    for (size_t i = 0; i < dev.size(); ++i) dev[i] = (char)(i * 37 + 1);
    Queue q;
    R r(Rt{&q, block.data()});
    for (int status = 0; status < 2; ++status)
        for (int with_large = 0; with_large < 2; ++with_large) {
            std::vector<char> large(kLarge), whole(R::kBytes - 32), odd(13), rest(64);
            unsigned s = 0, ok = 1;
            q.waits = 0;
            if (status) r.status(&s, &ok, sizeof ok);
            r.add(odd.data(), dev.data() + 5, odd.size());
            if (with_large) r.add(large.data(), dev.data(), large.size());
            r.add(whole.data(), dev.data() + 1, whole.size());  // does not fit beside what is staged
            r.add(rest.data(), dev.data() + 9, rest.size());
            int looked = 0;
            r.wait([&] { ++looked; });
            EXPECT(looked == status && (!status || s == 1));
            EXPECT(!std::memcmp(odd.data(), dev.data() + 5, odd.size()));
            EXPECT(!std::memcmp(rest.data(), dev.data() + 9, rest.size()));
            EXPECT(!std::memcmp(whole.data(), dev.data() + 1, whole.size()));
            if (with_large) EXPECT(large == dev);
        }
    std::vector<char> a(R::kBytes);
    q.waits = 0;
    r.add(a.data(), dev.data(), a.size());
    r.wait();
    EXPECT(q.waits == 1 && !std::memcmp(a.data(), dev.data(), a.size()));
}
""")


# Staging blocks are shared by all handles: a block is in one call at a time, at most four wait, the rest are freed,
# and a call that ends by an error gives its block back only after its copies ended, or not at all.
def test_blocks_are_given_back(tmp_path):
    run(tmp_path, r"""
#include <atomic>
#include <set>
#include <thread>
bgw::BlockPool pool;
std::atomic<int> made{0}, freed{0};
struct Pooled : Rt {
    void* take() { return pool.take([] { ++made; return std::malloc(R::kBytes); }); }
    void give(void* b) { pool.give(b, [](void* p) { ++freed; std::free(p); }); }
};
using P = bgw::Readback<Pooled>;
int main() {
    std::vector<char> dev(4096, 'd');
    {   // one call after the other: one block
        for (int k = 0; k < 50; ++k) {
            Queue q;
            P r(Pooled{{&q, nullptr}});
            std::vector<char> a(100);
            r.add(a.data(), dev.data(), a.size());
            r.wait();
            EXPECT(a[99] == 'd');
        }
        EXPECT(made == 1 && freed == 0);
    }
    {   // six at once: six blocks, two of them freed afterwards
        std::set<void*> seen;
        std::vector<void*> held;
        for (int k = 0; k < 6; ++k) held.push_back(Pooled().take());
        seen.insert(held.begin(), held.end());
        EXPECT(seen.size() == 6 && made == 6);
        for (void* b : held) Pooled().give(b);
        EXPECT(freed == 2);
    }
    {   // not waited for: the copy has ended before the block goes back, or the block does not go back
        for (int lost = 0; lost < 2; ++lost) {
            Queue q;
            char a[8] = {0};
            {
                P r(Pooled{{&q, nullptr}});
                r.add(a, dev.data(), sizeof a);
                q.fail = lost;
            }
            EXPECT(q.waits == 1 && a[0] == 0);
            EXPECT(q.queued.empty() == !lost);
        }
        std::vector<void*> held;
        const int before = made;
        for (int k = 0; k < 4; ++k) held.push_back(Pooled().take());
        EXPECT(made == before + 1);  // three were left
        for (void* b : held) Pooled().give(b);
    }
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([t] {
            std::vector<char> mine(512, (char)('a' + t));
            for (int k = 0; k < 2000; ++k) {
                Queue q;
                P r(Pooled{{&q, nullptr}});
                std::vector<char> a(512);
                r.add(a.data(), mine.data(), a.size());
                std::this_thread::yield();
                r.wait();
                EXPECT(a == mine);
            }
        });
    for (auto& t : threads) t.join();
}
""")
