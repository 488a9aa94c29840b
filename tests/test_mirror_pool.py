"""The idle-buffer bookkeeping of the step calls' device mirrors and scratch
(csrc/se_mirror_pool.h), compiled for the host with a counting allocator: a
buffer released on one device is never handed out on another, is reused on its
own, and what is idle beyond the limit is freed per device."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <set>
#include "se_mirror_pool.h"

static std::set<void*> live;
static bool full = false;
struct Buffers {
    static int alloc(void** p, size_t)
    {
        if (full) return 7;
        live.insert(*p = malloc(1));
        return 0;
    }
    static void free(void* p) { live.erase(p); ::free(p); }
};
#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int main()
{
    se::MirrorPool<Buffers> pool(1000);
    void *a = nullptr, *b = nullptr, *c = nullptr;
    size_t cap = 0;
    CHECK(pool.acquire(0, 100, &a, &cap) == 0 && cap == 100);
    pool.release(0, a, cap);
    CHECK(pool.acquire(1, 100, &b, &cap) == 0 && b != a);      // the other device's buffer stays idle
    CHECK(pool.acquire(0, 60, &c, &cap) == 0 && c == a && cap == 100);
    pool.release(0, c, cap);
    CHECK(pool.acquire(0, 49, &c, &cap) == 0 && c != a && cap == 49);   // more than twice the size
    pool.release(0, c, cap);
    pool.release(1, b, 100);
    CHECK(pool.acquire(1, 900, &b, &cap) == 0);
    pool.release(1, b, cap);
    CHECK(live.size() == 4);                                   // 149 idle on device 0, 1000 on device 1
    CHECK(pool.acquire(1, 10, &b, &cap) == 0);
    pool.release(1, b, cap);
    CHECK(live.size() == 4 && !live.count(nullptr));           // device 1's largest was freed
    CHECK(pool.acquire(0, 100, &c, &cap) == 0 && c == a);      // device 0 kept its own
    full = true;
    CHECK(pool.acquire(0, 100, &b, &cap) == 7);
    return 0;
}
"""


def test_buffers_stay_on_their_device(tmp_path):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "se_fast_gridding_b200", "csrc"),
                    str(src), "-o", str(exe), "-pthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
