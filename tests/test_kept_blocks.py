"""The device's kept blocks (csrc/blockcache.h) over a device made of counters: what an idle handle gave
back serves another handle's allocation and is given up when an allocation is refused; the bound holds
over all handles together; no block is handed out or freed twice."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include <set>
#include <utility>
#include "blockcache.h"

// stream: an id.  event: an id, with the stream's count of work at its record; work passes by settle()
static std::map<int, long> queued, done;
static std::map<int, std::pair<int, long>> events;
static std::set<void*> live, freed;
static int waits = 0;
struct Api {
    using Stream = int;
    using Event = int;
    static bool create(Event& e) { e = (int)events.size(); events[e] = {0, 0}; return true; }
    static bool record(Event e, Stream s) { events[e] = {s, queued[s]}; return true; }
    static bool passed(Event e) { return done[events[e].first] >= events[e].second; }
    static void wait(Stream, Event e) { waits += !passed(e); }
    static void free(void* p, Stream) {
        if (!live.erase(p)) { std::printf("freed twice\n"); std::exit(1); }
        freed.insert(p);
    }
};
static void settle(int s) { done[s] = queued[s]; }
static char arena[1 << 16];
static size_t used = 0;
static void* fresh() { void* p = arena + used++; live.insert(p); return p; }
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    const size_t MB = 1 << 20;
    const int A = 1, B = 2;                      // two handles, their streams, and their owner names
    const void *a = &arena[0], *b = &arena[1];
    size_t got = 0;
    {
        momed::KeptBlocks<Api> k(100 * MB);
        void* p = fresh();
        queued[A] = 1;                           // work of A in flight as it gives the block back
        CHECK(k.put(p, 40 * MB, a, A) && k.held() == 40 * MB);
        CHECK(!k.take(40 * MB, b, got));      // not to B while that work runs
        CHECK(k.take(40 * MB, a, got) == p && got == 40 * MB && k.held() == 0);
        CHECK(k.put(p, 40 * MB, a, A));
        settle(A);
        CHECK(!k.take(41 * MB, b, got));
        CHECK(k.take(33 * MB, b, got) == p && got == 40 * MB);   // an idle handle's block serves B
        CHECK(k.put(p, 40 * MB, b, B));
        CHECK(!k.take(31 * MB, a, got) && k.held() == 40 * MB);   // more than a quarter larger: stays
    }
    {
        momed::KeptBlocks<Api> k(100 * MB);      // a refused allocation of B gets A's blocks, behind A's work
        void *p = fresh(), *q = fresh();
        queued[A] = 5;
        CHECK(k.put(p, 50 * MB, a, A) && k.put(q, 30 * MB, a, A));
        waits = 0;
        CHECK(k.reclaim(B) && waits == 2 && k.held() == 0 && freed.count(p) && freed.count(q));
        CHECK(!k.reclaim(B));
        settle(A);
    }
    {
        momed::KeptBlocks<Api> k(100 * MB);      // one bound for all handles, the oldest leave first
        void *p = fresh(), *q = fresh(), *r = fresh(), *s = fresh();
        CHECK(k.put(p, 60 * MB, a, A) && k.put(q, 30 * MB, b, B) && k.put(r, 50 * MB, b, B));
        CHECK(k.held() == 80 * MB && freed.count(p));
        queued[B] = 9;
        CHECK(!k.put(s, 101 * MB, a, A) && !k.put(s, MB / 2, a, A));
        live.erase(s);
        k.drop(b, B);                            // a closing handle takes its own
        CHECK(k.held() == 0 && freed.count(q) && freed.count(r));
        settle(B);
    }
    std::mt19937 rng(1);
    momed::KeptBlocks<Api> k(200 * MB);
    std::map<void*, std::pair<size_t, int>> out; // blocks in use: size, handle
    live.clear();
    for (int t = 0; t < 20000; ++t) {
        const int h = 1 + rng() % 3;
        const void* o = &arena[h];
        switch (rng() % 8) {
            case 0: settle(h); break;
            case 1: if (rng() % 50 == 0) k.drop(o, h); break;
            case 2: if (rng() % 100 == 0) k.reclaim(h); break;
            case 3: case 4: case 5: {
                const size_t n = MB + rng() % (40 * MB);
                void* p = k.take(n, o, got);
                if (p) {
                    CHECK(!out.count(p) && live.count(p) && got >= n && got <= n + n / 4);
                } else {
                    if (used >= sizeof arena) break;
                    p = fresh();
                    got = n;
                }
                out[p] = {got, h};
                ++queued[h];
                break;
            }
            default:
                if (!out.empty()) {
                    auto it = out.begin();
                    std::advance(it, rng() % out.size());
                    const auto v = *it;
                    out.erase(it);
                    if (!k.put(v.first, v.second.first, &arena[v.second.second], v.second.second)) Api::free(v.first, 0);
                }
        }
        CHECK(k.held() <= 200 * MB);
        for (const auto& v : out) CHECK(live.count(v.first));
    }
    k.reclaim(1);
    CHECK(k.held() == 0 && live.size() == out.size());
    return 0;
}
"""


def test_accounting_of_kept_blocks(tmp_path):
    src, exe = tmp_path / "kept.cpp", tmp_path / "kept"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "momentumed.jl_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
def test_a_second_handle_solves_in_what_the_first_gave_back():
    """Two open handles, the same sweep on one and then on the other: the second maps little new memory."""
    import momed
    import torch
    from momed.core import pair_operator
    from momed.synthetic import mesh_para, u_grid

    para, _ = mesh_para(3, 8, 1)
    A = momed.MBOperator(momed.ED_scatterlist_onebody(para), upper_hermitian=True)
    B = momed.MBOperator(momed.ED_scatterlist_twobody(para), upper_hermitian=True)
    pair = pair_operator(A, B)
    handles = [momed.Handle(0) for _ in range(2)]
    basis = handles[0].enumerate_basis(para.k_list, para.Gk, 1, 1, (8,))[2][1]
    for h in handles:
        h.set_basis(basis)
        h.set_scatter_pair(*pair)
    free = [torch.cuda.mem_get_info()[0]]
    vals = []
    for h in handles:
        vals.append(h.batch_solve(u_grid(32, 0.5, 2.0), 4, krylovdim=60, tol=1e-12)[0])
        free.append(torch.cuda.mem_get_info()[0])
    for h in handles:
        h.close()
    first, second = free[0] - free[1], free[1] - free[2]
    assert first > 256 << 20                   # 30.6k states x 32 in 61 FP64 columns: 0.96 GB
    assert second < first / 2
    assert np.max(np.abs(vals[0] - vals[1]) / np.abs(vals[0])) < 1e-11
