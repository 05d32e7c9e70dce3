"""One event a batched update (lpma_gb300/csrc/spare_ring.h), without a GPU.

The graphs of a batched update share the event recorded behind their work and
hold it until their next one; lpma_destroy waits for it.  An event that a graph
still holds must not be recorded again by a later call, which may run on
another stream and for other graphs.  The bookkeeping is host-only C++, tested
here with counted stand-ins for the events."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "spare_ring.h"
using namespace lpma;
static int live = 0;
struct Ev { int call = 0; Ev() { live++; } ~Ev() { live--; } };
#define CHECK(c) do { if (!(c)) { std::printf("FAIL %s line %d\n", #c, __LINE__); return 1; } } while (0)
int main() {
    std::shared_ptr<Ev> A, B, C;  // what three graphs hold
    {
        SpareRing<Ev> r;
        int n = 0;
        auto make = [&] { n++; return std::make_shared<Ev>(); };
        auto call = [&](int k, std::initializer_list<std::shared_ptr<Ev> *> graphs) {
            std::shared_ptr<Ev> e = r.take(make);
            for (auto *g : graphs) *g = e;
            e->call = k;  // recorded behind the call's work
        };
        call(1, {&A});
        call(2, {&B});
        CHECK(A->call == 1 && B->call == 2);          // A's event still stands for its own call
        call(3, {&B, &C});
        CHECK(A->call == 1 && B->call == 3 && C == B);
        // the same graphs call after call: two events in turn, none made
        const int made = n;
        for (int k = 4; k < 100; k++) {
            call(k, {&B, &C});
            CHECK(A->call == 1 && B->call == k && C->call == k);
        }
        CHECK(n == made && (int)r.size() == n && n == 3);
        A.reset();                                     // a graph destroyed: its event is free again
        call(100, {&A, &B, &C});
        CHECK(n == made);
        CHECK(r.take([&] { return std::shared_ptr<Ev>(); }) != nullptr);  // spare ones first
        SpareRing<Ev> none;
        CHECK(none.take([&] { return std::shared_ptr<Ev>(); }) == nullptr && none.size() == 0);  // a failure is not kept
    }
    CHECK(live == 1 && A->call == 100);                // held events outlive the ring
    A.reset(), B.reset(), C.reset();
    CHECK(live == 0);
    std::printf("ok\n");
    return 0;
}
"""


def test_a_held_event_is_not_given_out_again(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "sr.cpp", tmp_path / "sr"
    src.write_text(PROGRAM)
    subprocess.check_call([gxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "lpma_gb300", "csrc"), str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr


def test_batched_updates_take_their_event_from_the_ring():
    abi = open(os.path.join(ROOT, "lpma_gb300", "csrc", "abi.cu")).read()
    assert "SpareRing<BatchEvent>" in abi and "events.take" in abi
    assert abi.count("shared_ptr<BatchEvent> all;") == 1  # a call's own, not the batcher's
