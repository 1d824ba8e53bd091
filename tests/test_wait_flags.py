"""The error words of concurrent calls (csrc/wait_flags.hpp): each call sees what
its own kernel raised, whatever calls begin and end beside it. Compiled for the
host; the kernels' part is played by plain stores."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "anc-field_b200", "csrc")
MAIN = r"""
#include <atomic>
#include <cstdio>
#include <memory>
#include <stdexcept>
#include <thread>
#include "wait_flags.hpp"

using afd::WaitFlags;
static std::atomic<int> made{0};
static bool refuse = false;
static int* make() {
    if (refuse) throw std::runtime_error("no memory");
    ++made;
    return new int(7);
}
#define CHECK(x) if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; }

int main() {
    WaitFlags flags(make);
    {
        // a call begins while another call's kernel has raised its word
        WaitFlags::Lease a(flags);
        *a.word() |= 1;
        WaitFlags::Lease b(flags);
        CHECK(a.word() != b.word());
        CHECK(a.raised() && !b.raised());
        *b.word() |= 1;
        { WaitFlags::Lease c(flags); CHECK(!c.raised()); }
        CHECK(a.raised() && b.raised());
    }
    // words come back cleared and are used again
    for (int k = 0; k < 100; ++k) {
        WaitFlags::Lease a(flags), b(flags);
        CHECK(!a.raised() && !b.raised());
        *a.word() = *b.word() = 1;
    }
    CHECK(made == 3);
    {
        // no word to be had: the call fails, those in flight and later ones do not
        WaitFlags::Lease a(flags), b(flags), c(flags);
        refuse = true;
        bool threw = false;
        try { WaitFlags::Lease d(flags); } catch (const std::runtime_error&) { threw = true; }
        CHECK(threw);
        refuse = false;
        WaitFlags::Lease d(flags);
        CHECK(made == 4 && !d.raised());
    }
    std::atomic<int> wrong{0};
    auto work = [&](int odd) {
        for (int k = 0; k < 20000; ++k) {
            WaitFlags::Lease a(flags);
            if (k % 2 == odd) *a.word() |= 1;
            if (a.raised() != (k % 2 == odd)) ++wrong;
        }
    };
    std::thread t[4];
    for (int k = 0; k < 4; ++k) t[k] = std::thread(work, k & 1);
    for (auto& q : t) q.join();
    CHECK(wrong == 0 && made <= 8);
    printf("ok\n");
}
"""


def test_each_call_has_its_own_word(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "flags.cpp", tmp_path / "flags"
    src.write_text(MAIN)
    subprocess.run([cxx, "-O1", "-std=c++17", "-pthread", "-Wall", "-Werror", "-I", CSRC, "-o", str(exe), str(src)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
