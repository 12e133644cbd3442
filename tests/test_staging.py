"""Memory that a step's results pass through (csrc/staging.h), in a host program whose source of memory refuses: nothing is lost, and a step whose results find no room
there is told so (it brings them by copies then)."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bpd_substrate_b200", "csrc")

PROGRAM = r"""
#include "staging.h"
#include <cstdio>
#include <cstdlib>
static int taken, given;
static size_t limit = 100;
static void* take(size_t n) { return n > limit ? nullptr : (taken++, std::malloc(n)); }
static void give(void* p) { given++; std::free(p); }
int main()
{
    bpdq::Staging s;
    if (s.reserve(101, take, give) || s.base || s.bytes) return 1;                  // refused at once
    if (!s.reserve(0, take, give) || s.base || taken) return 2;
    if (!s.reserve(40, take, give) || !s.base || s.bytes != 40) return 3;
    s.base[39] = 7;
    uint8_t* was = s.base;
    if (s.reserve(200, take, give) || s.base != was || s.bytes != 40 || s.base[39] != 7 || given) return 4;      // refused: what there is stays
    if (!s.reserve(40, take, give) || !s.reserve(1, take, give) || taken != 1) return 5;
    if (!s.reserve(100, take, give) || s.bytes != 100 || taken != 2 || given != 1) return 6;
    give(s.base);
    std::puts("ok");
    return 0;
}
"""


def test_refusals(tmp_path):
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-fsanitize=address", "-g", "-I", CSRC, str(src), "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stderr)
