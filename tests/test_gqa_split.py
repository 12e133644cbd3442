"""How the split attention deals keys over a cluster (csrc/gqa_split.h), in a host program, against the rule written out here a second time; and the contexts
that a decoded token of the Llama may have but the split kernel refuses, which then go step by step."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bpd_substrate_b200", "csrc")
LONGEST = 200 * 1024 // 4           # keys and head size of the longest cache of a Llama

PROGRAM = r"""
#include "gqa_split.h"
#include <cstdio>
int main()
{
    long clusters;
    int sees, R, D, largest;
    while (std::scanf("%ld %d %d %d %d", &clusters, &sees, &R, &D, &largest) == 5) {
        const bpdq::GqaSplit s = bpdq::gqa_split(clusters, sees, R, D, largest, 148);
        std::printf("%d %d %zu %d\n", s.ranks, s.stretch, s.smem, (int)s.fits);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    d = tmp_path_factory.mktemp("gqa_split")
    src, exe = d / "main.cpp", d / "main"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True, capture_output=True)

    def run(cases):
        r = subprocess.run([str(exe)], input="".join(" ".join(map(str, c)) + "\n" for c in cases), capture_output=True, text=True, timeout=60, check=True)
        return [tuple(map(int, line.split())) for line in r.stdout.splitlines()]
    return run


def expected(clusters, sees, R, D, largest):
    def smem(ranks):
        return 4 * (9 * R * D + -(-sees // ranks) * R)
    ranks = 1
    while ranks < largest and clusters * ranks < 148 and sees > 64 * ranks:
        ranks *= 2
    while ranks < largest and smem(ranks) > 96 * 1024:
        ranks *= 2
    return ranks, -(-sees // ranks), smem(ranks), int(smem(ranks) <= 96 * 1024)


def test_rule(split):
    cases = [(c, sees, R, D, largest) for c in (1, 8, 40, 148, 2000) for R in (1, 2, 4) for D in (64, 128) for largest in (8, 16)
             for sees in (65, 128, 129, 4001, 22000, 39936, 39937, 51072, 79872, 79873)]
    assert split(cases) == [expected(*c) for c in cases]


def test_contexts_of_a_decoded_token(split):
    """All that a forward allows with clusters of 16; with clusters of 8 not the longest of four heads of 128 on a key head."""
    for largest, refused in ((16, False), (8, True)):
        longest = LONGEST - 128
        (_, _, _, fits), (_, _, _, least) = split([(8, longest, 4, 128, largest), (8, 39936, 4, 128, largest)])
        assert bool(fits) != refused and least
