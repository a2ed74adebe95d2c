"""Byte offsets of the neighbour search's slots (csrc/sph_slots.h), on the host:
both forms give 16 bytes per slot over two ranges of slots, entered anywhere, and
the one with 32 bits is chosen only where its offsets do not wrap."""
import os
import subprocess

import pytest

from conftest import ROOT

SOURCE = r"""
#include <cstdio>
#include "sph_slots.h"
using namespace sph;

template <typename Off>
static bool walks(unsigned s1, unsigned n1, unsigned s2, unsigned n2)
{
    for (unsigned k = 0; k <= n1 + n2; ++k) {
        SlotWalk<Off> w(s1, n1, s2, k);
        for (unsigned j = k; j < n1 + n2; ++j, w.advance()) {
            const unsigned long long slot = j < n1 ? s1 + j : s2 + (j - n1);
            if ((unsigned long long)w.at != 16 * slot) return false;
        }
    }
    return true;
}

int main()
{
    const unsigned cases[][4] = {{0, 0, 0, 0}, {0, 5, 5, 3}, {7, 3, 40, 9}, {7, 0, 40, 9}, {7, 4, 0, 0}};
    for (const auto& c : cases)
        if (!walks<unsigned>(c[0], c[1], c[2], c[3]) || !walks<unsigned long long>(c[0], c[1], c[2], c[3])) return 1;
    const unsigned top = 1u << 28;
    if (!walks<unsigned>(top - 40, 9, top - 7, 7)) return 2;  /* the last slots that 32 bits reach */
    if (walks<unsigned>(top - 3, 9, top + 20, 7)) return 3;   /* and the first that they do not */
    const unsigned high[][4] = {{top - 3, 9, top + 20, 7}, {top + 5, 0, top + 9, 4}, {0x7ffffff0u, 8, 0x7ffffffcu, 3}};
    for (const auto& c : high)
        if (!walks<unsigned long long>(c[0], c[1], c[2], c[3])) return 4;
    if (!narrow_slots(top, top) || narrow_slots(top + 1, 1) || narrow_slots(1, top + 1)) return 5;
    std::puts("ok");
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("slots")
    (d / "slots.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "sph2o_b200", "csrc"),
                    str(d / "slots.cpp"), "-o", str(d / "slots")], check=True)
    return str(d / "slots")


def test_offsets_of_slots(program):
    r = subprocess.run([program], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.returncode
