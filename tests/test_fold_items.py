"""The numbering of queued triangles' work items (rust-sloth_gb300/csrc/fold_items.h), on the
host at counts far beyond what a test can draw: a batch's frames share one queue, and with 512
items a large triangle the items pass 2^32 from 8,388,608 large triangles on."""
import random
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "rust-sloth_gb300" / "csrc"
PARTS, MID, OVERFLOW = 512, 8, 64

PROGRAM = r"""
#include <cstdio>
#include "fold_items.h"
using namespace sloth;
int main()
{
    unsigned kind, a, b, cap, whole;
    unsigned long long it;
    while (scanf("%u %u %u %u %u %llu", &kind, &a, &b, &cap, &whole, &it) == 6) {
        uint32_t part = 0;
        if (kind == 0) {
            const FoldItems<uint64_t> f(a, b, cap, whole != 0);
            const uint32_t q = f.entry(it, part);
            printf("%llu %llu %u %u\n", (unsigned long long)f.cut, (unsigned long long)f.all, q, part);
            if ((unsigned long long)a + b <= 1u << 20) {   // a draw's: the same in 32 bits
                const FoldItems<uint32_t> n(a, b, cap, whole != 0);
                uint32_t p2 = 0;
                if (n.entry((uint32_t)it, p2) != q || p2 != part || n.all != f.all || n.cut != f.cut) return 1;
            }
        } else {
            const OverflowItems f(a, b, cap);
            const uint32_t q = f.entry(it, part);
            printf("0 %llu %u %u\n", (unsigned long long)f.all, q, part);
        }
    }
}
"""


@pytest.fixture(scope="module")
def items(tmp_path_factory):
    d = tmp_path_factory.mktemp("items")
    (d / "items.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(CSRC), str(d / "items.cpp"), "-o", str(d / "items")], check=True)

    def ask(rows):
        out = subprocess.run([str(d / "items")], input="\n".join(" ".join(map(str, r)) for r in rows),
                             capture_output=True, text=True, check=True).stdout.split("\n")
        return [tuple(int(v) for v in line.split()) for line in out if line]
    return ask


def spread(n, rng):
    return sorted({0, 1, n // 2, n - 1, *(k for k in (2**32 - 1, 2**32, 2**32 + 1) if k < n),
                   *(rng.randrange(n) for _ in range(40))})


@pytest.mark.parametrize("large,mid", [(1, 0), (0, 1), (3, 5), (700, 31), (1048576, 0), (0, 1048576), (8388312, 10), (8388607, 0), (8388608, 3),
                                       (8400000, 900000), (20000000, 0), (0, 600000000), (2**31 - 2, 1)])
@pytest.mark.parametrize("whole", [0, 1])
def test_fold_items(items, large, mid, whole):
    """Every item is one (entry, part) in part-major order, exact past 2^32."""
    cap, rng = max(large + mid, 7), random.Random(large + mid)
    cut, per = large * PARTS, 1 if whole else MID
    its = spread(cut + mid * per, rng)
    for it, got in zip(its, items([(0, large, mid, cap, whole, it) for it in its])):
        if it < cut:
            want = (it % large, it // large)
        else:
            want = (cap - 1 - (it - cut) % mid, (it - cut) // mid)
        assert got == (cut, cut + mid * per, *want), it


@pytest.mark.parametrize("front,back", [(0, 1), (5, 3), (67108864, 0), (30000000, 60000000), (2**31 - 2, 1)])
def test_overflow_items(items, front, back):
    cap, rng = front + back + 2, random.Random(front)
    its = spread((front + back) * OVERFLOW, rng)
    for it, got in zip(its, items([(1, front, back, cap, 0, it) for it in its])):
        k = it // OVERFLOW
        want = (k if k < front else cap - 1 - (k - front), it % OVERFLOW)
        assert got == (0, (front + back) * OVERFLOW, *want), it
