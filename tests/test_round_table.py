"""The table of captured rounds: what it holds, and which round goes when it is full.  Compiled for the host."""
import os
import random
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llama.cu_b200", "csrc")

MAIN = r"""
#include <cstdio>
#include "round_table.hpp"
int main() {  // the size, then the keys that are asked for in turn; prints hits, and what was dropped with a minus
    int most, key, hits = 0;
    if (scanf("%d", &most) != 1) return 1;
    auto drop = [](int &v) { printf("-%d ", v); };
    lcu::RoundTable<int, decltype(drop)> t(most, drop);
    while (scanf("%d", &key) == 1) {
        int *v = t.find({key, 1});
        if (v) ++hits; else v = t.insert({key, 1}, key);
        if (*v != key || (int)t.size() > most) return 2;
    }
    printf("%d\n", hits);
    t.clear();
    printf("\n");
    return t.size() ? 3 : 0;
}
"""


def test_least_recently_used_goes(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, str(tmp_path / "main.cpp"), "-o", str(tmp_path / "main")], check=True)

    def ask(most, keys):
        r = subprocess.run([str(tmp_path / "main")], input=" ".join(map(str, [most, *keys])), capture_output=True, text=True, check=True)
        a, b = r.stdout.split("\n")[:2]
        return [-int(x) for x in a.split()[:-1]], int(a.split()[-1]), sorted(-int(x) for x in b.split())
    assert ask(3, [1, 2, 3, 1, 4, 1, 2, 4]) == ([2, 3], 3, [1, 2, 4])
    # three output buffers, 30 batch sizes, two splits that the service moves between: all stay captured (the whole table of 96 went)
    assert ask(200, [i % 180 for i in range(1000)])[:2] == ([], 820)
    rng, held, dropped, hits = random.Random(3), [], [], 0
    keys = [rng.randrange(30) for _ in range(500)]
    for k in keys:
        if k in held:
            held.remove(k)
            hits += 1
        elif len(held) == 12:
            dropped.append(held.pop(0))
        held.append(k)
    assert ask(12, keys) == (dropped, hits, sorted(held))
