"""The helper threads that copy logits (csrc/copy_pool.h), on the CPU: everything is done once, whatever the number of helpers, also when
the caller is alone or finishes first, again and again, and a pool ends with its threads asleep."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sapient_b200", "csrc")
PROGRAM = r"""
#include "copy_pool.h"
#include <atomic>
#include <cstdio>

int main() {
    for (int helpers : {0, 1, 3, 7}) {
        sp::CopyPool pool;
        for (int round = 0; round < 2000; ++round) {
            const int n = round % 33;
            std::vector<std::atomic<int>> done(33);
            std::atomic<int> next{0}, inside{0};
            pool.run(round % 5 ? helpers : helpers / 2, [&] {
                inside.fetch_add(1);
                for (int g; (g = next.fetch_add(1)) < n;) done[g].fetch_add(1);
                inside.fetch_sub(1);
            });
            if (inside.load()) { std::printf("a helper is still at work\n"); return 1; }
            for (int i = 0; i < 33; ++i)
                if (done[i].load() != (i < n)) { std::printf("helpers %d round %d: piece %d done %d times\n", helpers, round, i, done[i].load()); return 1; }
        }
        if (pool.size() > helpers) { std::printf("%d threads for %d helpers\n", pool.size(), helpers); return 1; }
    }
    { sp::CopyPool never_used; }
    return 0;
}
"""


def test_every_piece_is_done_once_and_threads_end(tmp_path):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
