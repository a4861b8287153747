"""A kernel that gives up waiting for a chunk of its ring (the MoE router) waits for every other copy that is on its way.  The bound of that loop is taken from the
kernel's source, compiled for the host, and held against a replay of the copies: a ring of chunks at once, then one more for each that lands after the first."""
import os
import re
import subprocess

import infr_b200

PROGRAM = r"""
#include <cstdio>

int main() {
    int left = 0;
    for (int kRtRing = 2; kRtRing <= 5; kRtRing++)
        for (int n_chunks = 1; n_chunks <= 12; n_chunks++)
            for (int c0 = 0; c0 < n_chunks; c0++) {
                int asked = kRtRing, waited = c0;
                for (int c = 1; c < c0; c++) asked++;
                auto landed = [&](int c) { waited = c; };
                LOOP
                left += waited + 1 != (asked < n_chunks ? asked : n_chunks);
            }
    std::printf("%d\n", left);
}
"""


def test_no_copy_is_left_behind(tmp_path):
    with open(os.path.join(os.path.dirname(infr_b200.__file__), "csrc", "moe.cu")) as f:
        loop = re.search(r"atomicExch\(status, 14u\);\s*(for \(.*?landed\(c\);)", f.read(), re.S)
    src, exe = tmp_path / "ring.cpp", tmp_path / "ring"
    src.write_text(PROGRAM.replace("LOOP", loop.group(1)))
    subprocess.run(["g++", "-std=c++17", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "0\n"
