"""Kernels that give up waiting for a copy wait for every other one that is on its way, so that none lands in shared memory that has gone to another block.  No
wait runs out on a GPU here: the loops that do this are taken from the kernels' sources, compiled for the host and held against a replay of the copies."""
import os
import re
import subprocess

import pytest

import infr_b200


def _loop(source, pattern):
    with open(os.path.join(os.path.dirname(infr_b200.__file__), "csrc", source)) as f:
        return re.search(pattern, f.read(), re.S).group(1)


def _run(tmp_path, program):
    src, exe = tmp_path / "ring.cpp", tmp_path / "ring"
    src.write_text(program)
    subprocess.run(["g++", "-std=c++17", str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout


ROUTER = r"""
#include <cstdio>

// a ring of chunks at once, then one more for each chunk that lands after the first
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

ITEMS = r"""
#include <cstdio>
#include <cstdint>

// tile i in slot i % slots, asked for when tile i - slots has been read: a slot's last tile is any of its own
int main() {
    int left = 0;
    for (int slots = 4; slots <= 16; slots++)
        for (int n = 0; n <= 3 * slots; n++) {
            int s_tile[16], waited[16], parity[16], bars[16];
            for (int s = 0; s < slots; s++) s_tile[s] = -1, waited[s] = 0;
            for (int i = 0; i < n; i++) s_tile[i % slots] = i;
            auto sm6 = [&](int *b) { return (int)(b - bars); };
            auto wait_parity6 = [&](int s, uint32_t p) { waited[s]++, parity[s] = (int)p; };
            for (int lane = 0; lane < 32; lane++) {
                LOOP
            }
            for (int s = 0; s < slots; s++) {
                int uses = 0;  // of the slot: its last copy completes phase uses - 1
                for (int i = s; i < n; i += slots) uses++;
                left += waited[s] != (uses > 0) || (uses && parity[s] != ((uses - 1) & 1));
            }
        }
    std::printf("%d\n", left);
}
"""


def test_router(tmp_path):
    assert _run(tmp_path, ROUTER.replace("LOOP", _loop("moe.cu", r"atomicExch\(status, 14u\);\s*(for \(.*?landed\(c\);)"))) == "0\n"


def test_expert_items_q6k(tmp_path):
    assert _run(tmp_path, ITEMS.replace("LOOP", _loop("gemv_mma_q6.cu", r"if \(s_dead\)\s*(for \(.*?& 1u\);)"))) == "0\n"


WARP = r"""
#include <cstdio>
#include <cstdint>

// a warp's ring: copy j in slot j % slots; when the wait for one runs out, it and those behind it are on their way, no more than there are slots
int main() {
    int left = 0;
    for (int slots = 1; slots <= 12; slots++)
        for (int asked = 0; asked <= 4 * slots; asked++) {
            uint64_t bars[12];
            int waited[12] = {}, uses[12] = {};
            for (int j = 0; j < asked; j++) uses[j % slots]++;  // a slot's last copy completes phase uses - 1
            auto __cvta_generic_to_shared = [&](uint64_t *b) { return (uint64_t)(b - bars); };
            LOOP
                left += waited[bar]++ || parity != ((uint32_t)(uses[bar] - 1) & 1u);
            }
            for (int s = 0; s < slots; s++) left += waited[s] != (uses[s] > 0);
        }
    std::printf("%d\n", left);
}
"""


def test_ring_of_a_warp(tmp_path):
    assert _run(tmp_path, WARP.replace("LOOP", _loop("gemv_common.cuh", r"drain_ring\(.*?\{\n(.*?)\n\s*for \(uint32_t i"))) == "0\n"


@pytest.mark.parametrize("source", ["gemv_mma.cu", "gemv_mma_q2.cu", "gemv_mma_q6.cu", "gemv_wide.cu"])
def test_rings_of_warps_are_drained(source):
    # a warp that has given up asks for nothing more, and its kernel ends with the wait for what it had asked for
    body = _loop(source, r"auto issue = \[&\]\(int slot\) \{(.*?\n\}\n)")
    gives_up = _loop(source, r"if \(!dead && !\w+\(\w+\(wbar \+ slot\), phase\)\) \{(.*?)\n            \}\n")
    assert body.lstrip().startswith("if (j_issue >= n_jobs) return;")
    if "n_jobs = j_issue;" in gives_up:
        assert body.endswith("    if (dead) drain_ring(wbar, S, j_issue);\n}\n")
    else:
        assert "s_asked[warp] = j_issue, j_issue = n_jobs;" in gives_up and body.endswith("    if (dead) drain_ring(wbar, S, s_asked[warp]);\n}\n")


def test_gemm_producer_is_drained():
    assert re.match(r"[^\n]*\n\s*drain_ring\(bars, kStages, j\);\s*return;", _loop("mmq.cu", r"(if \(\*\(volatile int \*\)&s_dead\) .*)"))
