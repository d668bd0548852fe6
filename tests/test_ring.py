"""A block that gives up a wait leaves nothing of its own under way: what the persistent tcgen05 kernels wait for before they end."""
import re
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "delta_b200" / "csrc"

HARNESS = r'''
#include "ring.cuh"
#include <cstdio>
#include <vector>
// A ring of barriers as the hardware keeps them: a barrier counts its complete phases, and a wait for a parity is over when the phase in front of
// the current one has it.  Copies arrive as late as they may: only when somebody waits for their barrier, or the ring is used again.
int main() {
  for (int slots : {1, 2, 3, 4, 7})
    for (int asked = 0; asked < 4 * slots + 3; ++asked)
      for (int arrived = 0; arrived < (1 << (asked < slots ? asked : slots)); ++arrived) {      // which of the last uses have arrived by themselves
        std::vector<int> phases(slots, 0);
        int under_way = 0;
        for (int n = 0; n < asked; ++n) {
          const int left = asked - 1 - n;
          const bool late = left < slots && !(arrived >> left & 1);
          if (late) ++under_way; else ++phases[ring_slot(n, slots)];
        }
        std::vector<int> owed(slots, 0);
        for (int n = asked > slots ? asked - slots : 0; n < asked; ++n) owed[ring_slot(n, slots)] = n / slots + 1 - phases[ring_slot(n, slots)];
        const bool ok = ring_drain(asked, slots, [&](int s, unsigned parity) {
          if (((unsigned)(phases[s] - 1) & 1u) != parity) {      // not over: the copy that is owed arrives, or the wait gives up
            if (!owed[s]) return false;
            --owed[s]; ++phases[s]; --under_way;
          }
          return ((unsigned)(phases[s] - 1) & 1u) == parity;
        });
        if (!ok || under_way != 0) { printf("slots %d asked %d arrived %d: ok %d, %d under way\n", slots, asked, arrived, ok, under_way); return 1; }
      }
  int calls = 0;      // a wait that gives up ends the rest
  if (ring_drain(9, 4, [&](int, unsigned) { return ++calls < 2; }) || calls != 2) { printf("went on after a wait gave up\n"); return 1; }
  return 0;
}
'''


def test_ring_drain_leaves_nothing_under_way(tmp_path):
    (tmp_path / "ring.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), str(tmp_path / "ring.cpp"), "-o", str(tmp_path / "ring")], check=True)
    r = subprocess.run([str(tmp_path / "ring")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


# (kernel file, the calls that belong to the warp that copies, to the warps that multiply)
TWO_STAGES = ["s_full,", r"s_full \+ 8", "o_done,", r"o_done \+ 8"]


@pytest.mark.parametrize("name, copies, products", [("gemm_rows_tc.cu", ["full0"], ["empty0"]),
                                                    ("gemm_f32_tc.cu", ["wfull", "xfull"], ["xempty"]),
                                                    ("attention_rows_wide_tc.cu", ["q_full", "k_edge", "k_full"], ["s_full", "o_done"]),
                                                    ("attention_rows_tc.cu", ["q_full", "full,", r"full \+ 8", "v_edge"], TWO_STAGES),
                                                    ("attention_prefill_tc.cu", ["q_full", "full,", r"full \+ 8"], TWO_STAGES)])
def test_persistent_kernels_wait_for_what_they_started(name, copies, products):
    """Each warp that starts copies or products waits for their barriers on every way out: the calls stand behind its loop, under no condition
    on success, before the block's last barrier."""
    text = (CSRC / name).read_text()
    body = text[text.index("__global__"):text.index("tmem_dealloc")]
    for barrier in copies + products:
        calls = [m.start() for m in re.finditer(r"ring_drain\([^;]*?mbar_wait\(" + barrier, body)]
        assert len(calls) == 1, barrier
        line = body[body.rindex("\n", 0, calls[0]):calls[0]]
        assert "failed" not in line and "gave_up" not in line and "ok" not in line.split("//")[0], line
        assert body.rindex("__syncthreads") > calls[0]


def test_linear_attention_waits_for_each_product_it_issued():
    """Up to three products, each with a barrier that completes once: none is issued after a wait has given up, and the thread that issued them waits for every one
    of them before the block leaves.  (One barrier for all three was waited for by its parity: the first product's end passed for the third's.)"""
    text = re.sub(r"//[^\n]*", "", (CSRC / "decay_attention_tc.cu").read_text())
    most = int(re.search(r"constexpr int PRODUCTS = (\d+);", text).group(1))
    assert "done[PRODUCTS]" in text and re.search(r"for \(int p = 0; p < PRODUCTS; \+\+p\) mbar_init\(s2u\(&sh\.done\[p\]\), 1\)", text)
    assert len(re.findall(r"umma_commit\(", text)) == 1      # of issue_next, which counts what it issued
    body = text[text.index("void issue_next"):]
    body = body[:body.index("\n}")]
    assert re.search(r"failed == 0\)\) \{.*elect_one\(\).*umma_commit\(s2u\(&sh\.done\[issued\]\)\);\s*\}\s*\+\+issued;", body, re.S)
    for kernel in text.split("__global__")[1:]:
        assert len(re.findall(r"issue_next\(sh, issued,", kernel)) <= most
        assert len(re.findall(r"\bumma(?:_a_tmem)?\(", kernel)) == len(re.findall(r"issue_next\(", kernel))
        assert all(m == "issued" for m in re.findall(r"\bend\(sh, warp, lane, (\w+), err\)", kernel))
    end = text[text.index("void end("):]
    end = end[:end.index("\n}")]
    drain = re.search(r"ring_drain\(issued, PRODUCTS, [^;]*mbar_wait\(s2u\(&sh\.done\[p\]\), parity\)", end)
    assert drain and "failed" not in end[:drain.start()] and drain.end() < end.index("__syncthreads") < end.index("tmem_dealloc")
