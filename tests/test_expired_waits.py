"""What kernels do when a wait has run out, checked without a GPU: the wait functions of csrc/gemm_tc.cuh are compiled for
the host with a barrier that never completes, and the order of waits is read off the sources."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = os.path.join(ROOT, "colibri_b200", "csrc", "gemm_tc.cuh")

HARNESS = r"""
#include <cstdint>
#include <cstdio>
static long long polls, now;
static bool completes;
static inline bool mbar_try_wait(uint32_t, uint32_t) { polls++; now += 8000; return completes; }     // (cycles a try suspends)
static inline long long clock64() { return now; }
#define __device__
#define __forceinline__ inline
@FUNCTIONS@
int main() {
    volatile int abort_flag = 0;
    bool dead = false;
    completes = true;
    tc_wait_light(0, 0, &abort_flag, dead);
    if (dead || polls != 1) { std::printf("a wait that is over: dead %d, %lld polls\n", dead, polls); return 1; }
    completes = false; now = 0;
    tc_wait_light(0, 0, &abort_flag, dead);
    if (!dead || !abort_flag || now > 450000000LL) { std::printf("no end: dead %d, abort %d, %lld cycles\n", dead, abort_flag, now); return 1; }
    polls = 0;                                                                    // the waits left of a partial sum: one try each
    for (int i = 0; i < 6; i++) tc_wait_light(0, 0, &abort_flag, dead);
    if (polls > 6) { std::printf("%lld polls by a warp that has given up\n", polls); return 1; }
    polls = 0;
    bool other = false;                                                           // another warp, after the abort flag
    for (int i = 0; i < 6; i++) tc_wait_light(0, 0, &abort_flag, other);
    if (!other || polls > 7) { std::printf("%lld polls after another warp gave up\n", polls); return 1; }
    std::puts("ok");
}
"""


def function(text, name):
    m = re.search(r"^__device__ __forceinline__ \w+ " + name + r"\(.*?^}\n", text, re.M | re.S)
    assert m, name
    return m.group(0)


def test_an_expired_wait_is_not_waited_for_again(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    text = open(SOURCE).read()
    code = HARNESS.replace("@FUNCTIONS@", function(text, "tc_wait_slow") + function(text, "tc_wait_light"))
    (tmp_path / "waits.cpp").write_text(code)
    exe = str(tmp_path / "waits")
    subprocess.check_call([gxx, "-std=c++17", "-O1", "-o", exe, str(tmp_path / "waits.cpp")])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_decode_warps_leave_when_a_wait_has_expired():
    """The decode role's loops over tasks and partial sums end behind an expired wait of any lane, all lanes together. (Walking
    on, every one of thousands of waits would suspend the warp once more.)"""
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    role = text[text.index("if (warp >= TC_DEC_WARP0) {"):text.index("} else if (warp >= TC_EPI_WARP0) {")]
    loops = re.findall(r"(?:while|for) \([^\n]*(?:ntask|nflush)[^\n]*\) \{", role)
    assert len(loops) == 2 and all("!gone" in loop for loop in loops), loops
    flush = role[role.index(loops[1]):]
    assert re.search(r"gone = __any_sync\(0xffffffffu, dead\);", flush)


def test_copies_and_mmas_in_flight_are_waited_for_whoever_gave_up():
    """What a role has started is waited for by that role, not only when it gave up itself: the roles that would have
    waited for it may have."""
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    kernel = text[text.index("k_expert_gemm_tc(TcArgs a)"):]
    drains = [m.start() for m in re.finditer(r"mbar_wait_bounded\(", kernel)]
    assert len(drains) == 3                                  # MMAs; weight copies; activation copies
    for at in drains:
        before = kernel[:at]
        head = before[before.rindex("while (ct.task < ntask"):]
        tail = head[max(head.rfind("if (dead) break;"), head.rfind("umma_commit(bar_acc_full")):]
        assert "if (dead)" not in tail.replace("if (dead) break;", ""), tail


def test_a_raw_slot_is_given_back_behind_completed_stores():
    """The arrival that lets the next copy into a raw slot comes behind the wait for the tensor-memory stores, which need every
    word read from the slot, and behind a barrier of the warp, whose other lanes read from it too."""
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    role = text[text.index("if (warp >= TC_DEC_WARP0) {"):text.index("} else if (warp >= TC_EPI_WARP0) {")]
    arrive = [m.start() for m in re.finditer(r"mbar_arrive\([^;]*TC_BAR_RAW_EMPTY", role)]
    assert len(arrive) == 1
    stored = role.rindex("tmem_st_frag16(")
    waited = role.index("tcgen05.wait::st", stored)
    assert waited < role.index("__syncwarp()", waited) < arrive[0]


def test_router_waits_once_for_copies_that_do_not_come():
    """The chains of the router kernel wait for no tile after one that did not come (a wait per tile would add up to the limit times
    the tiles), and the copy warp, whose copies they then do not wait for, does so itself before it leaves."""
    text = open(os.path.join(ROOT, "colibri_b200", "csrc", "router.cuh")).read()
    kernel = re.sub(r"//[^\n]*", "", text[text.index("k_router_logits("):text.index("__global__ void k_router_logits_any")])
    copies, chains = kernel[:kernel.index("return;")], kernel[kernel.index("return;"):]
    assert re.search(r"for \(int i = max\(0, t - NS\); i < t; i\+\+\) mbar_wait_bounded\(smem_u32\(s_full \+ i % NS\), \(i / NS\) & 1\);\s*$", copies)
    assert re.findall(r"if \(([^\n]*?)!mbar_wait_bounded", chains) == ["ok && "]
