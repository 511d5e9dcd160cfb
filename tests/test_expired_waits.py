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


RING = r"""
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <map>
#include <vector>
using std::max;
#define __device__
#define __forceinline__ inline
struct DecPass { const uint8_t *wg, *wu, *wd; };
struct DecShared { DecPass pass[4]; };
static int dec_div(int n, unsigned long long m) { return n / (int)m; }
// barriers of one arrival each, by address: copies pending in the present phase, phases ended
struct Bar { int arrived = 0, pending = 0; unsigned phase = 0; };
static std::map<uint32_t, Bar> bars;
static std::map<uint32_t, int> slot;                    // copies in flight into a ring address
static std::vector<std::pair<uint32_t, uint32_t>> flight;
static int faults = 0, late = 1 << 30, copies = 0, landed_behind = 0;
static void land(size_t k) {
    slot[flight[k].first]--;
    Bar &b = bars[flight[k].second];
    if (--b.pending == 0 && b.arrived == 1) { b.arrived = 0; b.phase++; }
    flight.erase(flight.begin() + k);
}
static void mbar_expect_tx(uint32_t bar, uint32_t) { if (bars[bar].arrived++) { std::puts("a second arrival in one phase"); faults++; } }
static void bulk_g2s(uint32_t dst, const void *, uint32_t, uint32_t bar) {
    if (slot[dst]++) { std::puts("a copy into a slot with one in flight"); faults++; }
    bars[bar].pending++; copies++;
    flight.push_back({dst, bar});
}
static bool ended(uint32_t bar, uint32_t parity) { return (bars[bar].phase & 1) != parity; }
static bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
    if (ended(bar, parity)) return true;
    for (size_t k = 0; k < flight.size(); k++)
        if (flight[k].second == bar) {
            if (late-- == 0) return false;              // this one is later than the limit; the next wait finds it landed
            land(k);
            return ended(bar, parity);
        }
    return false;
}
@FUNCTIONS@
int main() {
    const int CH = 64;
    DecShared sh{};
    for (int first = 0; first < 40; first++) {          // which wait expires
        bars.clear(); slot.clear(); flight.clear();
        late = first; copies = 0;
        DecPhase ph{};
        ph.which = 1; ph.nt = 1; ph.nkb = 8; ph.wpk = 1; ph.ng = 1; ph.mg_nt = 1; ph.u1 = 2; ph.cnt = 8; ph.npass = 2;
        WarpRing wr; DecIt it;
        wr.ok = true;
        wr.start(4096, 0, 3, CH);
        for (int phase = 0; phase < 2; phase++) {
            if (phase) {
                if (!wr.ok) dec_drain(wr);
                wr.start(wr.ring, 1024, 6, CH / 2);
                ph.which = 2;
            }
            dec_it_start<CH>(it, ph, &sh);
            if (!wr.ok) it.live = 0;
            for (int s = 0; s < wr.nst; s++) dec_issue_one<CH>(wr, it, ph, &sh, 1);
            for (int b = 0; b < (phase ? 16 : 32); b++) {
                const bool was = wr.ok;
                const int before = copies;
                dec_wait_chunk@ARGS@;
                dec_release_chunk(wr);
                dec_issue_one<CH>(wr, it, ph, &sh, 1);
                if (!was && copies != before) { std::puts("a copy started behind an expired wait"); faults++; }
            }
        }
        if (!wr.ok) dec_drain(wr);
        if (!flight.empty()) { std::printf("wait %d expired: %zu copies in flight at the end\n", first, flight.size()); faults++; }
        if (faults) return 1;
    }
    std::puts("ok");
}
"""


def test_the_fused_kernels_stream_ends_with_an_expired_wait(tmp_path):
    """The weight ring of the fused decode kernel (csrc/moe_decode.cuh) over both phases, with one wait after the other expiring:
    no copy goes to a slot, or is counted on a barrier, that has one in flight, and none is in flight at the end."""
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    text = open(os.path.join(ROOT, "colibri_b200", "csrc", "moe_decode.cuh")).read()
    code = text[text.index("struct DecPhase {"):text.index("// This CTA's contiguous share")]
    (tmp_path / "ring.cpp").write_text(RING.replace("@FUNCTIONS@", code).replace("@ARGS@", "(wr, it)"))
    exe = str(tmp_path / "ring")
    subprocess.check_call([gxx, "-std=c++17", "-O1", "-o", exe, str(tmp_path / "ring.cpp")])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
    assert re.search(r"if \(!wr\.ok\) dec_drain\(wr\);\s*wr\.start\([^;]*;\s*dec_it_start<CH>\(it, ph2, sh\);\s*if \(!wr\.ok\) it\.live = 0;", text)
    assert re.search(r"if \(nslot > 0 && !mbar_wait_bounded\(hbar, 0\)\) \{\s*wr\.ok = false; it\.live = 0;\s*mbar_wait_bounded\(hbar, 0\);", text)
    assert re.search(r"if \(sh->failed\) \{[^}]*dec_drain\(wr\);", text)


@pytest.mark.parametrize("name,wait,drain", [
    ("gemv_rows.cuh", r"if \(!mbar_try_wait\(bars \+ s \* 8, par\) && !\(ok && mbar_wait_bounded\(bars \+ s \* 8, par\)\)\) ok = false;",
     r"for \(int i = max\(0, n - ROWS_NST\); i < n; i\+\+\) mbar_wait_bounded\(bars \+ i % ROWS_NST \* 8, \(i / ROWS_NST\) & 1\);"),
    ("gemv_stream.cuh", r"if \(!mbar_wait_bounded\([^;]*return false;",
     r"for \(int i = consumed; i < issued; i\+\+\) \{\s*if \(!mbar_wait_bounded\(bars \+ ci \* 8, par\)\) kstat_set\(status, KSTAT_MBAR_TIMEOUT\);")], ids=["rows", "stream"])
def test_streaming_kernels_wait_for_every_copy_in_flight(name, wait, drain):
    """Behind an expired wait no block is waited for any more (one try each at most), and before the kernel ends every copy in
    flight is, also those behind one that does not come."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, "colibri_b200", "csrc", name)).read())
    assert len(re.findall(drain, text)) == 1 and len(re.findall(wait, text)) == 1
