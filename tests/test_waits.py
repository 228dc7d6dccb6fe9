"""The bounded waits of the kernels, run on the host: the functions' own source with stand-ins for the instructions they use."""
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aegist-optimized-ai-library-_b200", "csrc")


def function(name, file="kernels.cuh"):
    """The text of one function of a source file, its template line included."""
    text = open(os.path.join(CSRC, file)).read()
    m = re.search(r"(?:^template <[^\n]*>\n)?^[^\n/]*\b" + name + r"\(.*?^}\n", text, re.M | re.S)
    assert m, name
    return m.group(0)


def run(tmp_path, source):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text("#include <cstdint>\n#include <cstdio>\n#define __device__\n#define __host__\n#define __forceinline__ inline\n" + source)
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", "-o", str(exe), str(src)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.split()


@pytest.mark.parametrize("away_after", [1, 2, 3, 10])
@pytest.mark.parametrize("away", [0, 1 << 31])
def test_a_wait_outlasts_a_warp_that_was_switched_out(tmp_path, away_after, away):
    """The warp is off the SM for `away` clocks behind a failed try, and its copy lands a few tries after it is back (it was switched out
    with it). Only tries that were made count, so the wait succeeds and leaves no error."""
    assert run(tmp_path, """
static long long now = 0; static int tries = 0;
static long long clock64() { return now; }
static int atomicExch(int* p, int v) { int o = *p; *p = v; return o; }
template <typename B> static bool mbar_try(B, uint32_t) {
    ++tries; now += 170;
    if (tries == %d) now += %dll;
    return tries == %d + 5;
}
""" % (away_after, away, away_after) + function("mbar_wait") + """
int main() { int err = 0; const bool ok = mbar_wait(0u, 0u, &err); std::printf("%d %d", (int)ok, err); }
""") == ["1", "0"]


@pytest.mark.parametrize("limit", [1, 2, 3, 1000, 1 << 16])
def test_a_wait_gives_up_after_its_tries(tmp_path, limit):
    """A phase that never ends: a bounded number of tries (two stand before the loop), then the error word."""
    ok, err, tries = map(int, run(tmp_path, """
static long long now = 0; static int tries = 0;
static long long clock64() { return now; }
static int atomicExch(int* p, int v) { int o = *p; *p = v; return o; }
template <typename B> static bool mbar_try(B, uint32_t) { ++tries; now += 170; return false; }
""" + function("mbar_wait") + """
int main() { int err = 0; const bool ok = mbar_wait(0u, 0u, &err, %d); std::printf("%%d %%d %%d", (int)ok, err, tries); }
""" % limit))
    assert (ok, err) == (0, 3) and tries == max(2, limit)


@pytest.mark.parametrize("never", [0, 1, 1 << 7, 1 << 31, 0x0000FFFF, 0xFFFFFFFE, 0xFFFFFFFF])
def test_a_warp_that_waits_has_one_verdict(tmp_path, never):
    """32 threads as a warp: the lanes in `never` never see the phase end, the others at once or, in a second wait, lane i at its i-th try.
    All lanes must go the same way, or some would meet the others at another barrier or in an instruction of the whole warp; behind a
    wait that gave up all of them skip the next one."""
    got = run(tmp_path, """
#include <atomic>
#include <barrier>
#include <thread>
#include <vector>
static std::barrier<> meet(32);
static std::atomic<unsigned> votes, tried;
static thread_local int lane, tries;
static int atomicExch(int* p, int v) { return __atomic_exchange_n(p, v, __ATOMIC_SEQ_CST); }
static void __syncwarp() { meet.arrive_and_wait(); }
static bool __any_sync(unsigned, bool p) {
    if (p) votes |= 1u << lane;
    meet.arrive_and_wait();
    const bool any = votes != 0;
    meet.arrive_and_wait();
    votes = 0;
    meet.arrive_and_wait();
    return any;
}
static bool __all_sync(unsigned m, bool p) { return !__any_sync(m, !p); }
template <typename B> static bool mbar_try(B late, uint32_t) {
    tried++;
    return late ? ++tries >= lane : !(%uu >> lane & 1);
}
""" % never + function("mbar_wait") + function("warp_wait") + """
int main() {
    int err = 0;
    std::atomic<unsigned> gone{0};
    auto warp = [&](unsigned late) {
        std::vector<std::thread> t;
        for (int i = 0; i < 32; i++)
            t.emplace_back([&, i] { lane = i; bool dead = gone >> i & 1; warp_wait(late, 0u, &err, dead, 64); if (dead) gone |= 1u << i; });
        for (auto& x : t) x.join();
    };
    warp(0);
    std::printf("%u %d ", gone.load(), err);
    if (gone != 0 && gone != 0xFFFFFFFFu) return 0;
    tried = 0;
    warp(1);
    std::printf("%u %d", gone.load(), tried > 0);
}
""")
    assert got == (["4294967295", "3", "4294967295", "0"] if never else ["0", "0", "0", "1"])


def test_registers_that_k_umma_q4_hands_over(tmp_path):
    """setmaxnreg.inc waits without a bound until the block's own pool holds what it asks for. Whatever the compiler made of the kernel, the
    launch rule says yes only where the epilogue's warpgroups get their registers once the others have given theirs back, and is asked
    before every launch."""
    text = open(os.path.join(CSRC, "ummaq4.cuh")).read()
    lines = [m.group(0) for m in re.finditer(r"^constexpr int UQ_(EPI|THREADS|REGS_LOW)\b.*$", text, re.M)]
    got = run(tmp_path, "\n".join(lines) + "\n" + function("uq_regs_suffice", "ummaq4.cuh") + """
int main() {
    for (int regs = 24; regs * UQ_THREADS <= 65536; regs += 8) {
        long pool = 0, low = UQ_THREADS / 128 - UQ_EPI / 4;       // warpgroups of 128 threads
        bool good = regs >= UQ_REGS_LOW && regs <= UQ_REGS_EPI;
        pool += low * 128 * (regs - UQ_REGS_LOW);
        for (int g = 0; g < UQ_EPI / 4; g++) { pool -= 128 * (UQ_REGS_EPI - regs); good = good && pool >= 0; }
        std::printf("%d %d %d ", regs, (int)good, (int)uq_regs_suffice(regs));
    }
}
""")
    rows = [got[i:i + 3] for i in range(0, len(got), 3)]
    assert all(good == says for _, good, says in rows)
    assert {regs: says for regs, _, says in rows}["88"] == "0" and {regs: says for regs, _, says in rows}["96"] == "1"
    asks = function("umma_q4_maps", "engine.cu")
    assert "cudaFuncGetAttributes(&built, k_umma_q4)" in asks and "if (!uq_regs_suffice(built.numRegs)) return false;" in asks


@pytest.mark.parametrize("file,kernel", [("ummagemm.cuh", "k_umma"), ("ummaq4.cuh", "k_umma_q4")])
def test_no_product_is_under_way_when_tensor_memory_goes_back(file, kernel):
    """Products that run on behind a block that has given back its tensor memory, and left, fault. The epilogue has waited for all of them
    unless one of its waits gave up, so the issuer itself ends with a commit behind its last product and a wait for it."""
    text = open(os.path.join(CSRC, file)).read()
    body = text[text.index(" " + kernel + "(const __grid_constant__"):]
    issuer = re.search(r"// ---- MMA issuer.*?\n    \} else if", body, re.S).group(0)
    drained, = re.findall(r"umma_commit\(([^;]*drained[^;]*)\);", issuer, re.I)
    last = max(issuer.rindex("um" + ("_issue<" if kernel == "k_umma" else "ma_commit(bar(P_EMPTY")), issuer.index("umma_commit(" + drained))
    wait = issuer.index("mbar_wait(" + drained + ", 0, a.err")
    assert issuer.index("umma_commit(" + drained) == last < wait and "if (dead)" not in issuer[last:wait]
    assert body.index("mbar_wait(" + drained) < body.index("tmem_dealloc(")
