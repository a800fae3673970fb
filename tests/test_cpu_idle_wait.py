"""CPU check of an idle warp's wait for work (csrc/idle_wait.h) against models
of the other side: it ends soon after a stop flag, never between a donor's claim
and its record, and also where a claimed warp's record never comes."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MODEL = r"""
#include <cstdio>
#include <cstdlib>
#include "idle_wait.h"
using namespace asdm;
constexpr uint64_t kPoll = 500, kNever = ~0ull, kHour = 3600ull * 1000000000ull;
struct Io {  // times at which things happen; a poll takes kPoll
    uint64_t record, done, stop, claim;
    uint64_t t = 0;
    bool idle = true, marked = false, over = false;
    bool ended() const { return over; }
    uint32_t mail() const { return t >= record ? kMailRecord : t >= done ? kMailDone : kMailEmpty; }
    bool stopped() const { return marked || t >= stop; }
    uint64_t now() const { return t; }
    bool take_back() {
        if (t >= claim) return false;
        idle = false;
        return true;
    }
    void lost() { marked = true; }
    void nap() {
        t += kPoll;
        if (t > 2 * kHour) { std::printf("still waiting\n"); std::exit(1); }
    }
};
static int bad = 0;
static void expect(const char *what, Io io, uint64_t until, bool got, bool marked, uint64_t least, uint64_t most) {
    const bool r = idle_wait(io, until);
    if (r == got && io.marked == marked && io.t >= least && io.t <= most) return;
    std::printf("%s: got %d, marked %d, after %llu ns\n", what, r, io.marked, (unsigned long long)io.t);
    bad = 1;
}
int main() {
    const uint64_t look = 256 * kPoll, T = 50'000'000;
    expect("record", {T, kNever, kNever, T}, kHour, true, false, T, T + kPoll);
    expect("end", {kNever, T, kNever, kNever}, kHour, false, false, T, T + kPoll);
    expect("deadline", {kNever, kNever, kNever, kNever}, T, false, false, T, T + 2 * look);
    expect("stop", {kNever, kNever, T, kNever}, kHour, false, false, T, T + look);
    expect("stop between claim and record", {T + 900'000'000, kNever, T, T - 1}, kHour, true, false, T, T + 901'000'000);
    expect("deadline between claim and record", {T + 900'000'000, kNever, kNever, T - 1}, T, true, false, T, T + 901'000'000);
    expect("record lost", {kNever, kNever, kNever, T - 1}, T, false, true, T + kHandoffNs, T + kHandoffNs + 3 * look);
    expect("record lost after a stop", {kNever, kNever, T, T - 1}, kHour, false, true, T + kHandoffNs,
           T + kHandoffNs + 3 * look);
    Io io{kNever, kNever, kNever, kNever};
    io.over = true;
    expect("over", io, kHour, false, false, 0, 0);
    return bad;
}
"""


def test_idle_wait(tmp_path):
    src, exe = str(tmp_path / "model.cpp"), str(tmp_path / "model")
    with open(src, "w") as fh:
        fh.write(MODEL)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "asdmatch_b200", "csrc"), src, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
