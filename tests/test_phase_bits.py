"""The barrier phases a kernel waits for (phase_bits.h), compiled for the host: after a
bounded wait has run out, the wait that guards the way out of the kernel is for the phase
that is still incomplete."""
import subprocess
from pathlib import Path

SRC = Path(__file__).resolve().parent.parent / "compchan3dmpi_b200" / "csrc"

# An mbarrier in the phase `done`: a wait for a parity succeeds unless that is the parity of
# the phase in progress (the one before it has the other parity and is complete).
MODEL = r"""
#include "phase_bits.h"
#include <cstdio>
struct Barrier {
    unsigned done = 0;   // phases completed
    bool test(unsigned parity) const { return (done & 1u) != parity; }
};
#define CHECK(x) do { if (!(x)) { std::printf("line %d, phase %u: %s\n", __LINE__, n, #x); return 1; } } while (0)
"""

WAITS = r"""
int main()
{
    for (unsigned n = 0; n < 9; n++)
        for (int s = 0; s < 4; s++) {
            Barrier b[4];
            PhaseBits ph;
            auto wait = [&](int q) {
                const bool ok = b[q].test(ph.next(q));
                ph.waited(q);
                return ok;
            };
            for (unsigned k = 0; k < n; k++) {   // n phases complete and are waited for
                b[s].done++;
                CHECK(wait(s));
            }
            // the next one is in flight.  Not waited for yet: the wait before leaving is not
            // satisfied until it completes
            CHECK(!b[s].test(ph.open(s, false)));
            CHECK(!wait(s));                     // its wait runs out: the same
            CHECK(!b[s].test(ph.open(s, true)));
            b[s].done++;
            CHECK(b[s].test(ph.open(s, true)));
            for (int q = 0; q < 4; q++)
                if (q != s) { CHECK(!wait(q)); }
        }
    return 0;
}
"""

COMMITS = r"""
int main()
{
    for (unsigned n = 1; n < 9; n++)
        for (int s = 0; s < 2; s++) {
            Barrier b[2];
            CommitBits log{};
            CHECK(!log.some(0) && !log.some(1));
            for (unsigned k = 0; k < n; k++) log.committed(s);
            CHECK(log.some(s) && !log.some(1 - s));
            b[s].done = n - 1;                   // all but the last are complete
            CHECK(!b[s].test(log.last(s)));
            b[s].done = n;
            CHECK(b[s].test(log.last(s)));
        }
    return 0;
}
"""


def run(tmp_path, program):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(MODEL + program)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", f"-I{SRC}", "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_wait_that_ran_out_keeps_its_phase(tmp_path):
    run(tmp_path, WAITS)


def test_wait_for_the_last_commit(tmp_path):
    run(tmp_path, COMMITS)
