"""CPU check of the order in which a GEMM tile fetches, multiplies and waits
for its K chunks (csrc/mma_steps.h), run against a model of the tensor cores: a
stage is never refilled under products that still read it, and on return no
products are in flight that the last wait, successful or not, did not cover,
also when any one of the waits runs out."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MODEL = r"""
#include <cstdio>
#include <cstdlib>
#include "mma_steps.h"
constexpr int kStages = %d;
static void check(bool x, const char *what, int nc, int bad) {
    if (x) return;
    std::printf("%%s (chunks %%d, failed wait %%d)\n", what, nc, bad);
    std::exit(1);
}
int main() {
    for (int nc = 0; nc <= 9; ++nc)
        for (int bad = -1; bad <= nc; ++bad) {  // the bad-th wait runs out (-1: none)
            int fetched = -1, issued = -1, covered = -1, complete = -1, waits = 0;
            auto fetch = [&](int i) {
                check(i == fetched + 1, "fetches in order", nc, bad);
                fetched = i;
                // the stage's last reader was chunk i - kStages
                if (i < nc) check(i - kStages <= complete, "stage refilled under its products", nc, bad);
            };
            auto issue = [&](int i) {
                check(i == issued + 1 && i <= fetched, "products before their copy", nc, bad);
                issued = i;
            };
            auto wait = [&](int i) {
                check(i <= issued, "wait for nothing", nc, bad);
                if (i > covered) covered = i;
                if (waits++ == bad) return false;
                if (i > complete) complete = i;
                return true;
            };
            const bool ok = asdm::tc::run_chunks<kStages>(nc, fetch, issue, wait, [](bool x) { return x; });
            check(covered == issued, "products in flight at the release", nc, bad);
            check(ok == (bad < 0 || bad >= waits), "result", nc, bad);
            if (ok) check(issued == nc - 1 && complete == nc - 1, "every chunk", nc, bad);
        }
    return 0;
}
"""


@pytest.mark.parametrize("stages", [2, 3, 4])
def test_steps(tmp_path, stages):
    src, exe = str(tmp_path / "model.cpp"), str(tmp_path / "model")
    with open(src, "w") as fh:
        fh.write(MODEL % stages)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "asdmatch_b200", "csrc"), src, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
