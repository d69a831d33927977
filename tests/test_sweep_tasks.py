"""The range sweep's task count over all unit and query counts (CPU only: the header's host function).

Task numbers and the ticket that deals them out have 32 bits: batches beyond kRangeTasksMax must be told
apart in 64 bits, and at every other size the blocks of queries must cover the batch.
"""
import os
import shutil
import subprocess

import pytest

from conftest import REPO

SOURCE = r"""
#include <cstdio>
#include "rangesweep.cuh"
using namespace tblaeq;
int main() {
    static_assert(kRangeTasksMax <= 0x80000000ull, "");
    const uint64_t units[] = {1, 2, 31, 1000, 12288, 3125000, 4200000, 30000000};
    const uint64_t queries[] = {1, 3, 4, 5, 31, 32, 33, 1023, 1024, 1025, 4096, 1u << 20, 1u << 21};
    bool beyond = false;
    for (uint64_t u : units)
        for (uint64_t q : queries) {
            const RangeSweepTasks t = rangeSweepTasks(u, q);
            if (t.qPer < 4 || t.qPer > kRangeTaskQueries || (t.qPer & (t.qPer - 1))) return 1;
            if (t.parts != 1 && t.parts != 2 && t.parts != 4) return 2;
            const uint64_t blocks = t.count / (u * t.parts);
            if (t.count % (u * t.parts) || blocks * t.qPer < q || (blocks - 1) * t.qPer >= q) return 3;
            beyond = beyond || t.count > 0xffffffffull;
        }
    return beyond ? 0 : 4;
}
"""


def test_tasks_cover_every_batch(tmp_path):
    cuda = next((d for d in ("/usr/local/cuda/include",) if os.path.exists(os.path.join(d, "cuda_runtime.h"))), None)
    if shutil.which("g++") is None or cuda is None:
        pytest.skip("no C++ compiler or CUDA headers")
    src, exe = tmp_path / "tasks.cpp", tmp_path / "tasks"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(REPO, "t-blaeq_b200", "csrc"), "-I", cuda, str(src), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)]).returncode == 0
