"""The host thread pool that stages pm_run's pageable operands, stressed on the CPU (no GPU).

A task set handed to the pool must run every task exactly once and have none still running
when the call returns: the tasks capture the caller's stack.  The pool hands out tasks as
tickets of one packed word (job, count, next ticket) with fetch_add, and replaces the job's
function only after every task of the job has finished.  Four shapes are exercised: many fresh
pools (a first call each), long runs of task sets of varying size, task sets that find the
workers parked on their futex and must wake them, and task sets opened on the workers alone
(start) and joined by the caller after its own work (wait), as the staging pipeline does."""
import os
import subprocess

import pytest

from conftest import PKG, ensure_library


def test_first_calls_of_fresh_pools():
    import polymult
    ensure_library()
    assert polymult.host_pool_selftest(pools=3000, runs=2) == 0


def test_varying_task_counts():
    import polymult
    ensure_library()
    assert polymult.host_pool_selftest(pools=40, runs=1000, vary=True) == 0


def test_parked_workers_are_woken():
    import polymult
    ensure_library()
    assert polymult.host_pool_selftest(pools=4, runs=300, vary=True, park=True) == 0


def test_started_sets_joined_later():
    import polymult
    ensure_library()
    assert polymult.host_pool_selftest(pools=40, runs=1000, vary=True, split=True) == 0
    assert polymult.host_pool_selftest(pools=4, runs=300, vary=True, park=True, split=True) == 0
    # no workers: wait() runs every task on the caller
    assert polymult.host_pool_selftest(pools=20, runs=100, workers=0, vary=True, split=True) == 0


def test_argument_check():
    import polymult
    ensure_library()
    with pytest.raises(polymult.PolymultError):
        polymult.host_pool_selftest(pools=1, runs=1, workers=100)


def test_copy_tasks_cover_a_chunk_in_small_pieces(tmp_path):
    """The tasks of a chunk's copy, whatever its rows: every word once, at least 32 KB each and at most
    128 KB or a 32nd of the chunk (a row more where a task has several), parts of a row on 32-byte
    boundaries."""
    src = tmp_path / "tasks.cpp"
    src.write_text(r"""
#include "pm_hostpool.h"
#include <cstdio>
#include <cstdlib>
int main() {
    const uint32_t rows[] = {1, 2, 4, 16, 32, 64, 128, 256, 1024};
    const size_t words[] = {1, 7, 8, 63, 1760, 2001, 7040, 28160, 56320, 65001, 225280};
    for (uint32_t r : rows)
        for (size_t w : words) {
            const pm::CopyTasks T(r, w);
            const size_t total = r * w;
            std::vector<unsigned char> seen(total, 0);
            bool ok = T.count() >= 1 && T.count() <= 128;
            for (uint32_t t = 0; t < T.count(); ++t) {
                size_t got = 0;
                T.each(t, [&](uint32_t row, size_t first, size_t n) {
                    ok = ok && row < r && first % 8 == 0 && first + n <= w;
                    for (size_t k = 0; ok && k < n; ++k) ++seen[row * w + first + k];
                    got += n;
                });
                ok = ok && (got * 4 + 32 >= 32768 || T.count() == 1 || t + 1 == T.count());
                const size_t share = std::max<size_t>(total / 64, 16384);
                ok = ok && got <= 2 * share + (T.rows_per > 1 ? w : 8);
            }
            for (unsigned char x : seen) ok = ok && x == 1;
            if (!ok) return std::printf("rows %u words %zu: %u tasks\n", r, w, T.count()), 1;
        }
    // quarters of 65536 coefficients of 55 words, of 32768 of 38 and of 28
    return pm::CopyTasks(16, 56320).count() == 64 && pm::CopyTasks(16, 19456).count() == 32 &&
                   pm::CopyTasks(16, 14336).count() == 16 ? 0 : 2;
}
""")
    exe = str(tmp_path / "tasks")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(PKG, "csrc"), str(src), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
