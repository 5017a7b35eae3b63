"""Host work shared out to threads (gd_workers.h), compiled for the host: an
exception in a share is reported to the caller instead of ending the process, and
where no thread can be started the caller does the work itself."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu_determ_gb300", "csrc")

PROGRAM = r"""
#include "gd_workers.h"
#include <atomic>
#include <cstdio>
#include <new>
#include <system_error>

int started = 0, allowed = 0;
struct FewThreads {   // a std::thread of which only some can be started
    std::thread t;
    template <typename F>
    FewThreads(F f, int k)
    {
        if (started++ >= allowed) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
        t = std::thread(f, k);
    }
    FewThreads(FewThreads &&) = default;
    void join() { t.join(); }
};

template <typename T>
bool run(int n, int bad, std::atomic<int> *done)
{
    return gd::run_workers<T>(n, [&](int k) {
        if (k == bad) throw std::bad_alloc();
        done[k]++;
    });
}

int main()
{
    for (int n = 1; n <= 8; n++)
        for (int bad = -1; bad < n; bad++)
            for (allowed = 0; allowed <= n; allowed++) {
                std::atomic<int> a[8] = {}, b[8] = {};
                started = 0;
                if (run<FewThreads>(n, bad, a) != (bad < 0) || run<std::thread>(n, bad, b) != (bad < 0)) return 1;
                for (int k = 0; k < n; k++)
                    if (a[k] != (k != bad) || b[k] != (k != bad)) return 2;
            }
    std::puts("ok");
}
"""


def test_run_workers_reports_and_completes(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    src = tmp_path / "w.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "w"
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok"
