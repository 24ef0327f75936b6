"""What is done once per device (csrc/per_device.h), on the host: every device
gets its own, a failure is tried again, and threads that come together all
find it done. The tensor-core launchers set their kernels' shared memory so."""
import subprocess

from pca_gb300.build import CSRC

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"

int main()
{
    pcagb::OncePerDevice once;
    int calls[80] = {};
    for (int round = 0; round < 3; round++)
        for (int d : {0, 1, 7, 63})
            if (!once.run(d, [&] { calls[d]++; return true; })) return 1;
    for (int d : {0, 1, 7, 63})
        if (calls[d] != 1) return 2;
    /* a failure is not kept */
    if (once.run(2, [] { return false; })) return 3;
    if (!once.run(2, [&] { calls[2]++; return true; }) || calls[2] != 1) return 4;
    /* past the flags: each time */
    for (int i = 0; i < 2; i++)
        if (!once.run(64, [&] { calls[64]++; return true; })) return 5;
    if (calls[64] != 2) return 6;
    for (int round = 0; round < 200; round++) {
        pcagb::OncePerDevice shared;
        int set[4] = {};   /* as a device's attribute: setting it again changes nothing */
        std::vector<std::thread> ts;
        std::atomic<int> bad{0};
        for (int t = 0; t < 8; t++)
            ts.emplace_back([&, t] {
                auto *s = reinterpret_cast<std::atomic<int> *>(&set[t % 4]);
                if (!shared.run(t % 4, [&] { s->store(1); return true; }) || !s->load()) bad++;
            });
        for (auto &t : ts) t.join();
        if (bad) return 7;
    }
    puts("ok");
    return 0;
}
"""


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.returncode
