"""The once-per-device preparation (csrc/epr_prepare.h) against a fake of its step: a failure is reported and tried
again by the next context, a success is not repeated, devices (also beyond 64) are prepared one by one."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "epr_prepare.h"
#include <cstdio>
#include <thread>
#include <vector>
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main()
{
    epr::PerDevice<int> d;
    int made = 0, v = -1;
    auto fails = [&](int &) { made++; return false; };
    auto works = [&](int &t) { t = 10 + made++; return true; };
    CHECK(!d.get(0, v, fails) && made == 1 && v == -1);
    CHECK(!d.get(0, v, fails) && made == 2);
    CHECK(d.get(0, v, works) && made == 3 && v == 12);
    CHECK(d.get(0, v, fails) && made == 3 && v == 12);
    CHECK(!d.get(70, v, fails) && made == 4);
    CHECK(d.get(70, v, works) && v == 14);
    CHECK(d.get(0, v, fails) && v == 12);
    int count = 0;
    std::vector<std::thread> t;
    for (int k = 0; k < 16; k++)
        t.emplace_back([&] { int w; d.get(1, w, [&](int &) { count++; return true; }); });
    for (auto &x : t) x.join();
    CHECK(count == 1);
    return 0;
}
"""


def test_prepared_once_and_after_a_failure(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if not cxx:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run([cxx, "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "exteriorpoissonrecon_gb300", "csrc"), str(tmp_path / "t.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
