"""CPU unit test of how a kernel's failure reaches the host (``tensorax_b200/csrc/status_report.h``): a report that lands
while the host is clearing up after an earlier one is neither lost nor left standing in the status word alone, where it
would stop every later launch without anyone being told."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r'''
#include <cstdio>
#include <functional>
#include "status_report.h"
using namespace txb;
struct Device {
    int word = 0, mirror = 0;
    bool memset_fails = false;
    std::function<void()> between = [] {};                      // what happens between the host's two steps
    void report(int code)
    {
        make_report([&](int c) { int was = word; if (was == 0) word = c; return was; }, [&](int c) { mirror = c; }, code);
    }
    int take()
    {
        return take_report([&](int v) { int was = mirror; mirror = v; return was; },
                           [&] { auto f = between; between = [] {}; f(); if (memset_fails) return false; word = 0; return true; });
    }
};
static int fails = 0;
static void expect(bool ok, const char *what) { if (!ok) { printf("failed: %s\n", what); ++fails; } }
int main()
{
    { Device d; expect(d.take() == 0 && d.word == 0, "nothing reported"); }
    { Device d; d.report(3); d.report(2);
      expect(d.take() == 3 && d.word == 0 && d.mirror == 0 && d.take() == 0, "the first code, once"); }
    { Device d; d.report(3); d.between = [&] { d.report(4); };  // another stream's kernel, before the word is cleared
      expect(d.take() == 3, "first of two"); expect(d.word == 0, "no word left behind"); expect(d.take() != 0, "the second is told too");
      expect(d.word == 0 && d.mirror == 0 && d.take() == 0, "clean afterwards"); }
    { Device d; d.report(3); expect(d.take() == 3, "taken"); d.report(4); expect(d.take() == 4 && d.word == 0, "a report after both steps"); }
    { Device d; d.report(3); d.memset_fails = true;
      expect(d.take() == 3 && d.word == 3 && d.mirror != 0, "a word that stays is still asked for");
      d.memset_fails = false; expect(d.take() == 3 && d.word == 0 && d.mirror == 0, "and cleared in the end"); }
    printf(fails ? "FAILED\n" : "all cases ok\n");
    return fails;
}
'''


def test_reports_between_the_hosts_two_steps(tmp_path):
    src, exe = tmp_path / "status_report_test.cpp", tmp_path / "status_report_test"
    src.write_text(PROGRAM)
    inc = os.path.join(ROOT, "tensorax_b200", "csrc")
    cc = subprocess.run(["g++", "-std=c++17", "-O1", "-I", inc, str(src), "-o", str(exe)], capture_output=True, text=True)
    assert cc.returncode == 0, cc.stderr[-3000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and "all cases ok" in run.stdout, run.stdout + run.stderr


def test_the_library_uses_that_rule():
    csrc = os.path.join(ROOT, "tensorax_b200", "csrc")
    assert "make_report(" in open(os.path.join(csrc, "ptx.cuh")).read()
    assert "txb::take_report(" in open(os.path.join(csrc, "sdpa_api.cu")).read()
