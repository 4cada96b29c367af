"""Host-side rules of the native library that need no GPU: compiled from its headers."""
from __future__ import annotations

import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DONE = r"""
#include "mpm_done.h"
#define CHECK(x) if (!(x)) return __LINE__
int main() {
  mpm::Done d;
  CHECK(!d.holds(0) && !d.holds(7));
  d.mark(7);  // recorded in capture 7, which may never run
  CHECK(d.holds(7) && !d.holds(0) && !d.holds(8));
  d.mark(8);
  CHECK(d.holds(8) && !d.holds(7) && !d.holds(0));
  d.mark(0);  // ran: for every later call, in a capture or not
  CHECK(d.holds(0) && d.holds(8) && d.holds(9));
  d.mark(9);
  CHECK(d.holds(0) && d.holds(10));
  return 0;
}
"""


RESTORED = r"""
#include "mpm_done.h"
#define CHECK(x) if (!(x)) return __LINE__
int main() {
  mpm::Restored z;
  z.now.mark(0);  // as a handle is created
  CHECK(z.begin(0));
  z.end(0);
  CHECK(z.begin(5));  // a capture of a state that holds restores nothing
  z.end(5);
  CHECK(z.begin(0));  // and this call fails: no end()
  CHECK(!z.begin(6));  // restored in capture 6
  z.end(6);
  CHECK(z.begin(6));  // once per capture
  z.end(6);
  CHECK(!z.begin(7));  // not in another
  z.end(7);
  CHECK(!z.begin(0));  // and not outside
  z.end(0);
  CHECK(z.begin(0));
  z.end(0);
  CHECK(z.begin(8));
  z.end(8);
  CHECK(z.begin(0));
  return 0;
}
"""


def _run(tmp_path, source):
    """0, or the line of the first check that fails."""
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "diffskill_gb300", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    return subprocess.run([str(exe)]).returncode


def test_recorded_work_is_done_for_its_own_capture_only(tmp_path):
    """What a capture only recorded must not count as done for a call outside it."""
    assert _run(tmp_path, DONE) == 0


def test_a_failed_call_is_followed_by_a_clearing_one_in_each_capture_and_outside(tmp_path):
    assert _run(tmp_path, RESTORED) == 0


def test_aligned_cluster_barriers_follow_a_warp_barrier():
    """barrier.cluster.*.aligned is undefined unless all threads of the warp execute it
    together, and nothing but a warp barrier brings them together after a branch: each
    arrive has one directly before it (the wait follows the arrive)."""
    arrives = 0
    for path in glob.glob(os.path.join(ROOT, "diffskill_gb300", "csrc", "*.cu*")):
        code = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"barrier\.cluster\.arrive[.a-z]*\.aligned", code):
            arrives += 1
            before = code[:code.rfind("asm", 0, m.start())].rstrip()
            assert before.endswith("__syncwarp();"), path
    assert arrives
