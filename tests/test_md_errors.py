"""The errors of a dynamics run: those of every step's evaluation stay in the
run's error word, beside its own, until the run ends (the next evaluation
clears the result record).  Folds and messages of the library's own header,
compiled here; no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SRC = r"""
#include "mdgpu_internal.h"
#include <cstdio>
using namespace mdgpu;
int main()
{
   mdgpu_status s;
   for (int bit = 1; bit <= 16; bit *= 2)
      for (int own = 0; own <= MD_ERR_QNORM; own += MD_ERR_QNORM) {
         int w = own;
         const int steps[4] = {0, bit, 0, 0};   // one step fails, later ones do not
         for (int e : steps) w = md_err_add(w, e);
         const char *m = eval_error(w >> MD_ERR_EVAL, s);
         std::printf("%d %d %d %d %s\n", bit, (w & MD_ERR_QNORM) == own, (int)s, w == own, m ? m : "-");
      }
   const char *m = eval_error(md_err_add(md_err_add(0, 8), 16) >> MD_ERR_EVAL, s);
   std::printf("both %s\n", m);
   std::printf("none %s\n", eval_error(0, s) ? "?" : "-");
   return 0;
}
"""


def test_errors_of_every_step_are_kept(tmp_path):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no compiler or CUDA headers")
    src, exe = tmp_path / "e.cpp", str(tmp_path / "e")
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "moldy_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(CUDA, "include"), str(src), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()
    rows = [r.split(" ", 4) for r in out if r[0].isdigit()]
    assert len(rows) == 10
    want = {1: ("5", "out of range"), 4: ("2", "tile copy"), 8: ("2", "structure-factor stage"), 16: ("2", "force-pass stage")}
    for bit, own, status, lost, msg in rows:
        assert own == "1" and lost == "0"
        st, text = want.get(int(bit), ("2", "unknown"))
        assert status == st and text in msg
    assert "structure-factor stage" in out[-2] and out[-1] == "none -"
