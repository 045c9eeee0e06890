"""The list of species that a compaction commits beside its own holds each species once (CPU: the host code is
compiled and run)."""
import os
import shutil
import subprocess

import pytest
from conftest import PKG_NAME, ROOT

SRC = r'''
#include "pic_kernels.h"
int main() {
    int counts[3][8] = {};
    pic::SpeciesDev s[3] = {};
    for (int k = 0; k < 3; k++) s[k].counts = counts[k];
    for (int a = 0; a < 3; a++)
        for (int b = 0; b < 3; b++)
            for (int c = 0; c < 3; c++) {  // any three entries beside the compaction of s[0]
                pic::CommitList l;
                l.add(s[a], s[0]);
                l.add(s[b], s[0]);
                l.add(s[c], s[0]);
                bool in[3] = {};
                for (int k = 0; k < l.n; k++)
                    for (int t = 0; t < 3; t++)
                        if (l.sp[k].counts == counts[t]) {
                            if (in[t]) return 1;  // twice
                            in[t] = true;
                        }
                for (int t = 0; t < 3; t++)
                    if (in[t] != (t != 0 && (a == t || b == t || c == t))) return 2;
            }
    return 0;
}
'''


def test_every_species_once(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "commit_list.cu", tmp_path / "commit_list"
    src.write_text(SRC)
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_103a,code=sm_103a", "-I",
                    os.path.join(ROOT, PKG_NAME, "csrc"), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
