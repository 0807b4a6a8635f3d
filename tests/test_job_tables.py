"""A clear or copy job that does not fit its table marks the table as full, and
the launch is refused (the launchers are host code: no device call is made)."""
import os
import subprocess


SOURCE = r"""
#include "sdl_kernels.h"
using namespace sdlg;
int main() {
    ClearJobs c{};
    for (int k = 0; k < kClearJobs; ++k) c.add(&c, 1);
    if (c.full || c.count != kClearJobs) return 1;
    c.add(&c, 1);
    if (!c.full || launch_clear(BatchDev{}, c, nullptr, nullptr) != cudaErrorInvalidValue) return 2;
    CopyJobs p{};
    for (int k = 0; k < kCopyJobs; ++k) p.add(&p, &p, 1);
    if (p.full || p.count != kCopyJobs) return 3;
    p.add(&p, &p, 1);
    if (!p.full || launch_copy_words(p, 1, nullptr) != cudaErrorInvalidValue) return 4;
    return 0;
}
"""


def test_full_tables_are_refused(tmp_path):
    from sdl_gb300 import build
    lib = build.build()
    src, exe = str(tmp_path / "jobs.cu"), str(tmp_path / "jobs")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I" + build.CSRC, src, lib, "-o", exe,
                    "-Xlinker", "-rpath=" + os.path.dirname(lib)], check=True)
    assert subprocess.run([exe]).returncode == 0
