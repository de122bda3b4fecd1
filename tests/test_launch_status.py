"""The cluster launches of the MGPCG (csrc/pfm_mgcluster.cuh) report a status that a caller cannot drop: a launch that
fails while a graph is captured would leave the graph without its node.  Compiled for the host, no GPU."""
import os
import subprocess

import pytest

from pfm import build as pfm_build

CODE = """
#include "pfm_mgcluster.cuh"
int f(pfm_handle* h, cudaStream_t s) {
  const pfm_solve_opts o{};
  %s pfm::cluster_solve_launch(h, o, s);
  %s pfm::cluster_tail_launch(h, 0, 1, nullptr, nullptr, nullptr, s);
  return a + b;
}
"""


@pytest.mark.parametrize("uses,ok", [(("int a =", "int b ="), True), (("int a = 0;", "int b ="), False),
                                     (("int a =", "int b = 0;"), False)])
def test_status_is_not_dropped(tmp_path, uses, ok):
    src = str(tmp_path / "status.cu")
    open(src, "w").write(CODE % uses)
    r = subprocess.run([pfm_build.nvcc(), "-std=c++17", "--expt-relaxed-constexpr", *pfm_build.ARCH, "-Werror",
                        "all-warnings", "-I", pfm_build.CSRC, "-I",
                        os.path.join(os.path.dirname(pfm_build.ROOT), "include"), "-c", src, "-o",
                        str(tmp_path / "status.o")], capture_output=True, text=True)
    assert (r.returncode == 0) == ok, r.stderr
    assert ok or "nodiscard" in r.stderr, r.stderr


def test_every_cluster_status_is_used():
    """Each V-cycle passes its cluster launch's status on (the compiler warns otherwise): no such warning in the
    solver's translation unit."""
    r = subprocess.run([pfm_build.nvcc(), *pfm_build.NVCC_FLAGS, "-ptx", "-O0",
                        os.path.join(pfm_build.CSRC, "pfm_mgpcg.cu"), "-o", os.devnull], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert "nodiscard" not in r.stderr, r.stderr


def test_no_constant_memory():
    """A __constant__ variable makes every launch of its file's kernels longer (0.1 us each in the solver's): small
    tables travel as kernel parameters."""
    for name in sorted(os.listdir(pfm_build.CSRC)):
        code = open(os.path.join(pfm_build.CSRC, name)).read()
        code = "\n".join(line.split("//")[0] for line in code.splitlines())
        assert "__constant__" not in code, name
