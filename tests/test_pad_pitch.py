"""The pitch of the padded velocity copies (csrc/pfm_internal.cuh, pad_pitch_of), compiled for the host: a copy holds
the field's rows and planes, takes at most four times its memory, and is indexed by 32-bit integers."""
import os
import subprocess

import pytest

from pfm import build as pfm_build

CODE = r"""
#include <cstdio>
#include <cstdlib>
#include "pfm_internal.cuh"
int main(int, char** v) {
  pfm::MacGeom g{};
  g.dim = 3;
  for (int a = 0; a < 3; ++a) g.N[a] = atoi(v[1 + a]);
  printf("%d\n", pfm::pad_pitch_of(g));
}
"""


@pytest.fixture(scope="module")
def pitch_of(tmp_path_factory):
    d = tmp_path_factory.mktemp("pitch")
    src, exe = str(d / "pitch.cu"), str(d / "pitch")
    open(src, "w").write(CODE)
    subprocess.check_call([pfm_build.nvcc(), "-std=c++17", "--expt-relaxed-constexpr", *pfm_build.ARCH, "-I",
                           pfm_build.CSRC, "-I", os.path.join(os.path.dirname(pfm_build.ROOT), "include"), src, "-o",
                           exe])
    return lambda res: int(subprocess.check_output([exe, *map(str, res)]))


# around the longest grids whose copies 32-bit integers index at each pitch, within pfm_create's limits (extents
# to 16,384, faces below 2^31)
@pytest.mark.parametrize("res,want", [((9000, 256, 256), 0), ((8191, 300, 300), 0), ((8190, 300, 300), 512),
                                      ((16383, 200, 200), 256), ((16384, 127, 100), 128), ((16384, 255, 300), 0),
                                      ((192, 192, 192), 256), ((70, 61, 75), 128), ((256, 256, 256), 0),
                                      ((100, 20, 300), 0), ((100, 600, 600), 0), ((63, 64, 64), 0)])
def test_pad_pitch(pitch_of, res, want):
    p = pitch_of(res)
    assert p == want
    if p:
        assert max(res[1:]) + 1 <= p and p * p <= 4 * (res[1] + 1) * (res[2] + 1)
        assert (res[0] + 1) * p * p < 2 ** 31
