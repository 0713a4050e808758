"""Shapes of the strided x pass (csrc/fx_shapes.h), read by a host program: the
direct form takes the TMA form's radix on every mesh and variant (so that both
round alike) and a shape that leaves its threads registers enough for two CTAs
per SM."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "cola_halo_b200", "csrc")
MESHES = (16, 32, 48, 64, 96, 128, 144, 192, 256, 384, 512, 768, 1024)

PROGRAM = r'''
#include "fx_shapes.h"
#include <cstdio>
#include <cstdlib>
int main(int, char** a) {
  for (; *++a;) {
    const int N = std::atoi(*a);
    for (int v = 0; v < (N >= cgfx::MIN_TUNED_N ? 3 : 1); v++) {
      const cgfx::FxCfg t = cgfx::fx_cfg(N, v);
      const cgfx::FxDirectCfg d = cgfx::fx_direct_cfg(N, v);
      std::printf("%d %d %d %d %d %d %d %d\n", N, v, t.tk, t.rm, d.tk, d.rm, d.thr, d.minb);
    }
  }
}
'''


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    """(mesh, variant) -> (TMA columns, radix, direct columns, radix, threads, minimum CTAs)."""
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not found")
    d = tmp_path_factory.mktemp("fx")
    (d / "fx.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-I", CSRC, str(d / "fx.cpp"), "-o", str(d / "fx")],
                   check=True)
    out = subprocess.run([str(d / "fx")] + [str(n) for n in MESHES], check=True,
                         capture_output=True, text=True).stdout
    rows = [[int(w) for w in line.split()] for line in out.splitlines()]
    return {(r[0], r[1]): tuple(r[2:]) for r in rows}


def test_direct_form_has_its_own_shape(shapes):
    """Both forms at one radix; no more than two radix-16 butterflies in a
    direct thread, three of which take over 200 registers (one CTA per SM); whole
    rows of columns."""
    for (n, v), (tk, rm, dtk, drm, thr, _) in shapes.items():
        assert drm == rm, (n, v)
        assert n % tk == 0 and n % dtk == 0 and thr % 32 == 0, (n, v)
        if rm == 16:
            assert n // 16 * dtk <= 2 * thr, (n, v)


def test_variant_numbers_keep_their_shapes(shapes):
    """Saved schedules hold variant numbers: 1 is 8 columns at radix 8 (16 from 768
    up) and 2 is 16 columns at radix 16 on every mesh that has them; the default
    is one of the shapes that were timed, and no mesh lists a shape twice but
    for the default."""
    for n in MESHES[MESHES.index(256):]:
        assert shapes[n, 1][:2] == (8, 16 if n >= 768 else 8), n
        assert shapes[n, 2][:2] == (16, 16), n
        assert shapes[n, 0][:2] in ((16, 16), (8, 16)), n
