"""Launch shapes that size device buffers (mdff_b200/csrc/shapes.h, plain host
arithmetic), over whole ranges of ion counts and meshes: what a launch uses never
exceeds what its buffer holds.  No GPU."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include "shapes.h"
using namespace mdff;
static int mesh_rows(int kx, int ky) { return ky + 1 + kx * (2 * ky + 1); }  // (nx, ny) of the half space
static int want_of(int nsm, int kx, int ky, int kz, int hm) {
  return rho_dm_want(nsm, mesh_rows(kx, ky), ceil_div(kz / 4 + 1, rho_dm_nt(kz, hm)));
}
extern "C" {
int dm_chunks(int nsm, int kx, int ky, int kz, int hm, int nion, int* chunk) {
  int n;
  rho_dm_split(nion, want_of(nsm, kx, ky, kz, hm), chunk, &n);
  return n;
}
int dm_most(int nsm, int kx, int ky, int kz, int hm, int natm) { return rho_dm_most(natm, want_of(nsm, kx, ky, kz, hm)); }
// launches over nion of natm ions (any nion <= natm, both kinds) that need more
// chunks than are allocated for natm, or whose chunks do not cover the ions
int dm_overruns(int nsm, int kmax, int natm_lo, int natm_hi) {
  int bad = 0;
  for (int natm = natm_lo; natm <= natm_hi; ++natm) {
    const int a = dm_most(nsm, kmax, kmax, kmax, 0, natm), b = dm_most(nsm, kmax, kmax, kmax, 1, natm);
    const int room = a > b ? a : b;
    for (int f = 1; f <= 24; ++f)
      for (int hm = 0; hm < 2; ++hm) {
        const int nion = (int)((long)natm * f / 24);
        if (nion < 1) continue;
        int chunk;
        const int n = dm_chunks(nsm, kmax, kmax, kmax, hm, nion, &chunk);
        bad += n > room || (long)n * chunk < nion || (long)(n - 1) * chunk >= nion || chunk % 8 != 0;
      }
  }
  return bad;
}
int cache_fits(double gb, double free_gb, double total_gb) {
  return pair_cache_fits((size_t)(gb * 1e9), (size_t)(free_gb * 1e9), (size_t)(total_gb * 1e9));
}
// stagings of the batched engine's structure factor over the meshes that a batch
// takes (kx, ky <= 64, kz <= 12), 0-2048 ions, one or two weights an ion, for one
// buffer size: records that do not fit, none at all, or fewer than four although eight fit
int batch_staging_faults(int stage, int* least) {
  int bad = 0;
  *least = 1 << 30;
  for (int kxy = 0; kxy <= 128; ++kxy)
    for (int kz = 0; kz <= 12; ++kz) {
      const int rs = brec_bytes(kxy / 2, kxy - kxy / 2, kz);
      for (int cnt = 0; cnt <= 2048; cnt += cnt < 64 ? 1 : 13)
        for (int nw = 1; nw <= 2; ++nw) {
          const BStaging s = brec_staging(stage, cnt, nw, rs);
          bad += s.ch < 1 || s.ch > 32 || s.weights + 2 * s.ch * rs > stage || s.weights % 128 != 0;
          bad += s.weights && s.weights < cnt * 32 * nw;
          bad += s.ch >= 4 ? s.ch % 4 != 0 : stage >= 8 * rs;
          if (s.ch < *least) *least = s.ch;
        }
    }
  return bad;
}
}
"""


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("shapes")
    src, lib = d / "probe.cpp", d / "libprobe.so"
    src.write_text(PROBE)
    subprocess.run([gxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-Wno-unused-function", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "mdff_b200", "csrc"), str(src), "-o", str(lib)], check=True)
    return ctypes.CDLL(str(lib))


@pytest.mark.parametrize("natm,nion,kmax,chunks", [(5103, 3402, 9, 48), (1188, 792, 10, 33)])
def test_subset_of_the_ions_can_need_more_chunks(shapes, natm, nion, kmax, chunks):
    c = ctypes.c_int()
    assert shapes.dm_chunks(148, kmax, kmax, kmax, 1, nion, ctypes.byref(c)) == chunks
    assert shapes.dm_chunks(148, kmax, kmax, kmax, 1, natm, ctypes.byref(c)) < chunks
    assert shapes.dm_most(148, kmax, kmax, kmax, 1, natm) >= chunks


@pytest.mark.parametrize("nsm", [148, 132])
@pytest.mark.parametrize("kmax", [1, 3, 4, 6, 8, 9, 10, 12, 16, 19, 20, 24, 31])
def test_structure_factor_chunks_fit_their_buffer(shapes, kmax, nsm):
    assert shapes.dm_overruns(nsm, kmax, 1, 6000) == 0
    assert shapes.dm_overruns(nsm, kmax, 13600, 13800) == 0
    assert shapes.dm_overruns(nsm, kmax, 100000, 100050) == 0


@pytest.mark.parametrize("stage", [16384] + list(range(20480, 40960 + 1, 1280)))
def test_batch_staging_holds_records(shapes, stage):
    least = ctypes.c_int()
    assert shapes.batch_staging_faults(stage, ctypes.byref(least)) == 0
    assert least.value >= 3


@pytest.mark.parametrize("gb,free,total,fits", [(0.09, 180, 190, 1), (20, 180, 190, 1), (47, 180, 190, 0),
                                                (20, 30, 190, 0), (0.09, 0.15, 190, 0), (0.0, 0.0, 190, 1)])
def test_pair_cache_leaves_room(shapes, gb, free, total, fits):
    d = ctypes.c_double
    assert shapes.cache_fits(d(gb), d(free), d(total)) == fits
