"""A tuning report set on another context makes it run the kernels that the
report's times are of, the horizontal WAF tiles by the members' sizes included:
the report carries that choice, and setting it returns a context to it."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from regcm_gb300 import abi, build
from regcm_gb300 import case as cs
from regcm_gb300 import moloch as ml


class FakeLib:
    """mlc_autotune fills a report; mlc_set_launch_shapes keeps what it gets."""

    def __init__(self, **fields):
        self.fields, self.got = fields, None

    def mlc_autotune(self, ctx, steps, rep):
        for n, v in self.fields.items():
            setattr(rep._obj, n, v)
        return abi.MLC_OK

    def mlc_set_launch_shapes(self, ctx, rep):
        self.got = {n: v for n, v in rep._obj.as_dict().items() if not n.startswith("ms_")}
        return abi.MLC_OK


@pytest.mark.parametrize("by_size", [0, 1])
def test_report_dict_round_trip(by_size):
    shapes = dict(col_x=64, col_y=2, solve_x=32, solve_y=1, vert_x=32, vert_y=8, htile=1, by_size=by_size)
    lib = FakeLib(ms_fixed=2.0, ms_tuned=1.0, **shapes)
    rep = ml._autotune(lib, None, 1)
    ml._set_launch_shapes(lib, None, rep)
    assert lib.got == shapes


def test_reports_of_earlier_builds():
    """The choice lies in what was padding (the structure keeps its size and its
    times their place), and a dict without it names explicit tiles."""
    assert C.sizeof(abi.mlc_tune_report) == 48 and abi.mlc_tune_report.ms_fixed.offset == 32
    lib = FakeLib()
    ml._set_launch_shapes(lib, None, dict(col_x=32, col_y=4, htile=2))
    assert lib.got["by_size"] == 0 and lib.got["htile"] == 2


# the library's own rule, on a context without members whose sizes call for
# 128-column tiles (4) and, in the increment form, 64-column ones (1)
SOURCE = """
#include "mlc_context.cu"
int main() {
  mlc_ctx x;
  x.mixed = true;
  LaunchGeom &L = x.key.L;
  L.htile = -1;
  L.size_tile = 4;
  L.size_tile_inc = 1;
  int htile, by_size;
  while (std::scanf("%d %d", &htile, &by_size) == 2) {
    mlc_tune_report r{};
    r.col_x = 32; r.col_y = 4; r.solve_x = 32; r.solve_y = 2; r.vert_x = 32; r.vert_y = 4;
    r.htile = htile;
    r.by_size = by_size;
    const int st = mlc_set_launch_shapes(&x, &r);
    std::printf("%d %d %d\\n", st, waf_tile(L), waf_tile_inc(L));
  }
}
"""


def test_by_size_is_set_and_left(tmp_path):
    (tmp_path / "set.cu").write_text(SOURCE)
    objs = [str(build.OUT / f"mlc_{n}.o") for n in ("sound", "advect", "end", "noalloc", "setup", "restart")]
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", str(build.CSRC), "-o",
                    str(tmp_path / "set"), str(tmp_path / "set.cu"), *objs, "-lcudart"], check=True, capture_output=True)
    # explicit, back to by size, refused (nothing changes), explicit
    queries = [(3, 0), (1, 1), (4, 1), (-1, 0), (2, 0), (0, 1)]
    out = subprocess.run([str(tmp_path / "set")], input="".join("%d %d\n" % q for q in queries), check=True,
                         capture_output=True, text=True).stdout
    got = [tuple(map(int, line.split())) for line in out.splitlines()]
    bad = abi.MLC_ERR_INVALID
    assert got == [(0, 3, 3), (0, 4, 1), (bad, 4, 1), (bad, 4, 1), (0, 2, 2), (0, 4, 1)]


@pytest.mark.gpu
def test_an_autotuned_report_can_be_set():
    members = [cs.config2_member(m, 120, 64, 12, precision=abi.MLC_PREC_MIXED) for m in range(2)]
    a, b = ml.MolochBatch(members), ml.MolochBatch(members)
    rep = a.autotune(1)
    assert rep["by_size"] in (0, 1) and rep["htile"] in (0, 1, 2, 3)
    b.set_launch_shapes(dict(ml.DEFAULT_SHAPES, htile=3))
    b.set_launch_shapes(rep)
    a.step(2)
    b.step(2)
    got = [members[1].empty_state() for _ in range(2)]
    for dom, g in zip((a, b), got):
        dom.download(1, members[1].state_ptrs_of(g))
        dom.close()
    for n in got[0]:
        assert np.array_equal(got[0][n], got[1][n]), n
