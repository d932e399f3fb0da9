"""The pressure solve on horizontal sizes that are no powers of two (divisible
by 4, 5, 6, 8 or 10, by none of them, primes: every number of outputs per
thread; up to 1000 points: blocks of 16, 8, 4 and 2 lines, divisors whose
twiddle table would be too large) and on the short power-of-two lengths,
against the FP64 oracle: pressure 1e-11 (the plain form's tolerance) and, in
the precision form with one refinement sweep, 1e-7 (the level means it cannot
correct; beyond 150 points in proportion to the points, the bound on the
rounding of an FP32 sum)."""
import os
import subprocess
import sys

import pytest

from helpers import ROOT, gpu_dv, gpu_sim, host_case, oracle_sim, rel_l2
from test_gpu_precision import _stir

pytestmark = pytest.mark.gpu

SIZES = [(96, 90), (150, 12), (100, 21), (49, 35), (22, 26), (97, 6), (18, 54), (30, 125), (13, 81), (32, 64)]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_pressure_on_composite_lengths(nx, ny, precision):
    _solve_and_compare(nx, ny, 1e-11 if precision == "fp64" else 1e-7, precision)


def _solve_and_compare(nx, ny, tol, precision):
    nl, rs, f = host_case(case="bomex", nx=nx, ny=ny, nz=7, dx=100.0, dy=100.0, dz=40.0)
    f = _stir(f)
    o, g = oracle_sim(nl, rs, f), gpu_sim(nl, rs, f, precision=precision)
    o.update_all_bcs()
    g.PV.Update_all_bcs(g.Gr)
    o.pr_update()
    g.Pr.update(g.Gr, g.RS, g.DV, g.PV)
    assert rel_l2(gpu_dv(g)["dynamic_pressure"], o.dv["dynamic_pressure"]) < tol


LONG = [(31, 33), (7, 29), (11, 304), (389, 4), (5, 511), (720, 5), (997, 6), (6, 1000)]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,ny", LONG)
def test_pressure_on_long_and_short_lengths(nx, ny, precision):
    _solve_and_compare(nx, ny, 1e-11 if precision == "fp64" else 1e-7 * max(1.0, max(nx, ny) / 150.0), precision)


# Widths whose block of lines, twiddles and reciprocals takes just over 48 KiB
# of shared memory in FP64 (on either side: 71 and 84, 308), each the first
# solve of its process: a wider solve before it would leave the kernel's limit
# raised.
EDGE = """
import sys
sys.path.insert(0, {tests!r})
from test_gpu_fft_sizes import test_pressure_on_composite_lengths as solve
solve({nx}, 7, "fp64")
"""


@pytest.mark.parametrize("nx", [72, 83, 306])
def test_first_solve_at_the_shared_memory_limit(nx):
    code = EDGE.format(tests=os.path.join(ROOT, "tests"), nx=nx)
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("nx", [71, 76, 82, 84, 159, 161, 301, 302, 303, 307, 308])
def test_widths_around_the_shared_memory_limit(nx):
    test_pressure_on_composite_lengths(nx, 5, "fp64")
