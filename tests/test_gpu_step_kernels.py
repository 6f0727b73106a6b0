"""The step's kernels that sum or group what separate launches did: the
direction-independent terms of the DPLUR sweeps, faces that share a launch and
the 2-D plane copy with the properties, against the CPU oracle."""
import numpy as np
import pytest

import openstc_b200 as ostc
from openstc_b200 import cases
from oracle_bridge import OracleSolver, interior

pytestmark = pytest.mark.gpu


def check(case, steps, fields, tol, precision="fp64"):
    gpu = ostc.Driver(case, precision=precision)
    gpu.initialize()
    orc = OracleSolver(ostc.Driver(case), threads=4)
    orc.initialize()
    for s in range(steps):
        gpu.step(1)
        orc.step(s + 1)
    for b in range(gpu.info().n_block):
        for f in fields:
            g, _ = gpu.layout(f)
            a = gpu.get(b, f)
            o = interior(orc.get(b, f, a.shape), g)
            a = interior(a, g)
            for l in range(a.shape[0]):
                scale = max(np.max(np.abs(o[1:4])) if f == "bv" and 1 <= l <= 3 else np.max(np.abs(o[l])), 1e-6)
                assert np.max(np.abs(a[l] - o[l])) <= tol * scale, (b, f, l)
    return gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-4)])
@pytest.mark.parametrize("dplur,chem", [(0, 1), (1, 1), (2, 2), (3, 0)])
def test_sweeps_with_stored_terms(tmp_path, precision, tol, dplur, chem):
    """No sweep, one (terms of dq0 only), two and three (the ping-pong of the
    stored terms), every chemistry treatment, on a grid with remainders.  FP64:
    libm differs by ulps (the bound of the phase tests over two steps);
    FP32-bulk: single-precision fluxes over two steps."""
    case = cases.mixing_layer_case(tmp_path / "c", mx=33, my=10, mz=5, total_step=2, output_screen=1, dplur=dplur,
                                   chem=chem)
    check(case, 2, ("bv", "sv"), tol, precision)


@pytest.mark.parametrize("mxs", [[9, 7], [6, 8, 7, 9]])
def test_faces_that_share_a_launch_keep_their_order(tmp_path, mxs):
    """Boundary and inner faces of several blocks: those that touch a common
    point (edges of the boundaries, both sides of an inner face, short blocks whose
    two inner faces reach the same layers) run in the reference's order."""
    case = cases.multiblock_case(tmp_path / "c", mxs, my=8, mz=5, total_step=3, output_screen=1)
    check(case, 3, ("bv", "sv"), 1e-9)  # the shared planes' Newton starts differ by the averages' order


@pytest.mark.parametrize("mx,my", [(5, 7), (33, 6), (40, 31)])
def test_plane_properties(tmp_path, mx, my):
    """2-D: the ghost planes repeat the plane, and the three planes within one
    ghost layer share its properties."""
    d = check(cases.ramp_case(tmp_path / "c", mx, my, total_step=3, output_screen=1), 3,
              ("bv", "mul", "conductivity", "acoustic"), 1e-12)
    g = d.info().ngg
    bv = d.get(0, "bv")
    for k in range(bv.shape[1]):
        assert np.array_equal(bv[:, k], bv[:, g])
    for f in ("mul", "conductivity", "acoustic"):
        a = d.get(0, f)[0]
        for k in (g - 1, g + 1):
            assert np.array_equal(a[k, g - 1:-g + 1, g - 1:-g + 1], a[g, g - 1:-g + 1, g - 1:-g + 1], equal_nan=True)
