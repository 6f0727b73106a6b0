"""Every model configuration of the engines (config_cases.py) against the CPU
oracle: the branches of the step that the shipped workloads do not take, among
them the sweeps' terms of air, DPLUR without a source stage, rows, columns and the
2-D plane kernel for mixtures."""
import numpy as np
import pytest

import openstc_b200 as ostc
from config_cases import FORM_GRIDS, MODELS, channel_case
from oracle_bridge import OracleSolver, interior

pytestmark = pytest.mark.gpu

STATE = ["bv", "sv", "cv", "vel", "acoustic", "mach", "mul", "conductivity", "mut", "turb_cond", "rho_d", "gamma", "cp"]


def compare(gpu, orc, fields, tol):
    bad = {}
    for f in fields:
        g, n = gpu.layout(f)
        if n == 0:
            continue
        a = gpu.get(0, f)
        o = interior(orc.get(0, f, a.shape), g)
        a = interior(a, g)
        for l in range(a.shape[0]):
            scale = np.max(np.abs(o[1:4])) if f in ("bv", "cv") and 1 <= l <= 3 else np.max(np.abs(o[l]))
            err = np.max(np.abs(a[l] - o[l])) / max(scale, 1e-30)
            if not err <= tol:
                bad[f, l] = err
    assert not bad, bad


@pytest.mark.parametrize("mz", [6, 1])
@pytest.mark.parametrize("implicit,dplur,chem", [(1, 2, 1), (1, 3, 2), (1, 0, 1), (0, 0, 1)])
@pytest.mark.parametrize("model", MODELS)
def test_three_steps_match_the_oracle(tmp_path, model, implicit, dplur, chem, mz):
    """Within the 1e-9 that CUDA's and libm's ulps grow to over ten steps of the
    shipped cases."""
    if chem == 2 and not MODELS[model].get("reaction"):
        pytest.skip("the chemistry treatment changes nothing without reactions")
    case = channel_case(tmp_path / "c", mz=mz, implicit=implicit, dplur=dplur, chem=chem, **MODELS[model])
    gpu = ostc.Driver(case)
    gpu.initialize()
    orc = OracleSolver(ostc.Driver(case), threads=4)
    orc.initialize()
    err = gpu.step(3)
    for s in range(1, 4):
        orc.step(s)
    compare(gpu, orc, STATE, 1e-9)
    assert np.isfinite(err)
    gpu.run_phase("residual")
    orc.phase("residual", 0)
    compare(gpu, orc, ["dq", "dt_local", "inv_spec"], 1e-8)  # differences of the state's fluxes
    gpu.close()


@pytest.mark.parametrize("dims", FORM_GRIDS)
@pytest.mark.parametrize("model", MODELS)
def test_flux_forms_agree(tmp_path, model, dims):
    """Rows or columns, as the grid takes them, against the per-cell kernel: dq and
    the time step bit for bit."""
    mx, my, mz = dims
    case = channel_case(tmp_path / "c", mx=mx, my=my, mz=mz, implicit=0, **MODELS[model])
    got = []
    for variant in (0, 1):
        d = ostc.Driver(case)
        d.initialize()
        d.set_tuning(0, variant)
        d.step(2)
        got.append((d.get(0, "dq"), d.get(0, "dt_local")))
        d.close()
    for x, y in zip(*got):
        assert np.array_equal(x, y, equal_nan=True)
