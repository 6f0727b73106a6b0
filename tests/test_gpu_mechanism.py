"""The chemistry kernels unrolled over the shipped mechanism's stoichiometry
(csrc/device/mechanism.hpp) against the general loops, which any other
mechanism takes: the same mechanism with a reaction of no consequence added
has the same sums in the same order, but is not the one known at compile time."""
import numpy as np
import pytest

import openstc_b200 as ostc
from openstc_b200 import cases

pytestmark = pytest.mark.gpu


def other_mechanism(case):
    """H + O2 = O + OH once more at a rate of 1e-200 of itself."""
    f = case / "input_files" / "chemistry" / "combustion_mechanism.inp"
    head, tail = f.read_text().rsplit("END", 1)
    f.write_text(head + "H+O2=O+OH       3.55E-185    -0.40   1.66E+04\nEND" + tail)
    return case


@pytest.mark.parametrize("precision,implicit,chem", [
    ("fp64", 1, 1), ("fp64", 0, 1), ("fp64", 0, 2), ("fp64", 1, 0), ("mixed", 1, 1), ("mixed", 1, 2)])
def test_unrolled_chemistry_matches_the_general_loops(tmp_path, precision, implicit, chem):
    """Source term, Jacobian and three steps on a grid with remainders: the
    same terms in the same order.  A net source is the difference of forward and
    backward rates that nearly cancel where a reaction is close to equilibrium
    (by up to 1e5 here), so an ulp of the rates may show at 1e-11 of the largest
    source; source and Jacobian get 1e-9 of their largest entry, the state 1e-13
    on the FP64 path and FP32 rounding (1e-6) on the FP32-bulk path."""
    out = []
    for q in range(2):
        case = cases.mixing_layer_case(tmp_path / f"c{q}", mx=35, my=9, mz=5, total_step=3, output_screen=1,
                                       implicit=implicit, chem=chem)
        d = ostc.Driver(other_mechanism(case) if q else case, precision=precision)
        assert d.info().n_reac == 19 + q
        d.initialize()
        d.step(2)
        d.run_phase("source")
        got = {"dq": d.get(0, "dq")}
        if chem:
            got["chem_jac"] = d.get(0, "chem_jac")
        d.step(1)
        got["bv"], got["sv"] = d.get(0, "bv"), d.get(0, "sv")
        out.append(got)
        d.close()
    for f in out[0]:
        a, b = out[0][f], out[1][f]
        kinds = {"dq": [slice(0, 1), slice(1, 4), slice(4, 5), slice(5, 14), slice(14, 15), slice(15, 16)],
                 "bv": [slice(0, 1), slice(1, 4), slice(4, 5), slice(5, 6)],
                 "sv": [slice(0, 9), slice(9, 10), slice(10, 11)]}.get(f, [slice(0, None)])
        for l in kinds:
            x, y = a[l][np.isfinite(b[l])], b[l][np.isfinite(b[l])]
            tol = 1e-6 if precision == "mixed" else (1e-9 if f in ("dq", "chem_jac") else 1e-13)
            assert np.max(np.abs(x - y)) <= tol * np.max(np.abs(y)), (f, l)


@pytest.mark.parametrize("n", [1, 127, 1000])
def test_unrolled_labels_match_the_general_loops(tmp_path, n):
    rng = np.random.default_rng(n)
    s = np.empty((n, 12))
    s[:, 0] = rng.uniform(250, 2800, n)
    s[:, 1] = 10 ** rng.uniform(4.5, 6, n)
    s[:, 2:11] = rng.dirichlet(np.ones(9), n)
    s[::3, 3:9] = 0.0  # no radicals: Jacobian columns below the floor
    s[:, 2:11] /= s[:, 2:11].sum(axis=1, keepdims=True)
    s[:, 11] = 10 ** rng.uniform(-9, -6, n)
    dy = []
    for q in range(2):
        case = cases.mixing_layer_case(tmp_path / f"c{q}", mx=8, my=6, mz=4, total_step=1, output_screen=1)
        d = ostc.Driver(other_mechanism(case) if q else case)
        sur = ostc.Surrogate(d, seed=1)
        dy.append(sur.label(s))
        sur.close()
        d.close()
    scale = np.maximum(np.max(np.abs(dy[1]), axis=1, keepdims=True), 1e-30)
    assert np.max(np.abs(dy[0] - dy[1]) / scale) < 1e-11  # the systems' condition times rounding


SICK = {"Y_NaN": ("sv", 4, np.nan), "Y_huge": ("sv", 1, 1e200), "Y_inf": ("sv", 2, np.inf), "Y_negative": ("sv", 5, -1e-3),
        "T_NaN": ("bv", 5, np.nan), "T_inf": ("bv", 5, np.inf), "T_zero": ("bv", 5, 0.0), "T_tiny": ("bv", 5, 1e-30),
        "T_huge": ("bv", 5, 1e60), "T_negative": ("bv", 5, -5.0), "rho_inf": ("bv", 0, np.inf)}


def same_beyond_rounding(a, b, tol):
    """Equal infinities, NaN in the same places, finite values within tol of the
    cell's largest (components along the first axis)."""
    assert np.array_equal(np.isnan(a), np.isnan(b))
    assert np.array_equal(a[np.isinf(a)], b[np.isinf(b)]) and np.array_equal(np.isinf(a), np.isinf(b))
    f = np.isfinite(a)
    x, y = np.where(f, a, 0.0), np.where(f, b, 0.0)
    assert np.all(np.abs(x - y) <= tol * np.max(np.abs(y), axis=0))


@pytest.mark.parametrize("precision,chem", [("fp64", 1), ("fp64", 2), ("mixed", 1), ("mixed", 2)])
def test_cells_whose_rates_are_not_finite_match_the_general_loops(tmp_path, precision, chem):
    """The general loops multiply every rate with every coefficient, the zeros
    too: an infinite or NaN rate reaches species it does not involve.  One sick
    cell per kind in a row, sources and Jacobian of each the same."""
    out = []
    for q in range(2):
        case = cases.mixing_layer_case(tmp_path / f"c{q}", mx=16, my=9, mz=5, total_step=3, output_screen=1, chem=chem)
        d = ostc.Driver(other_mechanism(case) if q else case, precision=precision)
        d.initialize()
        g = d.info().ngg
        fields = {f: d.get(0, f) for f in ("bv", "sv")}
        fields["sv"][:9] = np.maximum(fields["sv"][:9], 1e-6)  # every species there
        for i, (f, l, v) in enumerate(SICK.values()):
            fields[f][l, g + 2, g + 4, g + 1 + i] = v
        for f, v in fields.items():
            d.set(0, f, v)
        d.run_phase("source")
        out.append((interior_of(d, "dq")[5:14], interior_of(d, "chem_jac")))
        d.close()
    assert not np.all(np.isfinite(out[0][0]))
    for a, b in zip(*out):
        same_beyond_rounding(a, b, 1e-9)


def interior_of(d, f):
    a = d.get(0, f)
    g, _ = d.layout(f)
    return a[:, g:-g, g:-g, g:-g] if g else a


def test_labels_of_states_whose_rates_are_not_finite(tmp_path):
    dy = []
    for q in range(2):
        case = cases.mixing_layer_case(tmp_path / f"c{q}", mx=8, my=6, mz=4, total_step=1, output_screen=1)
        d = ostc.Driver(other_mechanism(case) if q else case)
        states = np.empty((len(SICK) + 1, 12))
        states[:] = [1500.0, 1e5, *([1.0 / 9] * 9), 1e-7]
        for i, (f, l, v) in enumerate(SICK.values()):
            states[i, {"sv": 2 + l, "bv": 0 if l == 5 else 1}[f]] = v
        sur = ostc.Surrogate(d, seed=1)
        dy.append(sur.label(states))
        sur.close()
        d.close()
    assert np.all(np.isfinite(dy[0][-1])) and not np.all(np.isfinite(dy[0]))
    same_beyond_rounding(dy[0].T, dy[1].T, 1e-9)
