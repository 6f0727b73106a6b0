"""CHEMKIN reader and chemistry known-answer / conservation checks (CPU).

The reference ships no tests; these pin the parse of its own mechanism
(input_files/chemistry) and physical invariants of the oracle's chemistry."""
import ctypes as C
import math
import random
import struct
import subprocess
from fractions import Fraction as F
from pathlib import Path

import numpy as np
import pytest

import openstc_b200 as ostc
from openstc_b200 import cases
from oracle_bridge import oracle_lib, orc_params_from

R_U, R_C = 8314.462618, 1.98720425864083
SPECIES = ["H2", "H", "O2", "O", "OH", "HO2", "H2O2", "H2O", "N2"]
ELEMENTS = {"H2": (2, 0, 0), "H": (1, 0, 0), "O2": (0, 2, 0), "O": (0, 1, 0), "OH": (1, 1, 0), "HO2": (1, 2, 0),
            "H2O2": (2, 2, 0), "H2O": (2, 1, 0), "N2": (0, 0, 2)}  # (H, O, N)


@pytest.fixture(scope="module")
def drv(case_factory):
    case = case_factory("ml", cases.mixing_layer_case, mx=12, my=10, mz=6, total_step=2, output_screen=1)
    return ostc.Driver(case)


@pytest.fixture(scope="module")
def params(drv):
    return drv.params()


def test_mechanism_shape(params):
    assert params.ns == 9 and params.nr == 19
    labels = list(params.label[:19])
    # third body (4) for the four "+M" reactions, Troe (6) for the two (+M)
    # fall-off reactions, DUPLICATE pairs merged into one type-3 reaction each
    assert labels == [1, 1, 1, 1, 4, 4, 4, 4, 6, 1, 1, 1, 1, 3, 6, 1, 1, 1, 3]


def test_molecular_weights(params):
    w = {"H": 1.008, "O": 15.999, "N": 14.007}
    for k, name in enumerate(SPECIES):
        h, o, n = ELEMENTS[name]
        expect = 0.0
        for sym, cnt in sorted({"H": h, "N": n, "O": o}.items()):  # element map order
            expect += w[sym] * cnt
        assert params.mw[k] == expect


def test_activation_energies_and_dup(params):
    # main-line Ea divided by R_c; LOW Ea kept in the file's units (reference quirk)
    assert params.Ea[0] == 1.66e4 / R_C
    assert params.A2[8] == 6.37e20 and params.b2[8] == -1.72 and params.Ea2[8] == 5.25e2
    # HO2+HO2 duplicate pair: second Arrhenius set, Ea divided by R_c
    assert params.A[13] == 4.2e14 and params.A2[13] == 1.3e11 and params.Ea2[13] == -1.63e3 / R_C
    # Troe parameters of H+O2(+M)
    assert (params.troe_alpha[8], params.troe_t3[8], params.troe_t1[8]) == (0.8, 1e-30, 1e30)
    # third-body efficiencies of H+O2(+M): H2 2.0, H2O 11.0, O2 0.78, others 1
    tb = [params.third_body[8 * 9 + k] for k in range(9)]
    assert tb == [2.0, 1.0, 0.78, 1.0, 1.0, 1.0, 1.0, 11.0, 1.0]
    # reaction orders: H2+M=H+H+M is +1, O+O+M=O2+M is -1
    assert params.order[4] == 1 and params.order[5] == -1


def test_nasa7_cp_known_values(drv, params):
    """cp(298.15 K) from the therm.dat coefficients, evaluated here directly."""
    p = orc_params_from(params)
    h = np.zeros(20)
    cp = np.zeros(20)
    oracle_lib().orc_enthalpy_cp(C.byref(p), 298.15, h.ctypes.data_as(C.POINTER(C.c_double)),
                                 cp.ctypes.data_as(C.POINTER(C.c_double)))
    # N2's own line sets T_low = 300 K, so below it cp is frozen at cp(300 K)
    # (src/Thermo.cu:47-61); its low-range coefficients from therm.dat:
    assert params.t_low[8] == 300.0
    t = 300.0
    a = [0.03298677e2, 0.14082404e-2, -0.03963222e-4, 0.05641515e-7, -0.02444854e-10]
    cp_n2 = (a[0] + a[1] * t + a[2] * t ** 2 + a[3] * t ** 3 + a[4] * t ** 4) * R_U / params.mw[8]
    assert cp[8] == pytest.approx(cp_n2, rel=1e-13)
    assert cp[8] == pytest.approx(1040.0, rel=0.01)  # tabulated cp of N2 at 298 K
    assert cp[7] == pytest.approx(1864.0, rel=0.01)  # H2O
    assert cp[0] == pytest.approx(14300.0, rel=0.01)  # H2


def _source(params, rho, t, Y):
    p = orc_params_from(params)
    om = np.zeros(20)
    jac = np.zeros(400)
    Yc = np.zeros(20)
    Yc[:9] = Y
    oracle_lib().orc_chemical_source(C.byref(p), rho, t, Yc.ctypes.data_as(C.POINTER(C.c_double)),
                                     om.ctypes.data_as(C.POINTER(C.c_double)),
                                     jac.ctypes.data_as(C.POINTER(C.c_double)))
    return om[:9], jac[:81].reshape(9, 9)


@pytest.mark.parametrize("t", [900.0, 1500.0, 2400.0])
def test_source_conserves_mass_and_elements(params, t):
    rng = np.random.default_rng(int(t))
    Y = rng.dirichlet(np.ones(9))
    om, _ = _source(params, 0.3, t, Y)
    scale = np.max(np.abs(om))
    assert scale > 0
    assert abs(om.sum()) < 1e-12 * scale
    for e in range(3):
        moles = sum(ELEMENTS[s][e] * om[k] / params.mw[k] for k, s in enumerate(SPECIES))
        assert abs(moles) < 1e-12 * scale


def test_jacobian_columns_conserve_mass_and_elements(params):
    """Every reaction conserves mass and elements, so each column of the EPI
    Jacobian sums to zero, by mass and by element moles."""
    rng = np.random.default_rng(7)
    Y = rng.dirichlet(np.ones(9)) * 0.9 + 0.1 / 9
    _, J = _source(params, 0.25, 1800.0, Y)
    scale = np.max(np.abs(J))
    assert scale > 0
    assert np.max(np.abs(J.sum(axis=0))) < 1e-12 * scale
    for e in range(3):
        w = np.array([ELEMENTS[s][e] / params.mw[k] for k, s in enumerate(SPECIES)])
        assert np.max(np.abs(w @ J)) < 1e-12 * scale


def test_epi_increment_conserves_mass(params):
    p = orc_params_from(params)
    Y = np.zeros(20)
    Y[:9] = [0.02, 1e-4, 0.2, 1e-4, 1e-3, 1e-5, 1e-6, 0.1, 0.0]
    Y[8] = 1.0 - Y[:8].sum()
    dY = np.zeros(20)
    oracle_lib().orc_epi_increment(C.byref(p), 0.2, 1800.0, Y.ctypes.data_as(C.POINTER(C.c_double)), 1e-6,
                                   dY.ctypes.data_as(C.POINTER(C.c_double)))
    assert np.max(np.abs(dY[:9])) > 0
    assert abs(dY[:9].sum()) < 1e-12 * np.max(np.abs(dY[:9]))


def test_compile_time_mechanism_is_the_shipped_one(params):
    """The stoichiometry the chemistry kernels unroll over (mechanism.hpp) is
    that of the mechanism file, or the shipped cases would take the general
    loops."""
    import re
    from pathlib import Path

    text = (Path(ostc.__file__).parent / "csrc" / "device" / "mechanism.hpp").read_text()

    def table(name):
        body = text[text.index(name):].split("=", 1)[1].split(";", 1)[0]
        return [int(v) for v in re.findall(r"-?\d+", body)]

    assert table("label[nr]") == list(params.label[:19])
    assert table("sf[nr][ns]") == list(params.stoi_f[:19 * 9])
    assert table("sb[nr][ns]") == list(params.stoi_b[:19 * 9])


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    """quotients(y, xs): the two parts of 1 / y and div_by of every x."""
    d = tmp_path_factory.mktemp("div")
    (d / "div.cpp").write_text("""
#include <cstdio>
#include <cstdlib>
#include "device/known_divisor.hpp"
int main(int, char **argv) {
  const ostc::Reciprocal z = ostc::reciprocal(std::strtod(argv[1], nullptr));
  std::printf("%a %a\\n", z.h, z.l);
  char text[64];
  while (std::scanf("%63s", text) == 1) std::printf("%a\\n", ostc::div_by(std::strtod(text, nullptr), z.h, z.l));
}
""")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I", str(Path(ostc.__file__).parent / "csrc"),
                    str(d / "div.cpp"), "-o", str(d / "div")], check=True)

    def run(y, xs):
        out = subprocess.run([str(d / "div"), y.hex()], input="\n".join(float(x).hex() for x in xs),
                             capture_output=True, text=True, check=True).stdout.split()
        v = [float.fromhex(t) for t in out]
        return v[:2], v[2:]

    return run


def near_middles(y, widest=64):
    """Every significand x whose quotient x / y lies within widest 2^-106 of the
    middle between two doubles, in units of the quotient: x 2^s - (odd) y = d has
    one x for each small d, modulo the odd part of y's significand."""
    Y = int(math.frexp(y)[0] * 2 ** 53)
    t = (Y & -Y).bit_length() - 1
    odd = Y >> t
    xs = []
    if widest >> t == 0:
        return xs  # no d but 0, and no quotient of doubles is a middle
    for s in (53, 54):  # x >= Y: quotient in [1, 2); x < Y: in [1/2, 1)
        for e in range(-(widest >> t), (widest >> t) + 1):
            x = e * pow(2, -(s - t), odd) % odd
            while x < 2 ** 53:
                if x >= 2 ** 52 and (x >= Y) == (s == 53) and (x * 2 ** s - (e << t)) // Y % 2 == 1:
                    xs.append(float(x))
                x += odd
    return xs


def test_division_by_known_divisors_is_the_division(params, quotients):
    """div_by (known_divisor.hpp) gives the bits of x / y for the divisors the FP64
    path uses it for, the molecular weights and 3, and for powers of two: over
    the exponents its operands have, at the quotients nearest to the middle
    between two doubles, and for zeros, infinities and NaN."""
    rng = random.Random(7)
    special = [0.0, -0.0, math.inf, -math.inf, math.nan, 1.7e308, -1.7e308]
    for y in [3.0, 2.0, 16.0] + list(params.mw[:9]):
        xs = [rng.choice([-1, 1]) * rng.uniform(1, 2) * 2.0 ** rng.randint(-950, 1020) for _ in range(2000)]
        hard = near_middles(y)
        assert len(hard) > 20 or y in (3.0, 2.0, 16.0)
        xs += special + hard + [-x for x in hard]
        (h, l), got = quotients(y, xs)
        assert l > 0 and abs(F(h) + F(l) - 1 / F(y)) < F(2) ** -104 / F(y)
        if y == 3.0:
            assert (h, l) == (1.0 / 3.0, 1.850371707708594e-17)  # the literals of div_3
        want = [x / y for x in xs]
        wrong = [x for x, a, b in zip(xs, got, want) if struct.pack("d", a) != struct.pack("d", b) and x == x]
        assert not wrong, (y, [x.hex() for x in wrong[:5]])
        assert math.isnan(got[2000 + special.index(special[4])])


def test_division_of_the_smallest_numbers_is_one_double_off_at_most(params, quotients):
    """Below 2^-960 x zl underflows: the quotient or the double beside it."""
    rng = random.Random(8)
    for y in [3.0] + list(params.mw[:9]):
        xs = [rng.uniform(1, 2) * 2.0 ** rng.randint(-1074, -960) for _ in range(2000)] + [5e-324, 2.3e-308]
        _, got = quotients(y, xs)
        for x, q in zip(xs, got):
            assert abs(F(q) - F(x / y)) <= F(math.ulp(x / y)), (y, x)
