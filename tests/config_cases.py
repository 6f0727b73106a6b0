"""Small channels in every model configuration the engines are built for: air
or the nine species, frozen or reacting, laminar or k-omega SST, explicit or DPLUR,
2-D or 3-D, on a bent grid without walls (the wall row of SST cases is subject to
the reference's race in limit_flow)."""
import numpy as np

from openstc_b200 import cases


def channel_case(case, mx=18, my=10, mz=6, species=False, reaction=False, turbulence=False, implicit=1, dplur=2, chem=1,
                 total_step=3):
    i, j, k = np.meshgrid(np.arange(mx), np.arange(my), np.arange(mz), indexing="ij")
    x = 0.002 * i + 2e-4 * np.sin(0.7 * j)
    y = 0.001 * j + 1e-4 * np.sin(0.9 * i + 0.4 * k)
    z = 0.001 * k + (5e-5 * np.cos(0.5 * i) if mz > 1 else 0.0) + 0.0 * x
    cases.write_grid(case, [tuple(np.ascontiguousarray(a.transpose(2, 1, 0)) for a in (x, y, z))])
    js, ie, je, ke = my // 2, mx - 1, my - 1, mz - 1
    faces = [(0, 0, js, je, 0, ke, 5), (0, 0, 0, js - 1, 0, ke, 9), (ie, ie, 0, je, 0, ke, 6),
             (0, ie, 0, 0, 0, ke, 3), (0, ie, je, je, 0, ke, 3)]
    if mz > 1:
        faces += [(0, ie, 0, je, 0, 0, 3), (0, ie, 0, je, ke, ke, 3)]
    cases.write_boundary(case, [faces])
    upper = dict(cases.UPPER, w=0.05)
    lower = dict(cases.LOWER, temperature=900.0, v=0.05)
    if species:
        upper["Y"] = {"O2": 0.24, "H2O": 0.17, "OH": 0.005, "H": 0.001, "N2": 0.584}
    cases.write_setup(case, cases.setup_files(
        dimension=3 if mz > 1 else 2, total_step=total_step, output_file=10 ** 9, output_screen=1, cfl=0.4,
        implicit_method=implicit, dplur_inner_step=dplur, species=species, reaction=reaction, turbulence=turbulence,
        chem_src_method=chem, inflows=[upper, lower]))
    cases.copy_chemistry(case)
    return case


MODELS = {"air": dict(), "air_sst": dict(turbulence=True), "mix": dict(species=True),
          "mix_sst": dict(species=True, turbulence=True), "fr": dict(species=True, reaction=True),
          "fr_sst": dict(species=True, reaction=True, turbulence=True)}

# grids on which the FP64 flux takes rows and columns (test_flux_cuts.py)
FORM_GRIDS = [(33, 9, 7), (65, 37, 19), (129, 65, 33), (97, 61, 31), (41, 23, 1), (250, 130, 1)]
