"""Performance cases of the framework, each one pass through its public entry points.

A case is a dict of plain values; ``listed()`` gives the ones that are always
timed, ``draw(rng)`` more of the same ranges.  ``kind`` says which path:

* ``flow``: a batch of steps of the steady loop (``Driver.step``) and the fetch of
  the primitive fields it ends with, as a program does that monitors or saves a run:
  the 2-D laminar ramp, and the 3-D reacting mixing layer in both precisions, with
  the options of its setup files, one or several blocks, with and without the
  chemistry surrogate.
* ``train``: Adam steps of the chemistry surrogate (``Surrogate.train``).
* ``gradients``: loss and gradients of one batch of host samples.
* ``label``: point-implicit chemistry increments of host states.

The case directories hold the repository's own workloads at other sizes; what a
seed changes is the flow field (smooth disturbances of the two streams and of the
radicals in the layer between them), the samples or the weights.

``exact`` restates the step in plain FP64 torch, term by term.  From the case it
takes only what the reader gives: the grid metric, the boundary faces, the model
constants and the initial field.
"""
import atexit
import math
import shutil
import tempfile
from pathlib import Path

import numpy as np
import torch

import openstc_b200 as ostc
from openstc_b200 import cases
from openstc_b200.plt import write_plt

RU, P_ATM, AIR_GAMMA, AIR_MW = 8314.462618, 101325.0, 1.4, 28.9647
LAYER_CFL = 0.02  # the layer ignites; thousands of repeated steps stay on its way there
SPECIES_TRACE = {"H": 4e-5, "O": 8e-4, "OH": 1.2e-3, "HO2": 2e-5, "H2O2": 4e-6}
NET_DIMS = [16, 256, 256, 256, 256, 16]  # the surrogate's padded layer widths
N_IN, N_OUT = 12, 9


# ------------------------------------------------------------------ the cases
def _flow(name, mx, my, mz, steps, **kw):
    c = dict(name=name, kind="flow", flow="ramp" if mz == 1 else "layer", mx=mx, my=my, mz=mz, steps=steps,
             precision="fp64", implicit=1, chem=1, dplur=4, blocks="", surrogate=False)
    c.update(kw)
    return c


def listed():
    return [
        # the laminar ramp at the size of its tests: every kernel is a launch and little more
        _flow("ramp-48x24", 48, 24, 1, 50),
        # the plain-method workload of the benchmark
        _flow("ramp-256x128", 256, 128, 1, 50),
        # the reacting layer at the size of its tests, FP64 with the coupled implicit step
        _flow("layer-fp64-24x16x8", 24, 16, 8, 8),
        # odd sizes, explicit stepping with the diagonal chemistry treatment
        _flow("layer-fp64-explicit-61x43x19", 61, 43, 19, 8, implicit=0, chem=2),
        # the plain FP64 path on a grid that does not fit L2
        _flow("layer-fp64-160x96x64", 160, 96, 64, 4),
        # FP32-bulk arithmetic at odd sizes, small enough for latency to show
        _flow("layer-mixed-45x37x21", 45, 37, 21, 8, precision="mixed"),
        # FP32-bulk arithmetic at the size of the benchmark's reacting workload
        _flow("layer-mixed-384x192x64", 384, 192, 64, 8, precision="mixed"),
        # the same with the surrogate taking the chemistry of the quiet cells
        _flow("layer-surrogate-256x128x64", 256, 128, 64, 8, precision="mixed", surrogate=True),
        # uneven blocks along x with inner faces in the same launches
        _flow("blocks-mixed-5", 0, 53, 43, 8, precision="mixed", blocks="61,34,97,45,76"),
        # training at its benchmark batch
        dict(name="train-65536", kind="train", samples=1 << 20, batch=65536, steps=12, lr=1e-3),
        # one batch's gradients
        dict(name="gradients-8192", kind="gradients", n=8192),
        # labels of host states
        dict(name="label-200003", kind="label", n=200003),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["ramp", "fp64", "fp64", "mixed", "mixed", "surrogate", "blocks", "train", "gradients", "label"])
    if what == "ramp":
        return _unnamed(_flow("", _log(rng, 40, 512), _log(rng, 20, 256), 1, 50))
    if what == "train":
        return dict(kind="train", samples=_log(rng, 100000, 1 << 20), batch=128 * _log(rng, 16, 512), steps=12, lr=1e-3)
    if what == "gradients":
        return dict(kind="gradients", n=128 * _log(rng, 1, 256))
    if what == "label":
        return dict(kind="label", n=_log(rng, 1000, 200000))
    mx, my, mz = _log(rng, 20, 180), _log(rng, 12, 100), _log(rng, 6, 64)
    if what == "fp64":
        implicit = rng.choice([1, 1, 0])
        return _unnamed(_flow("", mx, my, mz, 4, implicit=implicit, chem=rng.choice([1, 1, 2]),
                              dplur=rng.choice([2, 3, 4])))
    if what == "blocks":
        widths = [_log(rng, 16, 90) for _ in range(rng.randint(2, 5))]
        return _unnamed(_flow("", 0, my, mz, 4, precision="mixed", blocks=",".join(map(str, widths))))
    return _unnamed(_flow("", mx, my, mz, 8, precision="mixed", dplur=rng.choice([2, 3, 4]),
                          surrogate=what == "surrogate"))


def _unnamed(c):
    return {k: v for k, v in c.items() if k != "name"}


# --------------------------------------------------------- case directories
_dirs = {}


def _case_dir(c):
    """The case directory of this size and these options, written once."""
    key = (c["flow"], c["mx"], c["my"], c["mz"], c["implicit"], c["chem"], c["dplur"], c["blocks"])
    if key not in _dirs:
        d = Path(tempfile.mkdtemp(prefix="cases_"))
        atexit.register(shutil.rmtree, d, ignore_errors=True)
        screen = 10 ** 6  # no residual falls due within a pass but the first step's
        if c["flow"] == "ramp":
            cases.ramp_case(d, c["mx"], c["my"], output_screen=screen)
            g = d / "input_files" / "setup" / "0_global_control.txt"
            g.write_text(g.read_text().replace("int initial = 0", "int initial = 1"))
            m = d / "output" / "message"
            m.mkdir(parents=True, exist_ok=True)
            (m / "step.txt").write_text("0")
            (m / "residual_scale.txt").write_text("1\n1\n1\n1\n")
        elif c["blocks"]:
            cases.multiblock_case(d, [int(v) for v in c["blocks"].split(",")], c["my"], c["mz"], output_screen=screen,
                                  dplur=c["dplur"], cfl=LAYER_CFL)
        else:
            cases.mixing_layer_case(d, c["mx"], c["my"], c["mz"], output_screen=screen, dplur=c["dplur"],
                                    chem=c["chem"], implicit=c["implicit"], cfl=LAYER_CFL)
        grid = ([cases._mixing_layer_grid(c["mx"], c["my"], c["mz"])] if c["mx"] and c["flow"] == "layer"
                else cases._read_grid(d))
        _dirs[key] = (d, grid)
    return _dirs[key]


def _waves(rng, x, y, z, amplitude):
    """1 + a few smooth waves over the domain, of this amplitude together."""
    s = 1.0
    for _ in range(3):
        a = amplitude / 3
        for q, length in ((x, 0.3), (y, 0.05), (z, 0.02)):
            a = a * np.cos(2 * np.pi * rng.uniform(0.7, 3) * q / length + rng.uniform(0, 6.3))
        s = s + a
    return s


def _write_field(c, seed):
    """The restart file of this case with the seed's flow field."""
    d, grid = _case_dir(c)
    rng = np.random.default_rng(seed)
    zones = []
    if c["flow"] == "ramp":
        gas = RU / AIR_MW
        u0 = 3.0 * math.sqrt(AIR_GAMMA * gas * 220.0)
        names = ["x", "y", "z", "density", "u", "v", "w", "pressure", "temperature", "mach"]
        for x, y, z in grid:
            t, p = 220.0 * _waves(rng, x, y, z, 0.03), 2500.0 * _waves(rng, x, y, z, 0.05)
            zones.append(dict(x=x, y=y, z=z, density=p / (gas * t), u=u0 * _waves(rng, x, y, z, 0.03),
                              v=0.02 * u0 * (_waves(rng, x, y, z, 1.0) - 1), w=0 * x, pressure=p, temperature=t,
                              mach=0 * x))
        write_plt(d / "output" / "field" / "flowfield.plt", names, zones)
        return d
    up, lo = cases.inflow_state(d, cases.UPPER), cases.inflow_state(d, cases.LOWER)
    species = cases._species_names(d)
    names = ["x", "y", "z", "density", "u", "v", "w", "pressure", "temperature", "mach"] + species + [
        "tke", "omega", "mut"]
    state = rng.bit_generator.state
    for full in grid:
        rng.bit_generator.state = state  # the same waves across the blocks
        x, y, z = full[0][:1, :1], full[1][:1, :, :1], full[2][:, :1, :1]  # the grid is a product of its axes
        phi = 0.5 * (1.0 + np.tanh((y - 0.025) / 1e-3))
        mix = lambda a, b: phi * b + (1.0 - phi) * a  # noqa: E731
        hot = 4 * phi * (1 - phi)
        zone = dict(x=full[0], y=full[1], z=full[2], mach=0 * x)
        zone["u"] = mix(lo["u"], up["u"]) * _waves(rng, x, y, z, 0.02)
        zone["v"] = 0.01 * up["u"] * (_waves(rng, x, y, z, 1.0) - 1)
        zone["w"] = 0.01 * up["u"] * (_waves(rng, x, y, z, 1.0) - 1)
        zone["pressure"] = up["pressure"] * _waves(rng, x, y, z, 0.02)
        zone["temperature"] = mix(lo["temperature"], up["temperature"] * _waves(rng, x, y, z, 0.02)) + 500.0 * hot
        Y = {n: mix(lo["sv"][q], up["sv"][q]) for q, n in enumerate(species)}
        strength = hot * _waves(rng, x, y, z, 0.3)
        for n, v in SPECIES_TRACE.items():
            if n in Y:
                Y[n] = Y[n] + v * strength
        total = sum(Y.values())
        Y = {n: v / total for n, v in Y.items()}
        zone["density"] = zone["pressure"] / (RU * zone["temperature"] * sum(Y[n] / w for n, w in zip(species, up["mw"])))
        zone.update(Y)
        ns = len(species)
        zone["tke"] = mix(lo["sv"][ns], up["sv"][ns])
        zone["omega"] = mix(lo["sv"][ns + 1], up["sv"][ns + 1])
        zone["mut"] = mix(lo["mut"], up["mut"])
        zones.append({n: np.broadcast_to(v, full[0].shape) for n, v in zone.items()})
    write_plt(d / "output" / "field" / "flowfield.plt", names, zones)
    return d


# ------------------------------------------------------------------- surrogate
def _tiny_driver():
    """The mechanism a surrogate is made from."""
    return ostc.Driver(_write_field(_flow("", 12, 10, 6, 1), 0), precision="mixed")


def _states(rng, n):
    """T, p, Y[9], dt in the ranges the layer meets."""
    s = np.empty((n, N_IN))
    s[:, 0] = rng.uniform(300.0, 2600.0, n)
    s[:, 1] = 10 ** rng.uniform(4.6, 5.6, n)
    y = rng.dirichlet([0.3, 0.02, 0.3, 0.02, 0.03, 0.2, 0.02, 0.02, 1.0], n) + 1e-12
    s[:, 2:11] = y / y.sum(axis=1, keepdims=True)
    s[:, 11] = 10 ** rng.uniform(-8.5, -6.5, n)
    return s


_NORM = dict(in_mu=[1400.0, 5.1] + [1.0 / 9] * 9 + [-7.5], in_sig=[650.0, 0.3] + [0.2] * 9 + [0.6],
             out_c=[1e-5] * 9, out_s=[2.0] * 9)


def _net_params(rng, out_scale):
    """Flat parameters (per layer the weight, then the bias), He scale."""
    flat = []
    for q in range(5):
        din, dout = NET_DIMS[q], NET_DIMS[q + 1]
        fan, rows = (N_IN if q == 0 else din), (N_OUT if q == 4 else dout)
        w = np.zeros((dout, din), np.float32)
        w[:rows, :fan] = rng.normal(0, math.sqrt(2.0 / fan) * (out_scale if q == 4 else 1.0), (rows, fan))
        b = np.zeros(dout, np.float32)
        b[:rows] = rng.normal(0, 0.05 * (out_scale if q == 4 else 1.0), rows)
        flat += [w.ravel(), b]
    return np.concatenate(flat)


def _load_net(driver, rng, out_scale):
    """A surrogate with the seed's weights, through its saved form."""
    gate = [250.0, 2800.0, 4.5, 6.0, -10.0, -5.5, 1e-3, 0.01, 6.0, 1e-10, 0.25, 1e-4]
    flat = _net_params(rng, out_scale)
    with tempfile.NamedTemporaryFile(suffix=".mlp") as f:
        f.write(b"OSTCMLP5")
        for part in (_NORM["in_mu"], _NORM["in_sig"], _NORM["out_c"], _NORM["out_s"], gate, flat):
            f.write(np.asarray(part, np.float32).tobytes())
        f.flush()
        s = ostc.Surrogate(driver, seed=1)
        s.load(f.name)
    return s, flat


def _increments(rng, states):
    """dY of a size the labels have."""
    return (states[:, 2:11] + 1e-10) * 1e-5 * np.sinh(2.0 * rng.normal(0, 0.8, (len(states), N_OUT)))


# ------------------------------------------------------------ prepare and run
def prepare(case, seed):
    rng = np.random.default_rng([seed, 17])
    if case["kind"] == "flow":
        d = ostc.Driver(_write_field(case, seed), precision=case["precision"])
        d.initialize()
        s = dict(case=case, driver=d, g=d.info().ngg, fields=[])
        for b in range(d.info().n_block):
            for f in ("bv", "sv") if case["flow"] == "layer" else ("bv",):
                t = torch.empty(d.field_shape(b, f), dtype=torch.float64, pin_memory=True)
                s["fields"].append((b, f, t, t.numpy()))
        s["species"] = cases._species_names(d.case_dir) if case["flow"] == "layer" else []
        if case["surrogate"]:
            s["net"], _ = _load_net(d, rng, 0.02)
            d.set_surrogate(s["net"])
        return s
    tiny = _tiny_driver()
    if case["kind"] == "train":
        net = ostc.Surrogate(tiny, seed=seed + 1)
        net.generate(case["samples"], seed=seed + 2)
        return dict(case=case, driver=tiny, net=net)
    states = _states(rng, case["n"])
    if case["kind"] == "label":
        return dict(case=case, driver=tiny, net=ostc.Surrogate(tiny, seed=1), states=states)
    net, _ = _load_net(tiny, rng, 0.5)
    return dict(case=case, driver=tiny, net=net, states=states, dy=_increments(rng, states))


def _parts(case, field, block, v, species):
    """The outputs of a block's interior field: each species by itself, on several blocks together."""
    if field == "bv":
        parts = dict(density=v[0], velocity=v[1:4], pressure=v[4], temperature=v[5])
    elif case["blocks"]:
        parts = dict(species=v[:-2], tke=v[-2], omega=v[-1])
    else:
        parts = {n: v[q] for q, n in enumerate(species + ["tke", "omega"])}
    return {"%s.%d" % (n, block) if case["blocks"] else n: p for n, p in parts.items()}


def run(state):
    case = state["case"]
    if case["kind"] == "flow":
        d, g, out = state["driver"], state["g"], {}
        d.step(case["steps"])
        for b, f, _, a in state["fields"]:
            d.get_into(b, f, a)
            v = a[:, g:-g, g:-g, g:-g]
            out.update(_parts(case, f, b, v, state["species"]))
        return out
    if case["kind"] == "train":
        losses = state["net"].train(case["steps"], batch=case["batch"], lr=case["lr"])
        return dict(losses=losses, params=state["net"].params())
    if case["kind"] == "gradients":
        loss, grads = state["net"].gradients(state["states"], state["dy"])
        return dict(loss=loss, grads=grads)
    return dict(dy=state["net"].label(state["states"]))


def _cells(c):
    mx = sum(int(v) for v in c["blocks"].split(",")) if c["blocks"] else c["mx"]
    return mx * c["my"] * c["mz"]


def work(case):
    """Bytes: of a flow step the conservative and primitive state read and written
    once and the geometry read once, per step, and the fields fetched at the end;
    of training the gathered samples, the weights and the optimiser's state, per
    step.  Operations per cell and step: 3 (2-D: 2) faces' fluxes and limiters, the
    turbulence and chemistry sources, the point-implicit factors and the sweeps."""
    if case["kind"] == "flow":
        n, layer = _cells(case), case["flow"] == "layer"
        state = (6 + 11) + 16 if layer else 6 + 5
        per_cell = 8 * (2 * state + 11)
        flops = 700
        if layer:
            flops = 3 * 900 + 300 + 1800 + (case["dplur"] * (6 * 90 + 162) + 500 if case["implicit"] else 100)
        return dict(bytes=n * (per_cell * case["steps"] + 8 * (17 if layer else 6)), flops=n * flops * case["steps"])
    weights = sum(a * b + b for a, b in zip(NET_DIMS, NET_DIMS[1:]))
    products = sum(a * b for a, b in zip(NET_DIMS, NET_DIMS[1:]))
    if case["kind"] == "train":
        return dict(bytes=case["steps"] * (case["batch"] * (32 + 64) + weights * 4 * 6),
                    flops=case["steps"] * case["batch"] * 6.0 * products)
    if case["kind"] == "gradients":
        return dict(bytes=case["n"] * 8 * (N_IN + N_OUT) + weights * 8, flops=case["n"] * 6.0 * products)
    return dict(bytes=case["n"] * 8 * (N_IN + N_OUT), flops=case["n"] * 2600)


def tolerance(case):
    """FP64: sums in another order, amplified by the stiff chemistry over a pass.
    FP32-bulk: rounding of the single-precision fluxes and properties.
    Training: BF16 products whose rounding Adam's normalised steps carry on."""
    if case["kind"] == "flow":
        return {"rel": 1e-9, "max": 1e-6} if case["precision"] == "fp64" else {"rel": 2e-5, "max": 5e-3}
    if case["kind"] == "train":
        return {"rel": 1e-2, "max": 0.5}
    if case["kind"] == "gradients":
        return {"rel": 5e-3, "max": 0.1}
    return {"rel": 1e-9, "max": 1e-6}


# ----------------------------------------------------------------------- exact
def exact(case, seed):
    if case["kind"] == "flow":
        if case["surrogate"] or _cells(case) * case["steps"] > 5e6:
            return None  # the network is no FP64 quantity; beyond this size it takes too long
        return _Flow(case, seed).outputs()
    if case["kind"] == "train":
        return None  # the samples are drawn on the device and not given back
    rng = np.random.default_rng([seed, 17])
    states = _states(rng, case["n"])
    if case["kind"] == "label":
        return dict(dy=_exact_label(states))
    flat = _net_params(rng, 0.5)
    return _exact_gradients(flat, states, _increments(rng, states))


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a, np.float64), device=_dev())


def _exact_gradients(flat, states, dy):
    f = np.concatenate([states[:, :1], np.log10(states[:, 1:2]), states[:, 2:11], np.log10(states[:, 11:])], axis=1)
    x = np.zeros((len(states), 16))
    x[:, :N_IN] = (f - _NORM["in_mu"]) / _NORM["in_sig"]
    target = _t(np.arcsinh(dy / (states[:, 2:11] + 1e-10) / _NORM["out_c"]) / _NORM["out_s"])
    p = _t(flat).requires_grad_()
    a, at = _t(x), 0
    for q in range(5):
        din, dout = NET_DIMS[q], NET_DIMS[q + 1]
        w, b = p[at:at + din * dout].view(dout, din), p[at + din * dout:at + din * dout + dout]
        at += din * dout + dout
        a = a @ w.T + b
        if q < 4:
            a = torch.nn.functional.gelu(a, approximate="tanh")
    loss = ((a[:, :N_OUT] - target) ** 2).mean()
    loss.backward()
    return dict(loss=float(loss), grads=p.grad.cpu().numpy().astype(np.float32).astype(np.float64))


def _exact_label(states):
    c = _Chem(_tiny_driver().params())
    s = _t(states)
    t, p, Y, dt = s[:, 0], s[:, 1], s[:, 2:11].T, s[:, 11]
    rho = p / (RU * t * (Y / c.mw[:, None]).sum(0))
    omega, jac, _ = c.source(rho, t, Y, jacobian=True)
    eye = torch.eye(c.ns, dtype=torch.float64, device=s.device)[:, :, None]
    x = _solve(eye - dt * jac, omega)
    return (x * dt / rho).T.cpu().numpy()


def _solve(a, b):
    """Per-point linear systems, a[m, n, ...] x[n, ...] = b[m, ...]."""
    n, shape = b.shape[0], b.shape[1:]
    x = torch.linalg.solve(a.reshape(n, n, -1).permute(2, 0, 1), b.reshape(n, -1).T.unsqueeze(-1))
    return x.squeeze(-1).T.reshape(n, *shape)


class _Chem:
    """Thermodynamics, transport and reactions of the mechanism over points [species, ...]."""

    def __init__(self, p):
        ns, nr = self.ns, self.nr = p.ns, p.nr
        vec = lambda a, n=ns: _t(np.ctypeslib.as_array(a)[:n])  # noqa: E731
        table = lambda a, r: np.ctypeslib.as_array(a)[:r * ns].reshape(r, ns).astype(float)  # noqa: E731
        self.mw, self.t_low, self.t_mid = vec(p.mw), vec(p.t_low), vec(p.t_mid)
        self.low = _t(np.ctypeslib.as_array(p.low_coeff)[:ns * 7].reshape(ns, 7))
        self.high = _t(np.ctypeslib.as_array(p.high_coeff)[:ns * 7].reshape(ns, 7))
        self.lj, self.visc = vec(p.lj_inv), vec(p.vis_coeff)
        self.wq, self.w8 = _t(table(p.w_quarter, ns)), _t(table(p.w_sqrt8, ns))
        self.sf, self.sb = table(p.stoi_f, nr), table(p.stoi_b, nr)
        self.tb = _t(table(p.third_body, nr))
        self.p, self.Sc = p, p.Sc

    def _c(self, t):
        """NASA-7 coefficients by species and point, and the temperature they are taken at."""
        sh = (self.ns,) + (1,) * t.dim()
        cold, mid = t < self.t_low.view(sh), t < self.t_mid.view(sh)
        c = [torch.where(mid | cold, self.low[:, q].view(sh), self.high[:, q].view(sh)) for q in range(7)]
        return c, torch.where(cold, self.t_low.view(sh), t.expand(self.ns, *t.shape)), sh

    def h_cp(self, t):
        c, tt, sh = self._c(t)
        cp = c[0] + tt * (c[1] + tt * (c[2] + tt * (c[3] + tt * c[4])))
        h = tt * (c[0] + tt * (c[1] / 2 + tt * (c[2] / 3 + tt * (c[3] / 4 + tt * c[4] / 5)))) + c[5] + cp * (t - tt)
        r = (RU / self.mw).view(sh)
        return h * r, cp * r

    def gibbs(self, t):
        c, tt, _ = self._c(t)
        return (c[0] * (1 - torch.log(tt)) - tt * (c[1] / 2 + tt * (c[2] / 6 + tt * (c[3] / 12 + tt * c[4] / 20)))
                + c[5] / tt - c[6])

    def mean_mw(self, Y):
        return 1 / (Y / self.mw.view((self.ns,) + (1,) * (Y.dim() - 1))).sum(0)

    def transport(self, t, Y, cp):
        """Mixture viscosity, conductivity and rho D by species."""
        sh = (self.ns,) + (1,) * t.dim()
        w = self.mean_mw(Y)
        X = Y * w / self.mw.view(sh)
        tdl = t * self.lj.view(sh)
        vis = self.visc.view(sh) * torch.sqrt(t) / (1.147 * tdl ** -0.145 + (tdl + 0.5) ** -2)
        mu, lam = 0, 0
        for m in range(self.ns):
            vt = X[m]
            for n in range(self.ns):
                if n != m:
                    vt = vt + (1 + torch.sqrt(vis[m] / vis[n]) * self.wq[m, n]) ** 2 * self.w8[m, n] * X[n]
            mu = mu + vis[m] * X[m] / vt
            lam = lam + vis[m] * (cp[m] + 1.25 * RU / self.mw[m]) * X[m] / (1.065 * vt - 0.065 * X[m])
        d = torch.where((X - 1).abs() < 1e-3, (mu / self.Sc).expand(X.shape), (1 - Y) * mu / ((1 - X) * self.Sc))
        return mu, lam, d

    def source(self, rho, t, Y, jacobian):
        """omega [kg/m^3/s], the Jacobian of the point-implicit treatment and the destruction rates."""
        p, ns, sh = self.p, self.ns, (self.ns,) + (1,) * t.dim()
        c = rho * Y / self.mw.view(sh) * 1e-3
        g = self.gibbs(t)
        rate = lambda a, b, e: a * t ** b * torch.exp(-e / t)  # noqa: E731
        omega, destroyed = torch.zeros_like(Y), torch.zeros_like(Y)
        jac = torch.zeros((ns,) + tuple(Y.shape), dtype=Y.dtype, device=Y.device) if jacobian else None
        for r in range(self.nr):
            label = p.label[r]
            kf = rate(p.A[r], p.b[r], p.Ea[r])
            if label == 3:
                kf = kf + rate(p.A2[r], p.b2[r], p.Ea2[r])
            if label > 3:
                cc = (c * self.tb[r].view(sh)).sum(0)
                if label == 4:
                    kf = kf * cc
                else:
                    pr = rate(p.A2[r], p.b2[r], p.Ea2[r]) * cc / kf
                    F = 1.0
                    if label > 5:
                        fc = ((1 - p.troe_alpha[r]) * torch.exp(-t / p.troe_t3[r])
                              + p.troe_alpha[r] * torch.exp(-t / p.troe_t1[r]))
                        if label == 7:
                            fc = fc + torch.exp(-p.troe_t2[r] / t)
                        lf = torch.log10(fc)
                        a = torch.log10(pr) - 0.4 - 0.67 * lf
                        F = 10 ** (lf / (1 + (a / (0.75 - 1.27 * lf - 0.14 * a)) ** 2))
                    kf = kf * pr / (1 + pr) * F
            nu = self.sb[r] - self.sf[r]
            if label == 2:
                kb = rate(p.A2[r], p.b2[r], p.Ea2[r])
            else:
                dg = sum(g[q] * nu[q] for q in range(ns) if nu[q] != 0)
                kb = kf / ((P_ATM / RU * 1e-3 / t) ** p.order[r] * torch.exp(-dg))
            for q in range(ns):
                for _ in range(int(self.sf[r, q])):
                    kf = kf * c[q]
                for _ in range(int(self.sb[r, q])):
                    kb = kb * c[q]
            for q in range(ns):
                m = self.mw[q] * 1e3
                if self.sf[r, q] or self.sb[r, q]:
                    omega[q] += m * nu[q] * (kf - kb)
                    destroyed[q] += m * (kf * self.sf[r, q] + kb * self.sb[r, q])
            if jacobian:
                for n in range(ns):
                    if self.sf[r, n] or self.sb[r, n]:
                        z = torch.where(Y[n] > 1e-25, (self.sf[r, n] * kf - self.sb[r, n] * kb) / (rho * Y[n]), 0.0)
                        for q in range(ns):
                            if nu[q] != 0:
                                jac[q, n] += self.mw[q] * 1e3 * nu[q] * z
        return omega, jac, destroyed


def _sutherland(t):
    return 1.716e-5 * (t / 273) ** 1.5 * (273 + 111) / (t + 111)


def _minmod(a, b):
    s = torch.where(a < 0, -0.5, 0.5) + torch.where(b < 0, -0.5, 0.5)
    return s * torch.minimum(a.abs(), b.abs())


class _Flow:
    """The steady step in FP64 torch; fields [component, k, j, i] with ghost layers."""

    SK1, SO1, B1, A1, SK2, SO2, B2, BS, KAPPA = 0.85, 0.5, 0.0750, 0.31, 1.0, 0.856, 0.0828, 0.09, 0.41

    def __init__(self, case, seed):
        self.case = case
        d = self.d = ostc.Driver(_write_field(case, seed), precision=case["precision"])
        self.p, self.bcs, info = d.params(), d.bcs(), d.info()
        self.g, self.two_d, self.ns = info.ngg, info.dimension == 2, info.n_spec
        self.c = _Chem(self.p) if self.ns else None
        G1 = self.B1 / self.BS - self.SO1 * self.KAPPA ** 2 / 0.3
        G2 = self.B2 / self.BS - self.SO2 * self.KAPPA ** 2 / 0.3
        self.G1, self.G2 = G1, G2
        self.blocks = []
        for b in range(info.n_block):
            B = {f: _t(d.host_field(b, f)) for f in ("jac", "metric", "bv")}
            B["sv"] = _t(d.host_field(b, "sv")) if self.ns else B["bv"][:0]
            B["m"], B["id"] = d.dims(b), b
            z = torch.zeros_like(B["jac"][0])
            for f in ("mul", "cond", "mut", "tcond", "a", "gamma", "cp"):
                B[f] = z.clone()
            B["rho_d"] = z.expand(max(self.ns, 1), *z.shape).clone()
            self.blocks.append(B)
        self.dirs = (0, 1) if self.two_d else (0, 1, 2)
        for B in self.blocks:
            if self.two_d:
                self.copy_k(B)
            self.boundary(B)
            B["cv"] = self.conservative(B)
            if self.ns:
                self.eddy_viscosity_init(B)
        self.exchange()
        for B in self.blocks:
            self.properties(B)

    # ---- windows: [lo, m + hi) in each direction around the interior
    def win(self, a, B, lo=(0, 0, 0), hi=(0, 0, 0)):
        g, m = self.g, B["m"]
        s = [slice(g + lo[q], g + m[q] + hi[q]) for q in range(3)]
        return a[..., s[2], s[1], s[0]]

    def along(self, a, B, d, q, t=None, s=0):
        """Over the faces along d (left cell -1 .. n - 1): the cells q from the left one, s aside along t."""
        lo, hi = [0, 0, 0], [0, 0, 0]
        lo[d], hi[d] = q - 1, q
        if t is not None:
            lo[t], hi[t] = lo[t] + s, hi[t] + s
        return self.win(a, B, lo, hi)

    def difference(self, F, d):
        """F(c + 1/2) - F(c - 1/2) of face values along d."""
        n = F.shape[F.dim() - 1 - d] - 1
        return F.narrow(F.dim() - 1 - d, 1, n) - F.narrow(F.dim() - 1 - d, 0, n)

    def outputs(self):
        for _ in range(self.case["steps"]):
            self.step()
        out = {}
        names = cases._species_names(self.d.case_dir) if self.ns else []
        for B in self.blocks:
            for f in ("bv", "sv") if self.ns else ("bv",):
                out.update(_parts(self.case, f, B["id"], self.win(B[f], B).cpu().numpy(), names))
        return out

    def step(self):
        for B in self.blocks:
            dq = self.residual(B)
            dq = self.implicit(B, dq)
            self.update(B, dq)
            self.boundary(B)
        self.exchange()
        for B in self.blocks:
            if self.two_d:
                self.copy_k(B)
            self.properties(B)

    # ---- state relations
    def conservative(self, B):
        bv, sv = B["bv"], B["sv"]
        rho, ke = bv[0], 0.5 * bv[0] * (bv[1:4] ** 2).sum(0)
        if self.ns:
            h, _ = self.c.h_cp(bv[5])
            E = ke + (h * rho * sv[:self.ns]).sum(0) - bv[4]
        else:
            E = ke + bv[4] / (AIR_GAMMA - 1)
        return torch.cat([rho[None], rho * bv[1:4], E[None], rho * sv])

    def primitives(self, cv, t):
        """bv, sv of conservative values; t: the temperature the Newton iteration starts from."""
        rho, V = cv[0], cv[1:4] / cv[0]
        if not self.ns:
            p = (AIR_GAMMA - 1) * (cv[4] - 0.5 * rho * (V ** 2).sum(0))
            return torch.cat([rho[None], V, p[None], (p * AIR_MW / rho / RU)[None]]), cv[5:]
        sv = cv[5:] / rho
        Y = sv[:self.ns]
        R = RU / self.c.mean_mw(Y)
        e = cv[4] / rho - 0.5 * (V ** 2).sum(0)
        live = torch.ones_like(t, dtype=torch.bool)
        for _ in range(1000):
            h, cp = self.c.h_cp(t)
            t1 = t - ((h * Y).sum(0) - R * t - e) / ((cp * Y).sum(0) - R)
            err = (1 - t1 / t).abs()
            t = torch.where(live, t1, t)
            live = live & (err > 1e-3)
            if not live.any():
                break
        return torch.cat([rho[None], V, (rho * t * R)[None], t[None]]), sv

    def properties(self, B):
        lo, hi = (-1, -1, -1), (1, 1, 1)
        w = lambda a: self.win(a, B, lo, hi)  # noqa: E731
        t = w(B["bv"][5])
        if self.ns:
            Y = w(B["sv"])[:self.ns]
            _, cp = self.c.h_cp(t)
            cpt = (cp * Y).sum(0)
            R = RU / self.c.mean_mw(Y)
            gamma = cpt / (cpt - (Y * (RU / self.c.mw).view(-1, 1, 1, 1)).sum(0))
            mu, lam, d = self.c.transport(t, Y, cp)
            w(B["cp"])[:], w(B["gamma"])[:], w(B["a"])[:] = cpt, gamma, torch.sqrt(gamma * R * t)
            w(B["mul"])[:], w(B["cond"])[:], w(B["rho_d"])[:] = mu, lam, d
        else:
            mu = _sutherland(t)
            w(B["a"])[:], w(B["mul"])[:] = torch.sqrt(AIR_GAMMA * RU / AIR_MW * t), mu
            w(B["cond"])[:] = mu * (AIR_GAMMA * RU / AIR_MW / (AIR_GAMMA - 1)) / self.p.Pr

    # ---- turbulence
    def gradient(self, f, B, lo=(0, 0, 0), hi=(0, 0, 0)):
        """Central d/dx, d/dy, d/dz of a field over a window."""
        met = self.win(B["metric"], B, lo, hi)
        dd = []
        for q in range(3):
            e = [int(q == r) for r in range(3)]
            up = self.win(f, B, [a + b for a, b in zip(lo, e)], [a + b for a, b in zip(hi, e)])
            dn = self.win(f, B, [a - b for a, b in zip(lo, e)], [a - b for a, b in zip(hi, e)])
            dd.append(up - dn)
        return [0.5 * (met[q] * dd[0] + met[3 + q] * dd[1] + met[6 + q] * dd[2]) for q in range(3)]

    def eddy(self, rho, rk, k, om, mul, vort):
        dy = 1e3  # no wall: the reader's distance
        a = torch.maximum(2 * torch.sqrt(k) / (0.09 * om * dy), 500 * mul / (rho * dy * dy * om))
        den = torch.maximum(self.A1 * om, vort * torch.tanh(a * a))
        return torch.where(den > 1e-25, self.A1 * rk / den, 0.0)

    def vorticity(self, gu, gv, gw):
        return torch.sqrt((gv[0] - gu[1]) ** 2 + (gw[0] - gu[2]) ** 2 + (gw[1] - gv[2]) ** 2)

    def eddy_viscosity_init(self, B):
        lo, hi = (-1, -1, -1), (1, 1, 1)
        w = lambda a: self.win(a, B, lo, hi)  # noqa: E731
        t, Y = w(B["bv"][5]), w(B["sv"])[:self.ns]
        mul, _, _ = self.c.transport(t, Y, self.c.h_cp(t)[1])
        vort = self.vorticity(*[self.gradient(B["bv"][q], B, lo, hi) for q in (1, 2, 3)])
        w(B["mut"])[:] = self.eddy(w(B["bv"][0]), w(B["cv"][5 + self.ns]), w(B["sv"][self.ns]), w(B["sv"][self.ns + 1]),
                                   mul, vort)

    def turbulence_source(self, B, dq):
        w = lambda a: self.win(a, B)  # noqa: E731
        ns, dy = self.ns, 1e3
        gu, gv, gw = [self.gradient(B["bv"][q], B) for q in (1, 2, 3)]
        gk, go = self.gradient(B["sv"][ns], B), self.gradient(B["sv"][ns + 1], B)
        rho, k, om, mul = w(B["bv"][0]), w(B["sv"][ns]), w(B["sv"][ns + 1]), w(B["mul"])
        cross = 2 * rho * self.SO2 / om * sum(a * b for a, b in zip(gk, go))
        p1, p2 = torch.sqrt(k) / (0.09 * om * dy), 500 * mul / (rho * dy * dy * om)
        p3 = 4 * rho * self.SO2 * k / (torch.clamp(cross, min=1e-20) * dy * dy)
        f1 = torch.tanh(torch.minimum(torch.maximum(p1, p2), p3) ** 4)
        mut = self.eddy(rho, rho * k, k, om, mul, self.vorticity(gu, gv, gw))
        w(B["mut"])[:] = mut
        w(B["tcond"])[:] = mut * w(B["cp"]) / self.p.Prt
        beta = self.B2 + (self.B1 - self.B2) * f1
        div = gu[0] + gv[1] + gw[2]
        prod = mut * (2 * (gu[0] ** 2 + gv[1] ** 2 + gw[2] ** 2) - 2.0 / 3 * div ** 2 + (gu[1] + gv[0]) ** 2
                      + (gu[2] + gw[0]) ** 2 + (gv[2] + gw[1]) ** 2) - 2.0 / 3 * rho * k * div
        jac, live = w(B["jac"][0]), mut > 1e-25
        dq[5 + ns] += torch.where(live, jac * (prod - self.BS * rho * k * om), 0.0)
        po = (self.G2 + (self.G1 - self.G2) * f1) * rho / mut * prod + (1 - f1) * cross
        dq[6 + ns] += torch.where(live, jac * (po - beta * rho * om * om), 0.0)
        return torch.stack([-2 * self.BS * om, -2 * beta * om])

    # ---- residual
    def residual(self, B):
        w = lambda a: self.win(a, B)  # noqa: E731
        dq = torch.zeros_like(w(B["cv"]))
        if self.ns:
            B["sst_jac"] = self.turbulence_source(B, dq)
            omega, B["J"], gone = self.c.source(w(B["bv"][0]), w(B["bv"][5]), w(B["sv"])[:self.ns],
                                                jacobian=self.p.chem_src_method == 1)
            dq[5:5 + self.ns] += w(B["jac"]) * omega
            if self.p.chem_src_method == 2:
                Y = w(B["sv"])[:self.ns]
                B["J"] = torch.where(Y > 1e-25, -gone / (Y * w(B["bv"][0])), 0.0)
        for d in self.dirs:
            dq -= self.difference(self.inviscid(B, d), d)
            dq += self.difference(self.viscous(B, d), d)
        met = w(B["metric"])
        V = w(B["bv"])[1:4]
        spec, srv = [], 0
        for d in range(3):
            k = met[3 * d:3 * d + 3]
            n = torch.sqrt((k ** 2).sum(0))
            if d in self.dirs:
                spec.append(((k * V).sum(0)).abs() + w(B["a"]) * n)
                srv = srv + n * n
            else:
                spec.append(torch.zeros_like(n))
        gamma = w(B["gamma"]) if self.ns else AIR_GAMMA
        c1 = (torch.clamp(gamma, min=4.0 / 3) if self.ns else AIR_GAMMA) / w(B["bv"][0])
        c2 = w(B["mul"]) / self.p.Pr + (w(B["mut"]) / self.p.Prt if self.ns else 0)
        B["spec"] = spec
        B["dt"] = self.p.cfl / (sum(spec) + srv * c1 * c2)
        return dq

    def inviscid(self, B, d):
        st = [torch.cat([self.along(B["bv"], B, d, q)[:5], self.along(B["sv"], B, d, q)]) for q in (-1, 0, 1, 2)]
        d0, d1, d2 = st[1] - st[0], st[2] - st[1], st[3] - st[2]
        L, R = st[1] + 0.5 * _minmod(d0, d1), st[2] - 0.5 * _minmod(d1, d2)
        jl, jr = self.along(B["jac"][0], B, d, 0), self.along(B["jac"][0], B, d, 1)
        met = B["metric"][3 * d:3 * d + 3]
        k = 0.5 * (jl * self.along(met, B, d, 0) + jr * self.along(met, B, d, 1))
        gk = torch.sqrt((k ** 2).sum(0))
        side = []
        for s in (L, R):
            ke = 0.5 * (s[1:4] ** 2).sum(0)
            if self.ns:
                Y = s[5:5 + self.ns]
                h, cp = self.c.h_cp(s[4] / (s[0] * RU / self.c.mean_mw(Y)))
                cpt = (cp * Y).sum(0)
                gam = cpt / (cpt - (Y * (RU / self.c.mw).view(-1, 1, 1, 1)).sum(0))
                E = s[0] * (ke + (h * Y).sum(0)) - s[4]
            else:
                gam, E = AIR_GAMMA, ke * s[0] + s[4] / (AIR_GAMMA - 1)
            side.append((s, (k * s[1:4]).sum(0) / gk, torch.sqrt(gam * s[4] / s[0]), E))
        c = 0.5 * (side[0][2] + side[1][2])
        ml, mr, al = side[0][1] / c, side[1][1] / c, 3.0 / 16
        quad = lambda m, s: (m + s) ** 2 * 0.25  # noqa: E731
        b, br = (ml * ml - 1) ** 2, (mr * mr - 1) ** 2
        fast, fastr = ml.abs() > 1, mr.abs() > 1
        up, un = 0.5 * (ml + ml.abs()), 0.5 * (mr - mr.abs())
        mp = torch.where(fast, up, quad(ml, 1) + 0.125 * b)
        pp = torch.where(fast, up / ml, quad(ml, 1) * (2 - ml) + al * ml * b)
        mn = torch.where(fastr, un, -quad(mr, -1) - 0.125 * br)
        pn = torch.where(fastr, un / mr, quad(mr, -1) * (2 + mr) - al * mr * br)
        pc, mh = pp * L[4] + pn * R[4], mp + mn
        mass = c * (L[0] * 0.5 * (mh + mh.abs()) + R[0] * 0.5 * (mh - mh.abs()))
        coeff, left = mass * gk, mass >= 0
        s, E = torch.where(left, L, R), torch.where(left, side[0][3], side[1][3])
        return torch.cat([coeff[None], coeff * s[1:4] + pc * k, (coeff * (E + s[4]) / s[0])[None], coeff * s[5:]])

    def viscous(self, B, d):
        ns = self.ns
        mid = lambda a: 0.5 * (self.along(a, B, d, 0) + self.along(a, B, d, 1))  # noqa: E731
        met = mid(B["metric"])

        def grad(f):
            dd = []
            for t in range(3):
                if t == d:
                    dd.append(self.along(f, B, d, 1) - self.along(f, B, d, 0))
                else:
                    dd.append(0.25 * (self.along(f, B, d, 0, t, 1) - self.along(f, B, d, 0, t, -1)
                                      + self.along(f, B, d, 1, t, 1) - self.along(f, B, d, 1, t, -1)))
            return [dd[0] * met[q] + dd[1] * met[3 + q] + dd[2] * met[6 + q] for q in range(3)]

        bv, sv = B["bv"], B["sv"]
        k = mid(B["metric"][3 * d:3 * d + 3] * B["jac"])
        u, v, w = [grad(bv[q]) for q in (1, 2, 3)]
        gt = grad(bv[5])
        mul, mut = mid(B["mul"]), mid(B["mut"])
        vis = mul + mut
        txx = vis * (4 * u[0] - 2 * v[1] - 2 * w[2]) / 3
        tyy = vis * (4 * v[1] - 2 * u[0] - 2 * w[2]) / 3
        tzz = vis * (4 * w[2] - 2 * u[0] - 2 * v[1]) / 3
        txy, txz, tyz = vis * (u[1] + v[0]), vis * (u[2] + w[0]), vis * (v[2] + w[1])
        if ns:
            tt = -2.0 / 3 * mid(bv[0] * sv[ns])
            txx, tyy, tzz = txx + tt, tyy + tt, tzz + tt
        f1 = k[0] * txx + k[1] * txy + k[2] * txz
        f2 = k[0] * txy + k[1] * tyy + k[2] * tyz
        f3 = k[0] * txz + k[1] * tyz + k[2] * tzz
        V = mid(bv[1:4])
        q = V[0] * f1 + V[1] * f2 + V[2] * f3 + mid(B["cond"] + B["tcond"]) * (k[0] * gt[0] + k[1] * gt[1] + k[2] * gt[2])
        rows = [torch.zeros_like(f1), f1, f2, f3, q]
        if ns:
            h, _ = self.c.h_cp(mid(bv[5]))
            normal, total = [], 0
            for s in range(ns):
                g = grad(sv[s])
                flux = (mid(B["rho_d"][s]) + mut / self.p.Sct) * (k[0] * g[0] + k[1] * g[1] + k[2] * g[2])
                rows[4] = rows[4] + h[s] * flux
                total = total + flux
                normal.append(flux)
            rows += [normal[s] - mid(sv[s]) * total for s in range(ns)]
            gk, go = grad(sv[ns]), grad(sv[ns + 1])
            rho, tk, om, dy = mid(bv[0]), mid(sv[ns]), mid(sv[ns + 1]), 1e3
            cross = torch.clamp(2 * rho * self.SO2 / om * sum(a * b for a, b in zip(gk, go)), min=1e-20)
            a1 = torch.minimum(torch.maximum(torch.sqrt(tk) / (0.09 * om * dy), 500 * mul / (rho * dy * dy * om)),
                               4 * rho * self.SO2 * tk / (cross * dy * dy))
            f = torch.tanh(a1 ** 4)
            rows.append((mul + mut * (self.SK2 + (self.SK1 - self.SK2) * f)) * sum(a * b for a, b in zip(k, gk)))
            rows.append((mul + mut * (self.SO2 + (self.SO1 - self.SO2) * f)) * sum(a * b for a, b in zip(k, go)))
        return torch.stack(rows)

    # ---- implicit treatment
    def divide(self, B, x, diag):
        """x / (diag - dt * source Jacobian), row by row or as the point-implicit system."""
        ns, dt = self.ns, B["dt"]
        out = x / diag
        if not ns:
            return out
        if self.p.chem_src_method == 1:
            eye = torch.eye(ns, dtype=x.dtype, device=x.device).view(ns, ns, 1, 1, 1)
            out[5:5 + ns] = _solve(eye * diag - dt * B["J"], x[5:5 + ns])
        elif self.p.chem_src_method == 2:
            out[5:5 + ns] = x[5:5 + ns] / (diag - dt * B["J"])
        out[5 + ns:] = x[5 + ns:] / (diag - dt * B["sst_jac"])
        return out

    def implicit(self, B, dq):
        dt = B["dt"]
        if self.p.implicit_method == 0:
            return self.divide(B, dq, torch.ones_like(dt)) if self.ns else dq
        diag = 1 + dt * sum(B["spec"])
        dq0 = dq = self.divide(B, dq, diag)
        for _ in range(self.p.dplur_inner_step):
            tot = torch.zeros_like(dq)
            for d in range(3):
                n, ax = dq.shape[3 - d], 3 - d
                plus, minus = self.jacobian_dq(B, dq, d, 1), self.jacobian_dq(B, dq, d, -1)
                tot.narrow(ax, 1, n - 1).add_(plus.narrow(ax, 0, n - 1), alpha=0.5)
                tot.narrow(ax, 0, n - 1).sub_(minus.narrow(ax, 1, n - 1), alpha=0.5)
            dq = dq0 + self.divide(B, dt * tot, diag)
        return dq

    def jacobian_dq(self, B, x, d, sign):
        ns = self.ns
        bv, sv = self.win(B["bv"], B), self.win(B["sv"], B)
        k, V = self.win(B["metric"], B)[3 * d:3 * d + 3], bv[1:4]
        U = (k * V).sum(0)
        lam = U + sign * B["spec"][d]
        e, t, gamma = 0.5 * (V ** 2).sum(0), bv[5], self.win(B["gamma"], B)
        h, _ = self.c.h_cp(t)
        b3 = gamma * ((RU / self.c.mw).view(-1, 1, 1, 1) * t * x[5:5 + ns]).sum(0)
        b4 = (gamma - 1) * (h * x[5:5 + ns]).sum(0)
        H = (sv[:ns] * h).sum(0) + e
        b1 = (k * x[1:4]).sum(0) - U * x[0]
        b2 = (gamma - 1) * (e * x[0] - (V * x[1:4]).sum(0) + x[4]) + b3 - b4
        return torch.cat([(b1 + lam * x[0])[None], V * b1 + k * b2 + lam * x[1:4], (H * b1 + U * b2 + lam * x[4])[None],
                          lam * x[5:] + sv * b1])

    # ---- update, boundaries, blocks
    def update(self, B, dq):
        w = lambda a: self.win(a, B)  # noqa: E731
        cv = w(B["cv"]) + dq * B["dt"] / w(B["jac"])
        if self.two_d:
            cv[3] = 0
        w(B["cv"])[:] = cv
        bv, sv = self.primitives(cv, w(B["bv"])[5])
        w(B["bv"])[:] = bv
        if self.ns:
            w(B["sv"])[:] = sv

    def copy_k(self, B):
        g = self.g
        for f in ("bv", "sv"):
            B[f][:, :g], B[f][:, g + 1:] = B[f][:, g:g + 1], B[f][:, g:g + 1]

    def boundary(self, B):
        g = self.g
        for f in self.bcs:
            if f.block != B["id"]:
                continue
            d, sg = f.face, f.direction

            def at(a, off):
                s = [slice(g + f.start[q], g + f.end[q] + 1) for q in range(3)]
                s[d] = slice(s[d].start + sg * off, s[d].stop + sg * off)
                return a[..., s[2], s[1], s[0]]

            bv, sv, ns = B["bv"], B["sv"], self.ns
            state = [bv, sv] if ns else [bv]
            if f.type == 6:
                for o in range(1, g + 1):
                    for a in state + [B["mut"]]:
                        at(a, o)[:] = at(a, 0)
            elif f.type == 5:
                v = [f.density, f.u, f.v, f.w, f.pressure, f.temperature]
                for o in range(1, g + 1):
                    at(bv, o)[:] = _t(v).view(6, 1, 1, 1)
                    if ns:
                        at(sv, o)[:] = _t(list(f.sv)[:ns + 2]).view(-1, 1, 1, 1)
                        at(B["mut"], o)[:] = f.mut
            elif f.type == 3:
                k = at(B["metric"], 0)[3 * d:3 * d + 3]
                k = k / torch.sqrt((k ** 2).sum(0))
                inner = at(bv, -1).clone()
                uk = (k * inner[1:4]).sum(0)
                old = inner[1:4]
                inner[1:4] = old - k * uk
                at(bv, 0)[:] = inner
                if ns:
                    at(sv, 0)[:] = at(sv, -1)
                for o in range(1, g + 1):
                    ghost = at(bv, -o).clone()
                    ghost[1:4] = ghost[1:4] - 2 * (k * ghost[1:4]).sum(0) * k
                    at(bv, o)[:] = ghost
                    if ns:
                        at(sv, o)[:] = at(sv, -o)
                        at(B["mut"], o)[:] = at(B["mut"], -o)
                if "cv" in B:
                    self.plane(B, at)
            elif f.type == 2:
                tw = f.t_wall
                p = at(bv, -1)[4].clone()
                at(bv, 0)[:] = torch.stack([p * AIR_MW / (tw * RU), 0 * p, 0 * p, 0 * p, p, tw + 0 * p])
                for o in range(1, g + 1):
                    s = at(bv, -o).clone()
                    t = 2 * tw - s[5]
                    t = torch.where(t <= 0.1 * tw, tw, t)
                    at(bv, o)[:] = torch.cat([(s[4] * AIR_MW / (t * RU))[None], -s[1:4], s[4:5], t[None]])
                if "cv" in B:
                    self.plane(B, at)

    def plane(self, B, at):
        """The conservative values of a boundary plane from its primitives."""
        part = dict(bv=at(B["bv"], 0), sv=at(B["sv"], 0) if self.ns else B["sv"])
        if not self.ns:
            part["sv"] = part["bv"][:0]
        at(B["cv"], 0)[:] = self.conservative(part)

    def exchange(self):
        """The faces between blocks tiled along x: the shared plane averaged, ghosts from the neighbour."""
        g = self.g
        for A, C in zip(self.blocks, self.blocks[1:]):
            n = A["m"][0]
            s = lambda a, B, i, w=1: self.win(a, B)[..., i:i + w]  # noqa: E731
            ave = 0.5 * (s(A["cv"], A, n - 1) + s(C["cv"], C, 0))
            for B, i in ((A, n - 1), (C, 0)):
                s(B["cv"], B, i)[:] = ave
                bv, sv = self.primitives(ave, s(B["bv"], B, i)[5])
                s(B["bv"], B, i)[:], s(B["sv"], B, i)[:] = bv, sv
            for f in ("bv", "sv"):
                rows = (slice(None), slice(g, g + A["m"][2]), slice(g, g + A["m"][1]))
                A[f][rows + (slice(g + n, g + n + g),)] = C[f][rows + (slice(g + 1, g + 1 + g),)]
                C[f][rows + (slice(0, g),)] = A[f][rows + (slice(g + n - 1 - g, g + n - 1),)]
