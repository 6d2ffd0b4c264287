"""Performance cases: what a program of this framework has it do, through its public entry points.

A weather code calls the ten stencils on device fields in the reference layout
(``call``), their tangent-linear and adjoint forms in variational assimilation
(``tangent_linear``, ``adjoint``), the chained dycore step with its adjoint (``ChainPlan``)
and ensembles of uneven members (``BatchPlan``).  A case is one such pass:

* ``call``    -- each stencil of ``kernels`` once, in order, on the current stream;
* ``adjoint`` -- the adjoint of each stencil of ``kernels`` once;
* ``tl``      -- the tangent-linear form of each stencil of ``kernels`` once;
* ``chain``   -- one chained step, forward and then adjoint;
* ``batch``   -- the same for every member of an ensemble, replayed by one plan.

Fields have the shapes and distributions of the benchmark's workloads: velocities of smooth
modes plus noise, pressures and heights monotone in k, Courant numbers within 0.8, and, for
``fronts``, steep tanh fronts on the dynamic fields so that limiters and upwind switches
change branch often.  Everything is made on the GPU from the seed alone.
"""
import math
import zlib

import numpy as np
import torch
import torch.nn.functional as F

from __graft_entry__ import load_package

STENCILS = ("laplace", "hdiffsa", "hdiffsmag", "hadvuv", "hadvuv5th", "fastwavesuv", "uvbke", "nh_p_grad", "p_grad_c",
            "fvtp2d")
# the stencils whose adjoints the benchmark's differentiation workload runs
DIFFERENTIATED = ("hdiffsmag", "hadvuv5th", "fastwavesuv", "fvtp2d")

# Per stencil: inputs (name -> generator), 1-D per-latitude inputs, outputs, the active inputs of
# the derivatives, the outputs that adjoint seeds stand for, scalars, and arithmetic operations a
# point (square roots and divisions counted as one).
_ADV1 = ("acrlat0", "acrlat1", "tgrlatda0", "tgrlatda1")
_TABLE = {
    "laplace": dict(in3={"in": "vel"}, in1=(), out=("out",), active=("in",), seeds=("out",), scalars=(), ops=5),
    "hdiffsa": dict(in3={"in": "vel", "mask": "mask"}, in1=("crlato", "crlatu"), out=("out",), active=("in",),
                    seeds=("out",), scalars=(), ops=22),
    "hdiffsmag": dict(in3={"uin": "vel", "vin": "vel", "mask": "unit"},
                      in1=("crlavo", "crlavu", "crlato", "crlatu", "acrlat0"), out=("uout", "vout"),
                      active=("uin", "vin"), seeds=("uout", "vout"),
                      scalars=("eddlat", "eddlon", "tau_smag", "weight_smag"), ops=56),
    "hadvuv": dict(in3={"uin": "vel", "vin": "vel"}, in1=_ADV1, out=("uout", "vout"), active=("uin", "vin"),
                   seeds=("uout", "vout"), scalars=("eddlat", "eddlon"), ops=62),
    "hadvuv5th": dict(in3={"uin": "vel", "vin": "vel"}, in1=_ADV1, out=("uout", "vout"), active=("uin", "vin"),
                      seeds=("uout", "vout"), scalars=("eddlat", "eddlon"), ops=74),
    "fastwavesuv": dict(in3={"uin": "vel", "vin": "vel", "utens": "tend", "vtens": "tend", "wgtfac": "weight",
                             "ppuv": "ppert", "hhl": "height", "rho": "density"}, in1=("fx",), out=("uout", "vout"),
                        active=("uin", "vin", "utens", "vtens", "ppuv"), seeds=("uout", "vout"),
                        scalars=("edadlat", "dt"), ops=35),
    "uvbke": dict(in3={"uc": "vel", "vc": "vel", "cosa": "cosa", "rsina": "rsina"}, in1=(), out=("ub", "vb"),
                  active=("uc", "vc"), seeds=("ub", "vb"), scalars=("dt5",), ops=10),
    "nh_p_grad": dict(in3={"uin": "vel", "vin": "vel", "rdx": "rdx", "rdy": "rdx", "gz": "geopot", "pp": "pres",
                           "pk3": "pres", "wk1": "thick"}, in1=(), out=("uout", "vout"),
                      active=("uin", "vin", "gz", "pp", "pk3", "wk1"), seeds=("uout", "vout"), scalars=("dt",), ops=43),
    "p_grad_c": dict(in3={"uin": "vel", "vin": "vel", "rdxc": "rdx", "rdyc": "rdx", "delpc": "thick", "gz": "geopot",
                          "pkc": "pres"}, in1=(), out=("uout", "vout"), active=("uin", "vin", "delpc", "gz", "pkc"),
                     seeds=("uout", "vout"), scalars=("dt2",), ops=24),
    "fvtp2d": dict(in3={"q": "tracer", "crx": "courant", "cry": "courant", "ra_x": "area", "ra_y": "area",
                        "xfx": "courant", "yfx": "courant", "area": "area"}, in1=(),
                   out=("q_i", "q_j", "fx1", "fx2", "fy1", "fy2"), active=("q",), seeds=("fx1", "fy1"),
                   scalars=("p1", "p2"), ops=100),
}
_PPM = {"p1": 0.583333, "p2": 0.083333}

# The chained step's inputs: (name, generator), 1-D inputs, and where its scalars come from.
_CHAIN3 = {"u": "vel", "v": "vel", "utens": "tend", "vtens": "tend", "wgtfac": "weight", "ppuv": "ppert",
           "hhl": "height", "rho": "density", "mask": "unit", "crx": "courant", "cry": "courant", "ra_x": "area",
           "ra_y": "area", "xfx": "courant", "yfx": "courant", "area": "area"}
_CHAIN1 = ("fx",) + _ADV1 + ("crlavo", "crlavu", "crlato", "crlatu", "smag_acrlat0")
_CHAIN_OUT = ("uout", "vout", "fx1", "fy1")
_CHAIN_HALO = 8


# ---------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------
def _case(name, kind, kernels, dtype, nx, ny, nz, workload="physical", halo=3):
    return {"name": name, "kind": kind, "kernels": kernels, "dtype": dtype, "nx": nx, "ny": ny, "nz": nz,
            "workload": workload, "halo": halo}


def listed():
    ten, four = ",".join(STENCILS), ",".join(DIFFERENTIATED)
    return [
        # the smallest benchmark domain, one limited diffusion a call: a single-column-block run or a
        # nest, where the launch and the call's own latency count
        _case("hdiffsa_f64_64x64x60", "call", "hdiffsa", "f64", 64, 64, 60, "smooth"),
        # the headline workload: all ten stencils in the reference's own precision
        _case("ten_f64_128x128x80", "call", ten, "f64", 128, 128, 80),
        # the FP32-storage workload with fronts: all ten stencils at the benchmark's FP32 size
        _case("ten_f32_256x256x80", "call", ten, "f32", 256, 256, 80, "fronts"),
        # tracer transport, called once per tracer and sub-step: the most expensive single stencil
        _case("fvtp2d_f32_256x256x80", "call", "fvtp2d", "f32", 256, 256, 80, "fronts"),
        # the widest-reach advection on the largest ensemble domain (320 wide, 137 levels)
        _case("hadvuv5th_f32_320x304x137", "call", "hadvuv5th", "f32", 320, 304, 137),
        # horizontal diffusion of a regional domain whose sides are odd: ragged tiles everywhere
        _case("hdiffsmag_f32_201x173x61", "call", "hdiffsmag", "f32", 201, 173, 61, "fronts", 4),
        # a pressure gradient on a small ensemble member
        _case("nh_p_grad_f32_96x80x40", "call", "nh_p_grad", "f32", 96, 80, 40),
        # the adjoint sweep of a variational assimilation, in both precisions
        _case("adjoint_f64_128x128x80", "adjoint", four, "f64", 128, 128, 80),
        _case("adjoint_f32_128x128x80", "adjoint", four, "f32", 128, 128, 80),
        # its inner loop's tangent-linear sweep
        _case("tl_f32_128x128x80", "tl", four, "f32", 128, 128, 80),
        # the chained dycore step, forward and adjoint with recomputation
        _case("chain_f32_128x128x80", "chain", "", "f32", 128, 128, 80),
        # an uneven ensemble of both precisions, replayed by one batch plan (the members' sizes
        # follow from nx, ny, nz: see _members)
        _case("batch_mixed_240x208x60", "batch", "", "mixed", 240, 208, 60),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: any stencil and form, both precisions, sides 32 to 320 (every
    integer), 5 to 137 levels, a halo of 3 or 4 (8 or 9 for the chained step)."""
    kind = rng.choices(("call", "adjoint", "tl", "chain", "batch"), (50, 20, 10, 12, 8))[0]
    dtype = rng.choice(("f64", "f32"))
    kernels = "" if kind in ("chain", "batch") else rng.choice(STENCILS)
    if kind == "call" and rng.random() < 0.15:
        kernels = ",".join(STENCILS)
    # points: no drawn case costs more than the largest listed ones
    most = {"call": 13000000 if dtype == "f32" else 6000000, "adjoint": 4000000, "tl": 4000000, "chain": 1300000,
            "batch": 2900000}[kind]
    if "," in kernels:
        most = 5200000 if dtype == "f32" else 1300000
    while True:
        nx, ny, nz = _log_int(rng, 32, 320), _log_int(rng, 32, 320), _log_int(rng, 5, 137)
        if nx * ny * nz <= most:
            break
    halo = rng.choice((3, 4)) if kind not in ("chain", "batch") else rng.choice((8, 9))
    workload = rng.choice(("physical", "fronts"))
    return {"kind": kind, "kernels": kernels, "dtype": "mixed" if kind == "batch" else dtype, "nx": nx, "ny": ny,
            "nz": nz, "workload": workload, "halo": halo}


def _members(case):
    """(nx, ny, nz, dtype) of a batch case's members: uneven, both precisions."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return [(nx, ny, nz, "f32"), (max(16, nx // 2), max(16, (2 * ny) // 3), nz, "f64"),
            (max(16, nx // 3), ny, max(4, nz // 2), "f32"), (max(16, (3 * nx) // 5), max(16, ny // 4), nz, "f64")]


def _size(dtype):
    return 8 if dtype == "f64" else 4


def _kernels(case):
    return case["kernels"].split(",")


def work(case):
    """Every 3-D input read once, every 3-D output written once, over the interior."""
    kind = case["kind"]
    if kind in ("chain", "batch"):
        members = _members(case) if kind == "batch" else [(case["nx"], case["ny"], case["nz"], case["dtype"])]
        nbytes = flops = 0
        for nx, ny, nz, dtype in members:
            # forward: the inputs and four outputs; adjoint: the inputs again, four seeds, two gradients
            nbytes += nx * ny * nz * _size(dtype) * (2 * len(_CHAIN3) + 10)
            flops += nx * ny * nz * 3 * (sum(_TABLE[k]["ops"] for k in DIFFERENTIATED) + 4)
        return {"bytes": nbytes, "flops": flops}
    pts = case["nx"] * case["ny"] * case["nz"]
    fields = ops = 0
    for k in _kernels(case):
        t = _TABLE[k]
        if kind == "call":
            fields += len(t["in3"]) + len(t["out"])
            ops += t["ops"]
        elif kind == "tl":
            fields += len(t["in3"]) + len(t["active"]) + len(t["out"])
            ops += 2 * t["ops"]
        else:
            fields += len(_adjoint_state(k)) + len(t["seeds"]) + len(t["active"])
            ops += 2 * t["ops"]
    return {"bytes": pts * fields * _size(case["dtype"]), "flops": pts * ops}


def _adjoint_state(kernel):
    """The 3-D state fields an adjoint's value depends on (inputs it is linear in are not read)."""
    return {"laplace": (), "fastwavesuv": ("wgtfac", "hhl", "rho"), "uvbke": ("cosa", "rsina"),
            "nh_p_grad": ("rdx", "rdy", "gz", "pp", "pk3", "wk1"),
            "p_grad_c": ("rdxc", "rdyc", "delpc", "gz", "pkc")}.get(kernel, tuple(_TABLE[kernel]["in3"]))


# ---------------------------------------------------------------------------------------
# inputs, made on the GPU
# ---------------------------------------------------------------------------------------
class _Maker:
    """Fields of one domain (whole allocations, halo included), each from its own stream."""

    def __init__(self, nx, ny, nz, halo, workload, seed, device):
        self.nx, self.ny, self.nz, self.h, self.workload, self.seed = nx, ny, nz, halo, workload, seed
        self.device = device
        axis = lambda n: torch.arange(-halo, n + halo, dtype=torch.float64, device=device)  # noqa: E731
        self.i, self.j, self.k = axis(nx)[None, None, :], axis(ny)[None, :, None], axis(nz)[:, None, None]
        self.shape = (nz + 2 * halo, ny + 2 * halo, nx + 2 * halo)

    def begin(self, label):
        key = zlib.crc32(label.encode())
        self.rng = np.random.default_rng([self.seed, key])
        self.gen = torch.Generator(device=self.device).manual_seed((self.seed * 1000003 + key) % (1 << 62))

    def normal(self, scale):
        return scale * torch.randn(self.shape, generator=self.gen, device=self.device, dtype=torch.float64)

    def uniform(self, lo, hi, shape=None):
        u = torch.rand(shape or self.shape, generator=self.gen, device=self.device, dtype=torch.float64)
        return lo + (hi - lo) * u

    def modes(self, vertical=True):
        out = 0.0
        for _ in range(3):
            kx, ky = (int(v) for v in self.rng.integers(1, 5, size=2))
            phi, psi, chi = (float(v) for v in self.rng.uniform(0, 2 * math.pi, size=3))
            m = torch.sin(2 * math.pi * kx * self.i / self.nx + phi) * torch.cos(2 * math.pi * ky * self.j / self.ny + psi)
            if vertical:
                kz = int(self.rng.integers(1, 3))
                m = m * (1.0 + 0.5 * torch.sin(2 * math.pi * kz * self.k / self.nz + chi))
            out = out + m
        return out

    def front(self):
        """A straight tanh front two cells wide, zero where the workload has none."""
        if self.workload != "fronts":
            return 0.0
        theta = float(self.rng.uniform(0, 2 * math.pi))
        ci, cj = float(self.rng.uniform(0.25, 0.75)) * self.nx, float(self.rng.uniform(0.25, 0.75)) * self.ny
        return torch.tanh(((self.i - ci) * math.cos(theta) + (self.j - cj) * math.sin(theta)) / 2.0)

    def profile(self, bottom, top):
        frac = self.k / max(self.nz - 1, 1)
        return (bottom + (top - bottom) * frac) * (1.0 + 0.01 * self.modes(vertical=False) / 3.0)

    def field(self, label, cls):
        self.begin(label)
        if self.workload == "smooth" and cls == "vel":
            f = self.modes() + self.uniform(0.0, 1e-3)
        elif cls == "vel":
            f = 10.0 * self.modes() + self.normal(0.1) + 10.0 * self.front()
        elif cls == "tend":
            f = 1e-3 * (10.0 * self.modes() + self.normal(0.1) + 10.0 * self.front())
        elif cls == "mask":
            f = self.uniform(0.0, 0.025)
        elif cls == "unit":
            f = self.uniform(0.0, 1.0)
        elif cls == "weight":
            f = self.uniform(0.4, 0.6)
        elif cls == "ppert":
            f = 100.0 * self.modes() + self.normal(1.0)
        elif cls == "height":
            f = 20000.0 * (1.0 - self.k / self.nz) * (1.0 + 0.01 * self.modes(vertical=False) / 3.0)
        elif cls == "density":
            f = 1.2 * (1.0 + 0.01 * self.modes())
        elif cls == "cosa":
            f = 0.2 * self.modes() / 3.0
        elif cls == "rsina":
            f = 1.0 + 0.05 * self.modes() / 3.0
        elif cls == "rdx":
            f = self.uniform(1.0, 1.1)
        elif cls == "geopot":
            f = 9.81 * self.profile(1000.0, 16000.0)
        elif cls == "pres":
            f = self.profile(1000.0, 100.0)
        elif cls == "thick":
            f = 10.0 * (1.0 + 0.01 * self.modes())
        elif cls == "tracer":
            f = self.modes() + self.normal(0.05) + self.front()
            f = f - f.mean()
        elif cls == "courant":
            f = self.modes() + self.normal(0.05) + self.front()
            f = 0.8 * f / f.abs().max()
        elif cls == "area":
            f = 1.0 + 0.1 * self.modes() / 3.0
        elif cls == "seed":
            f = self.normal(1.0)
        else:
            raise KeyError(cls)
        return f.expand(self.shape).contiguous()

    def line(self, label):
        self.begin(label)
        return self.uniform(1.0, 1.1, (self.ny + 2 * self.h,))

    def scalar(self, label):
        name = label.rsplit(".", 1)[-1]
        if name in _PPM:
            return _PPM[name]
        self.begin(label)
        return float(self.rng.uniform(0.01, 0.1))


def _round(x, dtype):
    return x.to(torch.float64 if dtype == "f64" else torch.float32)


def _stencil_inputs(case, seed, device):
    """{kernel: (fields, scalars, seeds, perturbations)} of the case, fields rounded to its type."""
    m = _Maker(case["nx"], case["ny"], case["nz"], case["halo"], case["workload"], seed, device)
    dt = case["dtype"]
    out = {}
    for k in _kernels(case):
        t = _TABLE[k]
        fields = {n: _round(m.field("%s.%s" % (k, n), c), dt) for n, c in t["in3"].items()}
        fields.update({n: _round(m.line("%s.%s" % (k, n)), dt) for n in t["in1"]})
        scalars = {n: m.scalar("%s.%s" % (k, n)) for n in t["scalars"]}
        seeds, dx = {}, {}
        if case["kind"] == "adjoint":
            seeds = {n: _round(m.field("%s.%sb" % (k, n), "seed"), dt) for n in t["seeds"]}
        if case["kind"] == "tl":
            dx = {n: _round(m.field("%s.d%s" % (k, n), "seed") * fields[n].double().std(), dt) for n in t["active"]}
        out[k] = (fields, scalars, seeds, dx)
    return out


def _chain_inputs(nx, ny, nz, halo, workload, dtype, seed, device):
    m = _Maker(nx, ny, nz, halo, workload, seed, device)
    fields = {n: _round(m.field("chain." + n, c), dtype) for n, c in _CHAIN3.items()}
    fields.update({n: _round(m.line("chain." + n), dtype) for n in _CHAIN1})
    scalars = {n: m.scalar("chain." + n) for n in ("edadlat", "dt", "eddlat", "eddlon", "tau_smag", "weight_smag")}
    # the advective tendencies move u by a few per cent
    scalars.update({"dt_adv": 0.01, "ppm_p1": _PPM["p1"], "ppm_p2": _PPM["p2"]})
    seeds = {n: _round(m.field("chain.%sb" % n, "seed"), dtype) for n in _CHAIN_OUT}
    return fields, scalars, seeds


def _chain_members(case, seed, device):
    """One (domain, fields, scalars, seeds) for a chain case, one a member for a batch case."""
    halo = max(case["halo"], _CHAIN_HALO)
    members = _members(case) if case["kind"] == "batch" else [(case["nx"], case["ny"], case["nz"], case["dtype"])]
    return [((nx, ny, nz), halo, dt) + _chain_inputs(nx, ny, nz, halo, case["workload"], dt, seed + 17 * q, device)
            for q, (nx, ny, nz, dt) in enumerate(members)]


# ---------------------------------------------------------------------------------------
# a pass
# ---------------------------------------------------------------------------------------
def prepare(case, seed):
    pkg = load_package()
    device = torch.device("cuda")
    kind = case["kind"]
    if kind in ("chain", "batch"):
        ch = pkg.chain
        members = []
        for dom, halo, dt, fields, scalars, seeds in _chain_members(case, seed, device):
            wrap = lambda x, halo=halo: pkg.Storage(x, halo)  # noqa: E731
            blank = lambda like: wrap(torch.zeros_like(like))  # noqa: E731
            members.append({"domain": dom, "scalars": scalars, "fields": {n: wrap(x) for n, x in fields.items()},
                            "outs": {n: blank(fields["u"]) for n in _CHAIN_OUT},
                            "seeds": {n: wrap(x) for n, x in seeds.items()},
                            "grads": {n: blank(fields["u"]) for n in ("u", "v")}})
        modes = ch.FORWARD | ch.ADJOINT
        if kind == "chain":
            plan = ch.ChainPlan(members[0]["fields"]["u"], members[0]["domain"], modes)
        else:
            plan = ch.BatchPlan(members, modes)
        return {"kind": kind, "plan": plan, "members": members}
    calls = []
    for k, (fields, scalars, seeds, dx) in _stencil_inputs(case, seed, device).items():
        t = _TABLE[k]
        st = {n: pkg.Storage(x, case["halo"]) for n, x in fields.items()}
        like = fields[next(iter(t["in3"]))]
        names = t["active"] if kind == "adjoint" else t["out"]
        out = {n: pkg.Storage(torch.zeros_like(like), case["halo"]) for n in names}
        if kind == "call":
            st.update(out)
        calls.append((k, st, {n: pkg.Storage(x, case["halo"]) for n, x in (seeds or dx).items()}, out, scalars))
    return {"kind": kind, "pkg": pkg, "calls": calls, "domain": (case["nx"], case["ny"], case["nz"])}


def run(state):
    kind = state["kind"]
    if kind == "chain":
        m = state["members"][0]
        state["plan"].forward(m["fields"], m["scalars"], m["outs"])
        state["plan"].adjoint(m["fields"], m["scalars"], m["seeds"], m["grads"])
    elif kind == "batch":
        state["plan"].run()
    if kind in ("chain", "batch"):
        return [{n: s.data for n, s in {**m["outs"], "ub": m["grads"]["u"], "vb": m["grads"]["v"]}.items()}
                for m in state["members"]]
    pkg, domain = state["pkg"], state["domain"]
    outputs = {}
    for k, fields, more, out, scalars in state["calls"]:
        if kind == "call":
            pkg.call(k, fields, scalars, domain=domain)
        elif kind == "adjoint":
            pkg.adjoint(k, fields, more, out, scalars, domain=domain)
        else:
            pkg.tangent_linear(k, fields, more, out, scalars, domain=domain)
        outputs[k] = {n: s.data for n, s in out.items()}
    return outputs


# ---------------------------------------------------------------------------------------
# the same in 64 bits, by plain torch
# ---------------------------------------------------------------------------------------
class _Dom:
    """Boxes of a domain (interior n widened by e in i and j) in allocations with halo h.  A box is
    (ilo, ihi, jlo, jhi, klo, khi), the cells beyond the widened interior on each side."""

    def __init__(self, nx, ny, nz, h, e=0):
        self.n, self.h, self.e = (nz, ny, nx), h, e

    def _range(self, axis, lo, hi, d):
        e = 0 if axis == 0 else self.e
        return slice(self.h - e - lo + d, self.h + self.n[axis] + e + hi + d)

    def at(self, f, box=(0, 0, 0, 0, 0, 0), i=0, j=0, k=0):
        ilo, ihi, jlo, jhi, klo, khi = box
        if f.dim() == 1:
            return f[self._range(1, jlo, jhi, j)][None, :, None]
        return f[self._range(0, klo, khi, k), self._range(1, jlo, jhi, j), self._range(2, ilo, ihi, i)]

    def put(self, v, box=(0, 0, 0, 0, 0, 0)):
        """A whole allocation, zero outside the box."""
        ilo, ihi, jlo, jhi, klo, khi = box
        h, e = self.h, self.e
        return F.pad(v, (h - e - ilo, h - e - ihi, h - e - jlo, h - e - jhi, h - klo, h - khi))


_RADIUS = 6371.229e3
_I = (0, 0, 0, 0, 0, 0)


def _x_laplace(d, x, s):
    a = lambda i=0, j=0: d.at(x["in"], _I, i, j)  # noqa: E731
    return {"out": d.put(-4.0 * a() + ((a(-1) + a(1)) + (a(0, 1) + a(0, -1))))}


def _x_hdiffsa(d, x, s):
    f = x["in"]
    b = (1, 1, 1, 1, 0, 0)
    c = d.at(f, b)
    lap = d.put(d.at(f, b, -1) + d.at(f, b, 1) - 2.0 * c + d.at(x["crlato"], b) * (d.at(f, b, 0, 1) - c)
                + d.at(x["crlatu"], b) * (d.at(f, b, 0, -1) - c), b)
    bx, by = (1, 0, 0, 0, 0, 0), (0, 0, 1, 0, 0, 0)
    flx = d.at(lap, bx, 1) - d.at(lap, bx)
    flx = d.put(torch.where(flx * (d.at(f, bx, 1) - d.at(f, bx)) > 0, torch.zeros_like(flx), flx), bx)
    fly = d.at(x["crlato"], by) * (d.at(lap, by, 0, 1) - d.at(lap, by))
    fly = d.put(torch.where(fly * (d.at(f, by, 0, 1) - d.at(f, by)) > 0, torch.zeros_like(fly), fly), by)
    div = d.at(flx, _I, -1) - d.at(flx) + d.at(fly, _I, 0, -1) - d.at(fly)
    return {"out": d.put(d.at(f) + div * d.at(x["mask"]))}


def _x_hdiffsmag(d, x, s):
    u, v = x["uin"], x["vin"]
    c1, el = s["eddlat"] / _RADIUS, s["eddlon"]
    bt, bs = (0, 1, 0, 1, 0, 0), (1, 0, 1, 0, 0, 0)
    t = (d.at(v, bt, 0, -1) - d.at(v, bt)) * c1 - (d.at(u, bt, -1) - d.at(u, bt)) * d.at(x["acrlat0"], bt) * el
    q = (d.at(u, bs, 0, 1) - d.at(u, bs)) * c1 + (d.at(v, bs, 1) - d.at(v, bs)) * d.at(x["acrlat0"], bs) * el
    t2, s2 = d.put(t * t, bt), d.put(q * q, bs)
    hd = s["weight_smag"] * d.at(x["mask"])

    def clamp(a):
        a = torch.where(a > 0, a, torch.zeros_like(a))
        return torch.where(a < 0.5, a, torch.full_like(a, 0.5))

    su = clamp(s["tau_smag"] * torch.sqrt(0.5 * (d.at(t2, _I, 1) + d.at(t2)) + 0.5 * (d.at(s2, _I, 0, -1) + d.at(s2))) - hd)
    sv = clamp(s["tau_smag"] * torch.sqrt(0.5 * (d.at(t2, _I, 0, 1) + d.at(t2)) + 0.5 * (d.at(s2, _I, -1) + d.at(s2))) - hd)
    out = {}
    for name, f, sm, co, cu in (("uout", u, su, "crlato", "crlatu"), ("vout", v, sv, "crlavo", "crlavu")):
        c = d.at(f)
        lap = d.at(f, _I, 1) + d.at(f, _I, -1) - 2.0 * c + d.at(x[co]) * (d.at(f, _I, 0, 1) - c) \
            + d.at(x[cu]) * (d.at(f, _I, 0, -1) - c)
        out[name] = d.put(c + sm * lap)
    return out


_UPWIND = {  # offsets and weights for a positive and for any other wind
    3: (((-2, -1 / 6), (-1, 1.0), (0, -0.5), (1, -1 / 3)), ((-1, -1 / 3), (0, -0.5), (1, 1.0), (2, -1 / 6))),
    5: (((-3, 1 / 30), (-2, -0.25), (-1, 1.0), (0, -1 / 3), (1, -0.5), (2, 0.05)),
        ((-2, 0.05), (-1, -0.5), (0, -1 / 3), (1, 1.0), (2, -0.25), (3, 1 / 30))),
}


def _advect(d, f, a, order, along_i):
    def side(terms):
        return sum(w * (d.at(f, _I, o, 0) if along_i else d.at(f, _I, 0, o)) for o, w in terms)

    pos, neg = _UPWIND[order]
    return torch.where(a > 0, a * side(pos), -a * side(neg))


def _x_hadv(order):
    def fn(d, x, s):
        u, v = x["uin"], x["vin"]
        uu = (d.at(u, _I, -1) + d.at(u) + d.at(u, _I, 1)) / 3.0
        vu = 0.25 * (d.at(v, _I, 1) + d.at(v, _I, 1, -1) + d.at(v) + d.at(v, _I, 0, -1))
        uv = 0.25 * (d.at(u, _I, -1) + d.at(u) + d.at(u, _I, 0, 1) + d.at(u, _I, -1, 1))
        vv = (d.at(v, _I, 0, -1) + d.at(v) + d.at(v, _I, 0, 1)) / 3.0
        ru = s["eddlat"] * _advect(d, u, d.at(x["acrlat0"]) * uu, order, True) \
            + s["eddlon"] * _advect(d, u, vu / _RADIUS, order, False)
        rv = s["eddlat"] * _advect(d, v, d.at(x["acrlat1"]) * uv, order, True) \
            + s["eddlon"] * _advect(d, v, vv / _RADIUS, order, False)
        return {"uout": d.put(ru + d.at(x["tgrlatda0"]) * d.at(u) * vu),
                "vout": d.put(rv - d.at(x["tgrlatda1"]) * uv * uv)}
    return fn


def _x_fastwavesuv(d, x, s):
    b, bk = (0, 1, 0, 1, 0, 0), (0, 1, 0, 1, 0, 1)
    w, p, hh, r = x["wgtfac"], x["ppuv"], x["hhl"], x["rho"]
    ppgk = d.put(d.at(w, bk) * d.at(p, bk) + (1.0 - d.at(w, bk)) * d.at(p, bk, k=-1), bk)
    c = d.put(d.at(ppgk, b, k=1) - d.at(ppgk, b), b)
    hs = d.put(d.at(hh, b, k=1) + d.at(hh, b), b)
    hd = d.put(d.at(hh, b, k=1) - d.at(hh, b), b)
    out = {}
    for name, at, tens, i, j, num in (("uout", "uin", "utens", 1, 0, 2.0 * d.at(x["fx"])),
                                      ("vout", "vin", "vtens", 0, 1, 2.0 * s["edadlat"])):
        g = (d.at(p, _I, i, j) - d.at(p)) + (d.at(c, _I, i, j) + d.at(c)) * 0.5 * (d.at(hs) - d.at(hs, _I, i, j)) \
            / (d.at(hd) + d.at(hd, _I, i, j))
        out[name] = d.put(d.at(x[at]) + s["dt"] * (d.at(x[tens]) - g * (num / (d.at(r, _I, i, j) + d.at(r)))))
    return out


def _x_uvbke(d, x, s):
    su = d.at(x["uc"], _I, 0, -1) + d.at(x["uc"])
    sv = d.at(x["vc"], _I, -1) + d.at(x["vc"])
    ca, rs = d.at(x["cosa"]), d.at(x["rsina"])
    return {"ub": d.put(s["dt5"] * (su - sv * ca) * rs), "vb": d.put(s["dt5"] * (sv - su * ca) * rs)}


def _x_nh_p_grad(d, x, s):
    gz, out = x["gz"], {}
    for name, at, rd, i, j in (("uout", "uin", "rdx", 1, 0), ("vout", "vin", "rdy", 0, 1)):
        n = lambda f, k=0: d.at(f, _I, i, j, k)  # noqa: E731
        o = lambda f, k=0: d.at(f, _I, 0, 0, k)  # noqa: E731
        pair = lambda p: (o(gz, 1) - n(gz)) * (n(p, 1) - o(p)) + (o(gz) - n(gz, 1)) * (o(p, 1) - n(p))  # noqa: E731
        pk, w1 = x["pk3"], x["wk1"]
        du = s["dt"] / ((o(pk, 1) - o(pk)) + (n(pk, 1) - n(pk))) * pair(pk)
        out[name] = d.put((d.at(x[at]) + du + s["dt"] / (o(w1) + n(w1)) * pair(x["pp"])) * d.at(x[rd]))
    return out


def _x_p_grad_c(d, x, s):
    gz, pk, out = x["gz"], x["pkc"], {}
    for name, at, rd, i, j in (("uout", "uin", "rdxc", -1, 0), ("vout", "vin", "rdyc", 0, -1)):
        n = lambda f, k=0: d.at(f, _I, i, j, k)  # noqa: E731
        o = lambda f, k=0: d.at(f, _I, 0, 0, k)  # noqa: E731
        pair = (n(gz, 1) - o(gz)) * (o(pk, 1) - n(pk)) + (n(gz) - o(gz, 1)) * (n(pk, 1) - o(pk))
        out[name] = d.put(d.at(x[at]) + s["dt2"] * d.at(x[rd]) / (n(x["delpc"]) + o(x["delpc"])) * pair)
    return out


def _ppm(d, f, c, s, box, along_i):
    """Upwind PPM flux of f at the low faces of `box`, for Courant number c there."""
    def at(g, b, o):
        return d.at(g, b, o, 0) if along_i else d.at(g, b, 0, o)

    def wider(lo, hi):
        ilo, ihi, jlo, jhi, klo, khi = box
        return (ilo + lo, ihi + hi, jlo, jhi, klo, khi) if along_i else (ilo, ihi, jlo + lo, jhi + hi, klo, khi)

    b2, b1 = wider(1, 1), wider(1, 0)
    al = d.put(s["p1"] * (at(f, b2, -1) + at(f, b2, 0)) + s["p2"] * (at(f, b2, -2) + at(f, b2, 1)), b2)
    m, r = at(al, b1, 0) - at(f, b1, 0), at(al, b1, 1) - at(f, b1, 0)
    b0 = d.put(m + r, b1)
    flag = d.put((m * r < 0).to(m.dtype), b1)
    m, r = d.put(m, b1), d.put(r, b1)
    either = torch.maximum(at(flag, box, -1), at(flag, box, 0))
    cc = d.at(c, box)
    up = at(f, box, -1) + (1.0 - cc) * (at(r, box, -1) - cc * at(b0, box, -1)) * either
    dn = at(f, box, 0) + (1.0 + cc) * (at(m, box, 0) + cc * at(b0, box, 0)) * either
    return d.put(torch.where(cc > 0, up, dn), box)


def _x_fvtp2d(d, x, s):
    q = x["q"]
    by, bx = (3, 2, 0, 1, 0, 0), (0, 1, 3, 2, 0, 0)
    bi, bj = (3, 2, 0, 0, 0, 0), (0, 0, 3, 2, 0, 0)
    fy2, fx2 = _ppm(d, q, x["cry"], s, by, False), _ppm(d, q, x["crx"], s, bx, True)
    fyy, fxx = d.put(d.at(x["yfx"], by) * d.at(fy2, by), by), d.put(d.at(x["xfx"], bx) * d.at(fx2, bx), bx)
    q_i = d.put((d.at(q, bi) * d.at(x["area"], bi) + d.at(fyy, bi) - d.at(fyy, bi, 0, 1)) / d.at(x["ra_y"], bi), bi)
    q_j = d.put((d.at(q, bj) * d.at(x["area"], bj) + d.at(fxx, bj) - d.at(fxx, bj, 1)) / d.at(x["ra_x"], bj), bj)
    fx1, fy1 = _ppm(d, q_i, x["crx"], s, _I, True), _ppm(d, q_j, x["cry"], s, _I, False)
    return {"q_i": q_i, "q_j": q_j, "fx1": d.put(0.5 * (d.at(fx1) + d.at(fx2)) * d.at(x["xfx"])), "fx2": fx2,
            "fy1": d.put(0.5 * (d.at(fy1) + d.at(fy2)) * d.at(x["yfx"])), "fy2": fy2}


_EXACT = {"laplace": _x_laplace, "hdiffsa": _x_hdiffsa, "hdiffsmag": _x_hdiffsmag, "hadvuv": _x_hadv(3),
          "hadvuv5th": _x_hadv(5), "fastwavesuv": _x_fastwavesuv, "uvbke": _x_uvbke, "nh_p_grad": _x_nh_p_grad,
          "p_grad_c": _x_p_grad_c, "fvtp2d": _x_fvtp2d}


def _x_chain(dom, h, x, s):
    """The chained step: each stage on the interior widened by what the later ones read."""
    nx, ny, nz = dom
    d7, d4, d3, d0 = (_Dom(nx, ny, nz, h, e) for e in (7, 4, 3, 0))
    w = _x_fastwavesuv(d7, {"uin": x["u"], "vin": x["v"], **{n: x[n] for n in (
        "utens", "vtens", "wgtfac", "ppuv", "hhl", "rho", "fx")}}, s)
    t = _x_hadv(5)(d4, {"uin": w["uout"], "vin": w["vout"], **{n: x[n] for n in _ADV1}}, s)
    u2 = {n: d4.put(d4.at(w[o]) + s["dt_adv"] * d4.at(t[o])) for n, o in (("uin", "uout"), ("vin", "vout"))}
    g = _x_hdiffsmag(d3, {**u2, "mask": x["mask"], "acrlat0": x["smag_acrlat0"],
                          **{n: x[n] for n in ("crlavo", "crlavu", "crlato", "crlatu")}}, s)
    f = _x_fvtp2d(d0, {"q": g["uout"], **{n: x[n] for n in ("crx", "cry", "ra_x", "ra_y", "xfx", "yfx", "area")}},
                  {"p1": s["ppm_p1"], "p2": s["ppm_p2"]})
    return {"uout": g["uout"], "vout": g["vout"], "fx1": f["fx1"], "fy1": f["fy1"]}


def _vjp(fn, primals, names, seeds, dom):
    """Gradients of sum over the interior of seed * output with respect to `names`."""
    x = {n: (v.detach().requires_grad_(True) if n in names else v) for n, v in primals.items()}
    y = fn(x)
    total = sum((dom.at(y[n]) * dom.at(sd)).sum() for n, sd in seeds.items())
    return dict(zip(names, torch.autograd.grad(total, [x[n] for n in names])))


def _rounded_scalars(scalars, dtype):
    """The scalars as a call of the case's type receives them (uvbke's dt5 is a double in both)."""
    return {n: v if dtype == "f64" or n == "dt5" else float(np.float32(v)) for n, v in scalars.items()}


def exact(case, seed):
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    kind = case["kind"]
    if kind in ("chain", "batch"):
        res = []
        for dom, h, dt, fields, scalars, seeds in _chain_members(case, seed, device):
            x, sd = ({n: v.double() for n, v in f.items()} for f in (fields, seeds))
            s = _rounded_scalars(scalars, dt)
            out = _x_chain(dom, h, x, s)
            grads = _vjp(lambda a, dom=dom, h=h, s=s: _x_chain(dom, h, a, s), x, ("u", "v"), sd, _Dom(*dom, h))
            res.append({**out, "ub": grads["u"], "vb": grads["v"]})
        return res
    d = _Dom(case["nx"], case["ny"], case["nz"], case["halo"])
    res = {}
    for k, (fields, scalars, seeds, dx) in _stencil_inputs(case, seed, device).items():
        x = {n: v.double() for n, v in fields.items()}
        s = _rounded_scalars(scalars, case["dtype"])
        fn = lambda a, k=k, s=s: _EXACT[k](d, a, s)  # noqa: E731
        if kind == "call":
            res[k] = fn(x)
        elif kind == "adjoint":
            res[k] = _vjp(fn, x, _TABLE[k]["active"], {n: v.double() for n, v in seeds.items()}, d)
        else:
            names = _TABLE[k]["active"]
            _, dy = torch.func.jvp(lambda *a, x=x, fn=fn, names=names: fn({**x, **dict(zip(names, a))}),
                                   tuple(x[n] for n in names), tuple(dx[n].double() for n in names))
            res[k] = dy
    return res
