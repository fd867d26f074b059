"""Timed cases of the microphysics framework: the calls a host model makes.

A host model calls the step once per physics time step on all columns of a
GPU, with the radiation-facing optics, droplet mixing and activation on the
same columns, and the adjoint in data assimilation and sensitivity runs.
Sizes are columns x levels (cells = columns * levels); the distributions of
the inputs are those of mam4xx_b200/workloads.py (configurations c1, c2 and
c4), drawn on the GPU.

Every case is one dict:
  kind    the entry point (see ENTRIES below)
  ncol, nlev
  sky     "clear" (no cloud, no cloud-borne aerosol), "uniform" (cloud
          fraction U(0, 1), mode numbers log-uniform 1e5..1e10: 1..1000 SOA
          sub-steps per cell) or "uneven" (60 % of the cells clear, the rest
          U(0.2, 1); numbers 1e5..1e6: 1..20 sub-steps)

prepare() builds the state a host keeps between calls (context, fields,
tables), run() is one call, exact() restates in plain torch (64 bits) what
has a value that does not hang on the last bit of a branch: the size and
water outputs of the step, the activation fractions and the optics. The
tendencies have none: the SOA sub-step control and the clips of the
algorithm branch on rounding, so that a second 64-bit evaluation takes other
branches in some cells.
"""

import math

import numpy as np
import torch

from mam4xx_b200 import native, process
from mam4xx_b200 import workloads as wl

DT = 1800.0
F64 = torch.float64

# entry: (doubles read and written per cell, flops per cell; a libm call is
# counted as 20). The step's counts are those of the operation-counting
# build of its CPU restatement; the others are counted from the formulas.
ENTRIES = {
    "process": (57 + 68, 11000),          # MicrophysicsProcess.compute_tendencies
    "process_diag": (57 + 68 + 155, 12000),  # with the 155 process tendencies
    "slab": (57 + 68, 11000),             # Context.step_slab as one CUDA graph
    "tracers": (57 + 68, 20000),          # Context.step_tracers
    "mixed": (57 + 68, 20000),            # Context.step_slab, MIXED
    "host": (57 + 68, 11000),             # Context.step_host
    "adjoint": (57 + 68 + 57, 50000),     # Context.adjoint_slab
    "chem": (57 + 68 + 55 + 4, 20000),    # Context.step_chem_slab
    "rad_sw": (57 + 3 + 3 * 14 + 4 * 14, 14000),  # Context.aero_rad_props_sw
    "rad_lw": (57 + 3 + 16 + 16, 9000),   # Context.aero_rad_props_lw
    "dropmix": (57 + 6 + 66, 4000),       # Context.dropmixnuc
    "activate": (26 + 2 + 17, 1500),      # Context.activate
}


def listed():
    return [
        # a single rank's few columns (regional or unit run): launches and
        # latency, through the AeroProcess mirror
        {"name": "process_small", "kind": "process", "ncol": 8, "nlev": 72, "sky": "clear"},
        # the headline: a full GPU's columns, uneven sub-stepping
        {"name": "step_large", "kind": "slab", "ncol": 65536, "nlev": 72, "sky": "uneven"},
        # the host's tracer arrays, odd column count, long sub-stepping
        {"name": "step_tracers", "kind": "tracers", "ncol": 4099, "nlev": 72, "sky": "uniform"},
        # the opt-in mixed-precision step
        {"name": "step_mixed", "kind": "mixed", "ncol": 8192, "nlev": 72, "sky": "uniform"},
        # state in host memory (a host model that runs on the CPU), pinned
        {"name": "step_host", "kind": "host", "ncol": 8192, "nlev": 72, "sky": "uneven"},
        # budget diagnostics: every process's tendencies written
        {"name": "step_budgets", "kind": "process_diag", "ncol": 1024, "nlev": 72,
         "sky": "uneven"},
        # gradient of the step (data assimilation, sensitivity)
        {"name": "adjoint", "kind": "adjoint", "ncol": 4096, "nlev": 72, "sky": "uniform"},
        # gas-phase and aqueous chemistry fused ahead of the microphysics
        {"name": "step_chem", "kind": "chem", "ncol": 8192, "nlev": 72, "sky": "uneven"},
        # radiation time step: shortwave and longwave aerosol optics
        {"name": "rad_sw", "kind": "rad_sw", "ncol": 16384, "nlev": 72, "sky": "uniform"},
        {"name": "rad_lw", "kind": "rad_lw", "ncol": 16384, "nlev": 72, "sky": "uniform"},
        # droplet nucleation and vertical mixing per column
        {"name": "dropmix", "kind": "dropmix", "ncol": 16384, "nlev": 72, "sky": "uneven"},
        # activation fractions alone, on another vertical grid (80 levels)
        {"name": "activate", "kind": "activate", "ncol": 8191, "nlev": 80, "sky": "uniform"},
    ]


def draw(rng):
    base = rng.choice(listed())
    top = base["ncol"] * 72
    nlev = rng.randrange(20, 129)
    cells = math.exp(rng.uniform(math.log(32 * 20), math.log(top)))
    ncol = max(1, min(int(cells / nlev), top // nlev))
    kind = base["kind"]
    sky = base["sky"]
    if kind in ("process", "process_diag", "slab", "chem", "dropmix"):
        sky = rng.choice(["clear", "uneven"])
    elif kind in ("tracers", "mixed", "activate", "rad_sw", "rad_lw"):
        sky = rng.choice(["uniform", "uneven"])
    return {"kind": kind, "ncol": ncol, "nlev": nlev, "sky": sky}


def work(case):
    n = case["ncol"] * case["nlev"]
    doubles, flops = ENTRIES[case["kind"]]
    return {"bytes": 8.0 * doubles * n + 8.0 * case["ncol"], "flops": float(flops) * n}


# ------------------------------------------------------------------ inputs
class _Draw:
    def __init__(self, seed, n):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)
        self.n = n

    def u(self, lo, hi, *shape):
        r = torch.rand(shape or (self.n,), generator=self.g, dtype=F64, device="cuda")
        return r.mul_(hi - lo).add_(lo)

    def logu(self, lo, hi, *shape):
        return self.u(math.log(lo), math.log(hi), *shape).exp_()

    def normal(self, *shape):
        return torch.randn(shape, generator=self.g, dtype=F64, device="cuda")


def _magnus_qv_sat(temp, pmid):
    eps = 0.018016 / 0.028966
    tc = temp - 273.15
    es = 1.00071 * torch.exp(4.5e-8 * pmid) * 610.94 * torch.exp(17.625 * tc / (234.04 + tc))
    return eps * es / (pmid - (1.0 - eps) * es)


def _fields(d, ncol, nlev, sky):
    """The 57 input fields (workloads.make_workload, on the GPU)."""
    n = ncol * nlev
    x = torch.zeros((wl.NIN, n), dtype=F64, device="cuda")
    plev = torch.tensor(np.geomspace(1000.0, 100000.0, nlev), device="cuda")
    temp = d.u(200.0, 310.0)
    x[wl.IN_T] = temp
    x[wl.IN_P] = plev.repeat(ncol)
    x[wl.IN_ZM] = _heights(temp.view(ncol, nlev), plev).reshape(-1)
    x[wl.IN_QV] = d.u(0.05, 0.99) * _magnus_qv_sat(temp, x[wl.IN_P])
    if sky == "uniform":
        x[wl.IN_CLD] = d.u(0.0, 1.0)
    elif sky == "uneven":
        x[wl.IN_CLD] = torch.where(d.u(0.0, 1.0) < 0.6, 0.0, d.u(0.2, 1.0))
    h2so4 = (1e-15, 1e-8) if sky == "uneven" else (1e-14, 1e-10)
    number = (1e5, 1e6) if sky == "uneven" else (1e5, 1e10)
    x[wl.IN_H2SO4] = d.logu(*h2so4) * (wl.ADV_MASS[2] / wl.MW_DRY_AIR)
    x[wl.IN_SOAG] = d.logu(1e-12, 1e-9) * (wl.ADV_MASS[5] / wl.MW_DRY_AIR)
    for base in (wl.IN_AER_I, wl.IN_AER_C):
        if base == wl.IN_AER_C and sky == "clear":
            break
        for slot, (_, species) in enumerate(wl.POPULATIONS):
            x[base + slot] = d.logu(*number) if species == "num" else d.logu(1e-14, 1e-8)
    return x


def _heights(t, plev):
    """Hypsometric mid-level heights of temperatures t (ncol, nlev)."""
    c = 287.04 / 9.80616
    low = c * t[:, -1:] * math.log(101325.0 / float(plev[-1]))
    dz = c * 0.5 * (t[:, :-1] + t[:, 1:]) * torch.log(plev[1:] / plev[:-1])
    up = torch.flip(torch.cumsum(torch.flip(dz, (1,)), 1), (1,))
    return torch.cat((low + up, low), 1)


def _atmosphere(d, x, ncol, nlev):
    """A column atmosphere with a tropopause (workloads.make_rad_props_inputs):
    replaces T, z and qv in x, returns interface pressures and heights and
    the layer thicknesses in pressure."""
    plev = x[wl.IN_P][:nlev].clone()
    pint = torch.empty(nlev + 1, dtype=F64, device="cuda")
    pint[1:nlev] = torch.sqrt(plev[:-1] * plev[1:])
    pint[0] = plev[0] * torch.sqrt(plev[0] / plev[1])
    pint[nlev] = 101325.0
    z = 7500.0 * torch.log(101325.0 / plev)[None, :]
    t0, zt = d.u(280.0, 305.0, ncol, 1), d.u(9000.0, 17000.0, ncol, 1)
    none = d.u(0.0, 1.0, ncol, 1) < 0.1  # columns without a tropopause
    temp = torch.where(z <= zt, t0 - 6.5e-3 * z, t0 - 6.5e-3 * zt + 1.5e-3 * (z - zt))
    z60 = 7500.0 * math.log(101325.0 / 6000.0)
    temp = torch.where(none, t0 - 8.0e-3 * z.clamp(max=z60), temp)
    temp = temp + 0.2 * d.normal(ncol, nlev)
    dz = (287.04 / 9.80616) * temp * torch.log(pint[1:] / pint[:-1])
    zi = torch.zeros((ncol, nlev + 1), dtype=F64, device="cuda")
    zi[:, :-1] = torch.flip(torch.cumsum(torch.flip(dz, (1,)), 1), (1,))
    x[wl.IN_T] = temp.reshape(-1)
    x[wl.IN_ZM] = (0.5 * (zi[:, :-1] + zi[:, 1:])).reshape(-1)
    x[wl.IN_QV] = d.u(0.05, 0.99) * _magnus_qv_sat(x[wl.IN_T], x[wl.IN_P]).clamp(min=0.0)
    return {"pint": pint.repeat(ncol), "zi": zi.reshape(-1),
            "pdel": (pint[1:] - pint[:-1]).repeat(ncol)}


def _chem_inputs(d, x):
    """The chemistry slab (workloads.make_chem_step_inputs, on the GPU)."""
    n = x.shape[1]
    ch = torch.zeros((wl.CHEM_NIN, n), dtype=F64, device="cuda")
    ranges = ((1e-8, 1e-6), (1e-12, 1e-9), (1e-12, 1e-8), (1e-12, 1e-9))  # O3 H2O2 SO2 DMS
    for k, (i31, r) in enumerate(zip((0, 1, 3, 4), ranges)):
        ch[k] = d.logu(*r) * (wl.ADV_MASS[i31] / wl.MW_DRY_AIR)
    ch[wl.CHEM_IN_PHOTO] = torch.where(d.u(0, 1) < 0.3, 0.0, d.logu(1e-7, 1e-5))
    for k in range(9):
        ch[wl.CHEM_IN_EXTFRC + k] = torch.where(d.u(0, 1) < 0.5, 0.0, d.logu(1e-3, 1e2))
    m = 10.0 * x[wl.IN_P] / (0.13806500000000001e-15 * x[wl.IN_T])
    inv = wl.CHEM_IN_INV
    ch[inv], ch[inv + 1], ch[inv + 2] = m, 0.79 * m, 0.21 * m
    ch[inv + 3] = x[wl.IN_QV].clamp(min=0.0) * (wl.MW_DRY_AIR / 18.015) * m
    for k, r in enumerate(((1e-15, 1e-12), (1e-14, 1e-10), (1e-13, 1e-10), (1e-8, 1e-6))):
        ch[inv + 4 + k] = d.logu(*r) * m
    for k in range(31):
        ch[wl.CHEM_IN_HET + k] = torch.where(d.u(0, 1) < 0.5, 0.0, d.logu(1e-8, 1e-3))
    wet = (x[wl.IN_CLD] > 0) & (d.u(0, 1) < 0.8)
    ch[wl.CHEM_IN_LWC] = torch.where(wet, d.logu(1e-6, 1e-3), 0.0)
    ch[wl.CHEM_IN_CLDNUM] = d.logu(1e7, 1e9)
    return ch


def _out(rows, n):
    return torch.empty((rows, n), dtype=F64, device="cuda")


def prepare(case, seed):
    kind, ncol, nlev = case["kind"], case["ncol"], case["nlev"]
    n = ncol * nlev
    d = _Draw(seed, n)
    x = _fields(d, ncol, nlev, case["sky"])
    s = {"kind": kind, "ncol": ncol, "nlev": nlev, "n": n, "x": x}
    s["pblh"] = torch.full((ncol,), 1000.0, dtype=F64, device="cuda")
    if kind in ("process", "process_diag"):
        s["proc"] = process.MicrophysicsProcess()
        s["out"] = _out(wl.NOUT, n)
        s["diag"] = _out(wl.NDIAG, n) if kind == "process_diag" else None
        s["atm"], s["prog"] = process.state_from_slab(x, s["pblh"], ncol, nlev)
        s["tend"], s["diags"] = process.outputs_from_slab(s["out"], ncol, nlev, s["diag"])
        return s
    ctx = s["ctx"] = native.Context()
    if kind in ("slab", "mixed"):
        s["out"] = _out(wl.NOUT, n)
        ctx.set_graph_mode(True)
    elif kind == "tracers":
        # E3SM state_q order: qv 0, H2SO4 11, SOAG 14, populations 15..39
        q = torch.zeros((40, n), dtype=F64, device="cuda")
        q[0], q[11], q[14] = x[wl.IN_QV], x[wl.IN_H2SO4], x[wl.IN_SOAG]
        q[15:40] = x[wl.IN_AER_I:wl.IN_AER_I + 25]
        qc = torch.zeros_like(q)
        qc[15:40] = x[wl.IN_AER_C:wl.IN_AER_C + 25]
        s["q"], s["qc"] = q, qc
        s["x"] = x[:wl.IN_AER_I].clone()  # T, p, z, cloud fraction
        s["tq"], s["tqc"] = torch.zeros_like(q), torch.zeros_like(q)
        s["modes"] = _out(16, n)
    elif kind == "host":
        pin = lambda t: t.cpu().pin_memory()  # noqa: E731
        s["x"], s["pblh"] = pin(x), pin(s["pblh"])
        s["out"] = torch.zeros((wl.NOUT, n), dtype=F64).pin_memory()
    elif kind == "adjoint":
        # cotangents of every output, in units of its typical size
        scale = torch.ones((wl.NOUT, 1), dtype=F64, device="cuda")
        for slot in wl.NUMBER_SLOTS:
            scale[2 + slot] = scale[27 + slot] = 1e-15
        scale[wl.OUT_DGN_A:wl.OUT_WETDENS] = 1e-3
        scale[wl.OUT_WETDENS:wl.OUT_QAERWAT] = 1e-12
        s["ybar"] = torch.randn((wl.NOUT, n), generator=d.g, dtype=F64, device="cuda") * scale
        s["xbar"] = _out(wl.NIN, n)
    elif kind == "chem":
        s["chem"], s["out"], s["chem_out"] = _chem_inputs(d, x), _out(wl.NOUT, n), _out(4, n)
    elif kind in ("rad_sw", "rad_lw"):
        s.update(_atmosphere(d, x, ncol, nlev))
        s["trop"] = torch.zeros(ncol, dtype=torch.int32, device="cuda")
        if kind == "rad_sw":
            ctx.optics_sw_set_tables(wl.make_optics_sw_tables())
            s["ext"], s["ssa"] = d.logu(1e-8, 1e-5, 14, n), d.u(0.9, 1.0, 14, n)
            s["af"] = d.u(0.6, 0.8, 14, n)
            s["out"] = _out(4 * 14, n)
            s["aod"] = torch.empty(ncol, dtype=F64, device="cuda")
        else:
            ctx.optics_lw_set_tables(wl.make_optics_lw_tables())
            s["ext"] = d.logu(1e-9, 1e-6, 16, n)
            s["out"] = _out(16, n)
    elif kind == "dropmix":
        s.update(_atmosphere(d, x, ncol, nlev))
        cldn = x[wl.IN_CLD]
        old = (cldn + d.u(-0.3, 0.3)).clamp(0.0, 1.0)
        old = torch.where(d.u(0, 1) < 0.7, old, cldn)
        drops = torch.where(old > 0, d.logu(1e6, 1e9), 0.0)
        s["mix"] = torch.stack((s["pdel"], old, drops, d.u(0.02, 2.0)))
        s["kvh"] = d.logu(1e-3, 200.0, ncol * (nlev + 1))
        s["out"] = _out(wl.DROPMIX_NOUT, n)
    elif kind == "activate":
        s["rho"] = x[wl.IN_P] / (6.022214076e23 * 1.380649e-23 / 0.028966 * x[wl.IN_T])
        w, cut = d.logu(0.01, 3.0), d.u(0, 1)
        s["w"] = torch.where(cut < 0.05, 0.0, torch.where(cut < 0.1, -w, w))
        s["out"] = _out(17, n)
    return s


# ------------------------------------------------------------------ outputs
def _populations(name, rows):
    """25 population rows as each mode's masses and its number."""
    out = {}
    for m in range(4):
        slots = wl.MODE_SPECIES_SLOTS[m]
        out["%s_mass%d" % (name, m)] = rows[slots[0]:slots[-1] + 1]
        out["%s_num%d" % (name, m)] = rows[wl.NUMBER_SLOTS[m]]
    return out


def _modes(rows):
    return {"dgn_a": rows[0:4], "dgn_awet": rows[4:8], "wetdens": rows[8:12],
            "qaerwat": rows[12:16]}


def _step_out(out):
    return {"h2so4": out[0], "soag": out[1], **_populations("i", out[2:27]),
            **_populations("c", out[27:52]), **_modes(out[52:68])}


def run(s):
    kind, ncol, nlev, n = s["kind"], s["ncol"], s["nlev"], s["n"]
    x, ctx = s["x"], s.get("ctx")
    stream = torch.cuda.current_stream().cuda_stream
    p = lambda k: s[k].data_ptr()  # noqa: E731
    if kind in ("process", "process_diag"):
        s["proc"].compute_tendencies(0.0, DT, s["atm"], None, s["prog"], s["diags"], s["tend"])
        out = _step_out(s["out"])
        if s["diag"] is not None:
            for k, name in enumerate(process.Diagnostics.PROCESSES):
                out[name] = s["diag"][31 * k:31 * k + 31]
        return out
    if kind in ("slab", "mixed"):
        ctx.step_slab(x.data_ptr(), p("pblh"), p("out"), n, ncol, nlev, DT,
                      precision=native.MIXED if kind == "mixed" else native.FP64, stream=stream)
        return _step_out(s["out"])
    if kind == "tracers":
        ctx.step_tracers(p("q"), p("qc"), n, x[0].data_ptr(), x[1].data_ptr(), x[2].data_ptr(),
                         x[4].data_ptr(), p("pblh"), p("tq"), p("tqc"), p("modes"), n, ncol,
                         nlev, DT, stream=stream)
        return {"h2so4": s["tq"][11], "soag": s["tq"][14], **_populations("i", s["tq"][15:40]),
                **_populations("c", s["tqc"][15:40]), **_modes(s["modes"])}
    if kind == "host":
        ctx.step_host(x.data_ptr(), p("pblh"), p("out"), n, ncol, nlev, DT, stream=stream)
        return _step_out(s["out"])
    if kind == "adjoint":
        ctx.adjoint_slab(x.data_ptr(), p("pblh"), p("ybar"), p("xbar"), n, ncol, nlev, DT,
                         stream=stream)
        g = s["xbar"]
        return {"T": g[wl.IN_T], "fixed": g[1:3], "qv": g[wl.IN_QV], "cld": g[wl.IN_CLD],
                "h2so4": g[wl.IN_H2SO4], "soag": g[wl.IN_SOAG],
                **_populations("i", g[wl.IN_AER_I:wl.IN_AER_C]),
                **_populations("c", g[wl.IN_AER_C:])}
    if kind == "chem":
        ctx.step_chem_slab(x.data_ptr(), p("pblh"), p("chem"), p("out"), p("chem_out"), n, ncol,
                           nlev, DT, stream=stream)
        co = s["chem_out"]
        return {**_step_out(s["out"]), "o3": co[0], "h2o2": co[1], "so2": co[2], "dms": co[3]}
    if kind == "rad_sw":
        ctx.aero_rad_props_sw(x.data_ptr(), n, p("pdel"), p("pint"), p("zi"), p("ext"), p("ssa"),
                              p("af"), p("out"), p("aod"), p("trop"), ncol, nlev, DT,
                              stream=stream)
        o = s["out"]
        return {"tau": o[0:14], "wa": o[14:28], "ga": o[28:42], "fa": o[42:56], "aod": s["aod"],
                "trop": s["trop"]}
    if kind == "rad_lw":
        ctx.aero_rad_props_lw(x.data_ptr(), n, p("pdel"), p("pint"), p("zi"), p("ext"), p("out"),
                              p("trop"), ncol, nlev, DT, stream=stream)
        return {"tau": s["out"], "trop": s["trop"]}
    if kind == "dropmix":
        ctx.dropmixnuc(x.data_ptr(), n, p("mix"), p("pint"), p("kvh"), p("out"), ncol, nlev,
                       min(6, nlev - 2), DT, stream=stream)
        o = s["out"]
        return {"qcld": o[0], "tendnd": o[1], "nsource": o[2], "ndropmix": o[3],
                "ndropcol": o[4], "wtke": o[5], "factnum": o[6:10], "ccn": o[10:16],
                **_populations("ptend", o[16:41]), **_populations("qqcw", o[41:66])}
    ctx.activate(x.data_ptr(), n, p("rho"), p("w"), p("out"), ncol, nlev, stream=stream)
    o = s["out"]
    return {"fn": o[0:4], "fm": o[4:8], "fluxn": o[8:12], "fluxm": o[12:16], "full": o[16]}


# ------------------------------------------------------ 64-bit restatement
SIG = (1.8, 1.6, 1.8, 1.60000002384186)
DNOM = (1.1e-7, 2.6e-8, 2e-6, 5e-8)
DMIN = (5.35e-8, 8.7e-9, 1e-6, 1e-8)
DMAX = (4.4e-7, 5.2e-8, 4e-6, 1e-7)
DENS = {"SOA": 1000.0, "SO4": 1770.0, "POM": 1000.0, "BC": 1700.0, "NaCl": 1900.0,
        "DST": 2600.0, "MOM": 1601.0}
HYGRO = {"SO4": 0.507, "POM": 1.000000083e-10, "SOA": 0.14, "BC": 1.000000013e-10,
         "DST": 0.068, "NaCl": 1.16, "MOM": 0.1000000015}
TYPES = {"SO4": 0, "POM": 3, "SOA": 4, "BC": 5, "NaCl": 6, "DST": 7, "MOM": 8}


def _v2n(d, m):
    return 1.0 / (d ** 3 * math.exp(4.5 * math.log(SIG[m]) ** 2) * math.pi / 6)


def _volume(x, base, m, only=None):
    return sum(x[base + s].clamp(min=0.0) / DENS[wl.POPULATIONS[s][1]]
               for s in wl.MODE_SPECIES_SLOTS[m] if only is None or wl.POPULATIONS[s][1] in only)


def _diam(v, m):
    return (v * 6 / math.pi) ** (1.0 / 3.0) * math.exp(-1.5 * math.log(SIG[m]) ** 2)


def _clip(lo, v, hi):
    return torch.maximum(lo, torch.minimum(hi, v))


def _size(drv, num, v2nlo, v2nhi, m):
    d = _diam(drv / num, m)
    d = torch.where(num >= drv * v2nhi, DMIN[m], d)
    d = torch.where(num <= drv * v2nlo, DMAX[m], d)
    return torch.where(drv > 0, d, DNOM[m])


def _dry_sizes(x):
    """Dry diameters of the four interstitial modes (calcsize)."""
    adj = 1.0 / max(86400.0, DT)
    frac = min(1.0, DT * adj)
    vi = [_volume(x, wl.IN_AER_I, m) for m in range(4)]
    vc = [_volume(x, wl.IN_AER_C, m) for m in range(4)]
    ni = [x[wl.IN_AER_I + wl.NUMBER_SLOTS[m]].clamp(min=0.0) for m in range(4)]
    nc = [x[wl.IN_AER_C + wl.NUMBER_SLOTS[m]].clamp(min=0.0) for m in range(4)]
    lo = [_v2n(DMAX[m], m) for m in range(4)]
    hi = [_v2n(DMIN[m], m) for m in range(4)]
    dgn = [None] * 4
    for m in (2, 3):  # numbers pulled towards the size bounds
        a, b, l, h = vi[m], vc[m], lo[m], hi[m]
        di = (_clip(a * l / 27, ni[m], a * h * 27) - ni[m]) * frac
        dc = (_clip(b * l / 27, nc[m], b * h * 27) - nc[m]) * frac
        i2 = torch.where((di == 0) & (dc != 0), _clip(a * l / 27, ni[m] - dc, a * h * 27),
                         ni[m] + di)
        c2 = torch.where((di != 0) & (dc == 0), _clip(b * l / 27, nc[m] - di, b * h * 27),
                         nc[m] + dc)
        t, v = i2 + c2, a + b
        add = torch.zeros_like(t)
        for want, low in ((v * l, True), (v * h, False)):
            hit = (t < want) if low else (t > want)
            edge = l if low else h
            oi = (i2 < a * edge) if low else (i2 > a * edge)
            oc = (c2 < b * edge) if low else (c2 > b * edge)
            d3 = (want - t) * frac
            add = torch.where(hit & oi & oc, d3 * i2 / t, torch.where(hit & oi & ~oc, d3, add))
        both = i2 + add
        only_i = ni[m] + (_clip(a * l, ni[m], a * h) - ni[m]) * frac
        num = torch.where(b <= 0, only_i, both)
        num = torch.where(a <= 0, 0.0, num)
        dgn[m] = _size(a, num, l, h, m)
    for m in (0, 1):  # bounds widened towards each other
        dgn[m] = _size(vi[m], ni[m], lo[m] / (1e6 if m == 1 else 1), hi[m] * (1e6 if m == 0 else 1),
                       m)
    v2n_ait, v2n_acc = _v2n(DNOM[1], 1), _v2n(DNOM[0], 0)
    gm = math.sqrt(v2n_ait) * math.sqrt(v2n_acc)
    drv, num = vi[1] + vc[1], ni[1] + nc[1]
    up = (drv > 0) & (num < drv * gm)
    fv = (num / drv - gm) / (v2n_acc - gm)
    fn = fv * (drv * v2n_acc / num)
    fn, fv = _fractions(fn, fv, num < drv * v2n_acc)
    up_n, up_v = torch.where(up, fn * adj, 0.0), torch.where(up, fv * adj, 0.0)
    drv, num0 = vi[0] + vc[0], ni[0] + nc[0]
    num = num0
    big = (drv > 0) & (num > drv * gm)
    keep = ("POM", "BC", "DST")
    noxf_i = torch.where(big, _volume(x, wl.IN_AER_I, 0, keep), 0.0)
    noxf = noxf_i + torch.where(big, _volume(x, wl.IN_AER_C, 0, keep), 0.0)
    num = torch.where(big, (num - noxf * hi[0]).clamp(min=0.0), num)
    drv = torch.where(big, (drv - noxf).clamp(min=0.0), drv)
    down = (drv > 0) & (num > drv * gm)
    fv = (num / drv - gm) / (v2n_ait - gm)
    fn = fv * (drv * v2n_ait / num)
    fn, fv = _fractions(fn, fv, num > drv * v2n_ait)
    dn_n = torch.where(down, fn * num / num0 * adj, 0.0)
    dn_v = torch.where(down, fv * adj, 0.0)
    dn = (ni[1] * up_n - ni[0] * dn_n) * DT
    dv = (vi[1] * up_v - (vi[0] - noxf_i) * dn_v) * DT
    moved = up | down
    for m, sign in ((0, 1.0), (1, -1.0)):
        new = _size((vi[m] + sign * dv).clamp(min=0.0), (ni[m] + sign * dn).clamp(min=0.0), lo[m],
                    hi[m], m)
        dgn[m] = torch.where(moved, new, dgn[m])
    return dgn


def _fractions(fn, fv, full):
    zero, one = (fn <= 0) | (fv <= 0), full | (fn >= 1) | (fv >= 1)
    one = one & (full | ~zero)
    pick = lambda f: torch.where(one, 1.0, torch.where(zero, 0.0, f))  # noqa: E731
    return pick(fn), pick(fv)


def _svp_water(t):
    r = 373.16 / t
    return 100.0 * 10.0 ** (-7.90298 * (r - 1) + 5.02808 * torch.log10(r)
                            - 1.3816e-7 * (10.0 ** (11.344 * (1 - 1 / r)) - 1)
                            + 8.1328e-3 * (10.0 ** (-3.49149 * (r - 1)) - 1)
                            + math.log10(1013.246))


def _svp_ice(t):
    r = 273.16 / t
    return 100.0 * 10.0 ** (-9.09718 * (r - 1) - 3.56654 * torch.log10(r)
                            + 0.876793 * (1 - 1 / r) + math.log10(6.1071))


def _qsat(es, p):
    eps = 0.018016 / 0.028966
    return torch.where(p - es <= 0, 1.0, eps * es / (p - (1 - eps) * es))


def _kohler(rdry, hygro, rh):
    """Equilibrium radius [m] at relative humidity rh (dry radius in m)."""
    aa = 2.0e4 * 18.0 * 76.0 / (8.3e7 * 273.0)
    r = rdry * 1e6
    slog = torch.log(rh.clamp(1e-10, 1.0 - 1e-4))
    pp = hygro * r / aa
    p3, h = -aa / (slog * r), -hygro / slog
    y = (1.0 + h) ** (1.0 / 3.0)  # without the curvature term: an upper bound
    for _ in range(60):  # convex above the root: Newton falls monotonically
        f = (y ** 3 - 1) * (y + p3) - h * y
        df = 3 * y * y * (y + p3) + y ** 3 - 1 - h
        y = torch.maximum(y - f / df, torch.ones_like(y))
    small = 1.0 + pp / 3.0 / (1.0 - slog * r / aa)
    return (r * torch.where(pp < 1e-4, small, y)).clamp(max=30.0) * 1e-6


def _wet_modes(x):
    """Dry and wet diameters, wet densities and aerosol water of the modes."""
    t, p, cld = x[wl.IN_T], x[wl.IN_P], x[wl.IN_CLD]
    qs = _qsat(_svp_water(t), p)
    rh = torch.where(qs > x[wl.IN_QV], x[wl.IN_QV] / qs, 0.98).clamp(0.0, 0.98)
    rh = torch.where(cld < 1.0, (rh - cld) / (1.0 - cld), rh).clamp(min=0.0)
    dgn = _dry_sizes(x)
    wet, dens, water = [], [], []
    for m in range(4):
        vol = hyg = mass = 0.0
        for s in wl.MODE_SPECIES_SLOTS[m]:
            sp, q = wl.POPULATIONS[s][1], x[wl.IN_AER_I + s]
            vol, hyg, mass = vol + q / DENS[sp], hyg + q / DENS[sp] * HYGRO[sp], mass + q
        hyg = hyg / vol
        dryvol = math.pi / 6 * dgn[m] ** 3 * math.exp(4.5 * math.log(SIG[m]) ** 2)
        dryrad = (dryvol * 3 / (4 * math.pi)) ** (1.0 / 3.0)
        rad = torch.maximum(_kohler(dryrad, hyg, rh), dryrad)
        wtr = (4 * math.pi / 3 * rad ** 3 - dryvol).clamp(min=0.0)
        hyst = wtr / (0.8 - 0.35) * (rh - 0.35)
        between, dry = rh < 0.8, rh < 0.35
        wtr = torch.where(dry, 0.0, torch.where(between, hyst, wtr))
        rad = torch.where(between, ((dryvol + wtr) * 3 / (4 * math.pi)) ** (1.0 / 3.0), rad)
        rad = torch.where(dry, dryrad, rad)
        wet.append(dgn[m] * rad / dryrad)
        dens.append((mass / vol * dryvol + 1e3 * wtr) / (dryvol + wtr))
        water.append(1e3 * vol / dryvol * wtr)
    return dgn, wet, dens, water


def _exact_activate(s):
    x, rho, w, t = s["x"], s["rho"], s["w"], s["x"][wl.IN_T]
    rgas, mwv = 6.022214076e23 * 1.380649e-23, 0.018016
    rair, rv, lat, cp, grav = rgas / 0.028966, rgas / mwv, 2.501e6, 1.00464e3, 9.80616
    na, vol, hyg = [], [], []
    for m in range(4):
        v = _volume(x, wl.IN_AER_I, m)
        h = sum(x[wl.IN_AER_I + k].clamp(min=0.0) / DENS[wl.POPULATIONS[k][1]]
                * HYGRO[wl.POPULATIONS[k][1]] for k in wl.MODE_SPECIES_SLOTS[m])
        hyg.append(torch.where(v > 1e-30, h / v, 0.0))
        vol.append(torch.where(v > 1e-30, v * rho, 0.0))
        na.append(_clip(vol[m] * _v2n(DMAX[m], m), x[wl.IN_AER_I + wl.NUMBER_SLOTS[m]] * rho,
                        vol[m] * _v2n(DMIN[m], m)))
    p = rair * rho * t
    warm = torch.where(t >= 253.15, _svp_water(t), 0.0)
    wgt = ((273.15 - t) / 20.0).clamp(0.0, 1.0)
    qs = _qsat(torch.where(t < 273.15, wgt * _svp_ice(t) + (1 - wgt) * warm, warm), p)
    aten = 2.0 * mwv * 1e3 * 0.076 / (rgas * 1e3 * 273.0 * 1e3)
    alpha = grav * (lat / (cp * rv * t * t) - 1.0 / (rair * t))
    gamma = (1.0 + lat / cp * lat / (rv * t * t) * qs) / (rho * qs)
    diff = 0.211e-4 * (1013.25e2 / p) * (t / 273.0) ** 1.94
    cond = (5.69 + 0.017 * (t - 273.0)) * 4.186e2 * 1e-5
    gth = 1.0 / (1e3 / (diff * rho * qs) + lat * 1e3 / (cond * t) * (lat / (rv * t) - 1.0))
    beta = 2.0 * math.pi * 1e3 * gth * gamma
    alw = alpha * w.clamp(min=1e-30)
    zeta = 2.0 / 3.0 * torch.sqrt(alw) * aten / torch.sqrt(gth)
    smc, eta = [], []
    for m in range(4):
        ls = math.log(SIG[m])
        am = 0.75 * vol[m] / (math.pi * math.exp(4.5 * ls * ls) * na[m])
        has = (vol[m] > 1e-39) & (na[m] > 1e-39)
        sc = torch.where(hyg[m] > 1e-10, 2 * aten * torch.sqrt(aten / (27.0 * hyg[m] * am)), 100.0)
        smc.append(torch.where(has, sc, 1.0))
        eta.append(alw ** 1.5 * torch.where(has, 1.0 / (na[m] * beta * torch.sqrt(gth)),
                                            1e10 / (alpha * 10.0) ** 1.5))
    total, weak = torch.zeros_like(t), torch.ones_like(t, dtype=torch.bool)
    for m in range(4):
        ls = math.log(SIG[m])
        weak &= (zeta > 1e5 * eta[m]) | (smc[m] ** 2 > 1e5 * eta[m])
        g = (0.5 * math.exp(2.5 * ls * ls) * (zeta / eta[m]) ** 1.5
             + (1.0 + 0.25 * ls) * (smc[m] / torch.sqrt(eta[m] + 3 * zeta)) ** 1.5) / smc[m] ** 2
        total = torch.where(eta[m] > 1e-20, total + g, 1e20)
    smax = torch.where(weak, 1e-20, 1.0 / torch.sqrt(total))
    fn, fm = [], []
    for m in range(4):
        ls = math.log(SIG[m])
        an = 2.0 / 3.0 * (torch.log(smc[m]) - torch.log(smax)) / (math.sqrt(2.0) * ls)
        fn.append(0.5 * torch.erfc(an))
        fm.append(0.5 * torch.erfc(an - 1.5 * math.sqrt(2.0) * ls))
    on = (na[0] >= 1e-20) & (w > 0)
    fn, fm = (torch.where(on, torch.stack(f), 0.0) for f in (fn, fm))
    return {"fn": fn, "fm": fm, "fluxn": fn * w, "fluxm": fm * w, "full": torch.where(on, w, 0.0)}


def _bracket(grid, v):
    """Bracket index and fraction of v in an ascending grid."""
    n = grid.numel()
    i = (torch.searchsorted(grid, v.contiguous(), right=True) - 1).clamp(0, n - 1)
    j = (i + 1).clamp(max=n - 1)
    dx = grid[j] - grid[i]
    return i, j, torch.where(dx.abs() > 1e-20, (v - grid[i]) / dx, torch.zeros_like(v))


def _tropopause(s):
    """Tropopause level of every column (WMO lapse rate, from below)."""
    ncol, nlev = s["ncol"], s["nlev"]
    t = s["x"][wl.IN_T].view(ncol, nlev)
    p = s["x"][wl.IN_P].view(ncol, nlev)
    rd = 6.022214076e23 * 1.380649e-23 / 0.028966
    kap, faktor = rd / 1.00464e3, -9.80616 / rd
    pk = p ** kap
    pmk = 0.5 * (pk[:, :-1] + pk[:, 1:])
    pm = pmk ** (1 / kap)
    a1 = (t[:, :-1] - t[:, 1:]) / (pk[:, :-1] - pk[:, 1:])
    tm = a1 * pmk + t[:, 1:] - a1 * pk[:, 1:]
    lapse = faktor * a1 * kap * pm ** (kap - 1) * pm / tm  # index k - 1 for layer k
    tp = torch.full((ncol,), -99.0, dtype=F64, device="cuda")
    for k in range(nlev - 2, 0, -1):
        l0, l1 = lapse[:, k], lapse[:, k - 1]
        ag = (l1 - l0) / (pmk[:, k - 1] - pmk[:, k])
        cross = ((-0.002 - (l0 - ag * pmk[:, k])) / ag) ** (1 / kap)
        ptph = torch.where(l0 < -0.002, cross, pm[:, k - 1])
        go = (tp < 0) & (l1 > -0.002) & (pm[:, k - 1] <= 45000.0)
        go &= (ptph >= 7500.0) & (ptph <= 45000.0)
        p2km = ptph + 2000.0 * (pm[:, k - 1] / tm[:, k - 1]) * faktor
        total, count = torch.zeros_like(ptph), torch.zeros_like(ptph)
        for j in range(k, 0, -1):
            seen = go & (pm[:, j - 1] <= ptph)
            found = seen & (pm[:, j - 1] < p2km)
            tp = torch.where(found, ptph, tp)
            go = go & ~found
            seen = seen & ~found
            total = total + torch.where(seen, lapse[:, j - 1], 0.0)
            count = count + seen
            go = go & ~(seen & (total / count.clamp(min=1) <= -0.002))
    pint = s["pint"].view(ncol, nlev + 1)
    k = torch.arange(nlev, device="cuda")[None, :]
    ok = (tp[:, None] >= pint[:, :nlev]) & (k > 1) & (tp[:, None] > 0)
    return torch.where(ok, k, 0).amax(1)


def _exact_rad(s):
    sw = s["kind"] == "rad_sw"
    tab = wl.make_optics_sw_tables() if sw else wl.make_optics_lw_tables()
    tab = {k: torch.tensor(np.ascontiguousarray(v), device="cuda") for k, v in tab.items()}
    x, ncol, nlev, n = s["x"], s["ncol"], s["nlev"], s["n"]
    _, wet, _, water = _wet_modes(x)
    mass = s["pdel"] / 9.80616
    nb = 14 if sw else 16
    out = torch.zeros(((4 if sw else 1) * nb, n), dtype=F64, device="cuda")
    lo, hi = math.log(0.01e-6), math.log(25e-6)
    aod = torch.zeros(n, dtype=F64, device="cuda")
    for m in range(4):
        rad = 0.5 * wet[m] * math.exp(2 * math.log(SIG[m]) ** 2)
        lrad = torch.log(rad)
        c1 = (2 * lrad.clamp(lo, hi) - hi - lo) / (hi - lo)
        cheb = [0.5 * torch.ones_like(c1), c1]
        prev = torch.ones_like(c1)
        for _ in range(3):
            prev, new = cheb[-1], 2 * c1 * cheb[-1] - prev
            cheb.append(new)
        wv = (water[m] / 1e3).clamp(min=0.0)
        for b in range(nb):
            re, im = wv * tab["water_refindex"][b, 0], wv * tab["water_refindex"][b, 1]
            vol = wv.clone()
            for k in wl.MODE_SPECIES_SLOTS[m]:
                sp = wl.POPULATIONS[k][1]
                v = x[wl.IN_AER_I + k] / DENS[sp]
                idx = tab["specrefindex"][b, TYPES[sp]]
                vol, re, im = vol + v, re + v * idx[0], im + v * idx[1]
            i0, i1, ft = _bracket(tab["refrtab"][m, b], re / vol)
            j0, j1, fu = _bracket(tab["refitab"][m, b], (im / vol).abs())

            def fit(t):
                tot = 0.0
                for c in range(5):
                    g = t[m, b, c]
                    tot = tot + cheb[c] * ((1 - ft) * (1 - fu) * g[i0, j0] + ft * (1 - fu) * g[i1, j0]
                                           + ft * fu * g[i1, j1] + (1 - ft) * fu * g[i0, j1])
                return tot

            pabs = fit(tab["absp"]) * vol * 1e3
            if not sw:
                out[b] += pabs.clamp(min=0.0) * mass
                continue
            pext = torch.where(lrad <= hi, torch.exp(fit(tab["extp"])), 1.5 / (rad * 1e3))
            pext = pext * vol * 1e3
            alb = 1.0 - _clip(torch.zeros_like(pabs), pabs, pext) / pext.clamp(min=1e-40)
            asm = fit(tab["asmp"])
            v = pext * mass
            if b == 9:
                aod += v
            for q in range(4):
                out[q * nb + b] += v
                v = v * (alb if q == 0 else asm)
    lev = _tropopause(s)
    zi = s["zi"].view(ncol, nlev + 1)
    thick = (zi[:, :-1] - zi[:, 1:]).reshape(-1)
    k = torch.arange(nlev, device="cuda")[None, :]
    above, at = (k < lev[:, None]).reshape(-1), (k == lev[:, None]).reshape(-1)
    for b in range(nb):
        v = thick * s["ext"][b]
        for q in range(4 if sw else 1):
            o = out[q * nb + b]
            out[q * nb + b] = torch.where(above, v, torch.where(at, 0.5 * (o + v), o))
            if sw:
                v = v * (s["ssa"][b] if q == 0 else s["af"][b])
    if not sw:
        return {"tau": out, "trop": None}
    return {"tau": out[0:14], "wa": out[14:28], "ga": out[28:42], "fa": out[42:56],
            "aod": aod.view(ncol, nlev).sum(1), "trop": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "activate":
        return _exact_activate(prepare(case, seed))
    if kind in ("rad_sw", "rad_lw"):
        return _exact_rad(prepare(case, seed))
    if kind in ("mixed", "adjoint", "dropmix"):
        return None  # mixed: FP32 inside; adjoint, dropmix: branches and sub-steps
    ncol, nlev = case["ncol"], case["nlev"]
    x = _fields(_Draw(seed, ncol * nlev), ncol, nlev, case["sky"])
    names = ("dgn_a", "dgn_awet", "wetdens", "qaerwat")
    return {k: torch.stack(v) for k, v in zip(names, _wet_modes(x))}
