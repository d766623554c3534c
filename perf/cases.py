"""Workloads of the column radiative transfer, from one latitude row to a large grid.

Each case is one radiation step as a host program asks for it, through the
public entry points of ``mgcm_rt.abi``:

  run      the drop-in call on the level arrays (host buffers or CUDA tensors)
  tracers  the call from tracer mixing ratios (aerosol optics on the device)
  state    the call from the model state (column prep on the device)
  multi    grids of several layer counts in one call
  graph    the same, captured once and replayed
  serve    a burst of requests through submit/wait
  partial  the partial radiation between full calls (dsolflux)

Columns are drawn by ``mgcm_rt.synth`` (surface pressure, temperature, dust,
water, ice and sun of Mars, half of the columns at night).  A case of more
than ``BASE`` columns repeats a batch of that many with another dust amount,
sun, albedo and emissivity for every column.  The k tables and the Mie tables
are smooth synthetic ones in the formats of the data files, written to a
temporary folder: the column optical depths per band and Gauss point span the
range of the CO2 and water bands, so about half of the visible and nine tenths
of the IR systems of a day column pass the optical-depth screens.
"""
import functools
import math
import pathlib
import sys
import tempfile

import numpy as np
import torch

_ROOT = pathlib.Path(__file__).resolve().parents[1]
sys.path.insert(0, str(_ROOT / "legacy-mars-global-climate-model_b200"))

from mgcm_rt import abi, data, synth  # noqa: E402

BASE = 4096
NV, NI, NG = 7, 5, 17
FP64, MIXED = "fp64", "mixed"
MANY = ("multi", "graph", "serve")       # several grids in one pass


# ------------------------------------------------------------------ cases
def listed():
    return [
        # one latitude circle of the default grid: the smallest call a host
        # makes, where latency counts
        dict(name="row60_l24_fp64", kind="run", where="device", precision=FP64, grids="60x24", cloud=True),
        # the reference's default grid, drop-in level arrays in host memory
        dict(name="grid36x60_l24_host_fp64", kind="run", where="host", precision=FP64, grids="2160x24",
             cloud=False),
        # the default grid from the model state, prescribed dust and ice clouds
        dict(name="grid36x60_l24_state_host", kind="state", where="host", precision=MIXED, grids="2160x24",
             cloud=True, active_dust=False),
        # partial radiation of a 180x360 grid, every time step between full calls
        dict(name="partial64800", kind="partial", where="device", precision=FP64, grids="64800x24", cloud=False),
        # an ordinary regional grid with more layers
        dict(name="grid72x120_l36_mixed", kind="run", where="device", precision=MIXED, grids="8640x36", cloud=True),
        # an odd number of columns and layers, no clouds, plain FP64
        dict(name="ragged10007_l49_fp64", kind="run", where="device", precision=FP64, grids="10007x49",
             cloud=False),
        # a 90x180 grid from tracers in host memory: active dust and ice
        dict(name="grid90x180_l24_tracers_host", kind="tracers", where="host", precision=MIXED, grids="16200x24",
             cloud=True, active_dust=True),
        # the 180x360 grid, inputs resident on the device, both precisions
        dict(name="grid180x360_l24_fp64", kind="run", where="device", precision=FP64, grids="64800x24", cloud=True),
        dict(name="grid180x360_l24_mixed", kind="run", where="device", precision=MIXED, grids="64800x24",
             cloud=True),
        # an ensemble of uneven grids in one captured graph
        dict(name="ensemble_graph_mixed", kind="graph", where="device", precision=MIXED,
             grids="2160x24 2160x24 8640x36 8640x36 16200x48 16200x48", cloud=True),
        # a burst of requests of different sizes and layer counts
        dict(name="serve_burst_fp64", kind="serve", where="device", precision=FP64,
             grids="1031x24 20000x48 4097x36 30011x24 2500x48", cloud=True),
        # a large single request
        dict(name="grid270x480_l48_mixed", kind="run", where="device", precision=MIXED, grids="129600x48",
             cloud=True),
    ]


def _grids(case):
    """(columns, layers) of each grid of a case: "2160x24 8640x36"."""
    return [tuple(int(x) for x in g.split("x")) for g in case["grids"].split()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _layers(rng):
    return rng.choice([24, 24, 36, 48, rng.randint(12, 60)])


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "tracers", "state", "multi", "graph", "serve", "partial"])
    case = dict(kind=kind, where="device", precision=rng.choice([FP64, MIXED]), cloud=rng.random() < 0.7)
    if kind == "run":
        case["where"], layers = rng.choice(["device", "device", "host"]), _layers(rng)
        case["grids"] = "%dx%d" % (_log_int(rng, 40, 20000 if case["where"] == "host" else 6000000 // layers), layers)
    elif kind in ("tracers", "state"):
        case["where"] = rng.choice(["device", "host"])
        case["active_dust"] = rng.random() < 0.5
        case["grids"] = "%dx%d" % (_log_int(rng, 500, 40000), _layers(rng))
    elif kind == "partial":
        case["grids"] = "%dx24" % _log_int(rng, 2000, 300000)
    else:
        n = rng.randint(2, 8)
        case["grids"] = " ".join("%dx%d" % (_log_int(rng, 500, 12000), _layers(rng)) for _ in range(n))
    return case


def work(case):
    """Inputs read once and outputs written once; operations of the reference
    algorithm per column (additions, products, quotients, roots, exponentials
    one each), linear in the layers."""
    nbytes = flops = 0
    for ncol, L in _grids(case):
        lev, lev1, nl = 2 * L + 3, 2 * L + 4, L + 1
        state = 2 * NG * NV          # DETAU, CUMTAUV
        out = 9 * nl + 7
        if case["kind"] == "partial":
            nbytes += 8 * ncol * (NG * NV + 3)
            flops += ncol * NG * NV * 5
            continue
        if case["kind"] == "state":
            inp = L + 6 + (2 * L if case["active_dust"] else 2) + L + (3 * L if case["cloud"] else 0)
        elif case["kind"] == "tracers":
            inp = 5 * lev + 4 + (2 * L if case["active_dust"] else lev1) + (3 * L if case["cloud"] else 0)
        else:
            inp = 5 * lev + 4 + 38 * lev1 * (2 if case["cloud"] else 1)
        nbytes += 8 * ncol * (inp + out + state)
        flops += ncol * (21700 * L + 18000)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ tables
# log10 of the gas optical depth of a 6.5 mbar column per band and Gauss point
# 1..16: the weights of points 9..16 sum to 0.05, so they sit in the line
# centres
_LOG_TAU_V = np.array([
    [-8.2, -7.4, -6.7, -5.3, -3.9, -2.7, 1.1, 2.8, 3.1, 3.2, 3.3, 3.5, 3.8, 4.3, 5.0, 7.4],
    [-5.7, -5.0, -4.3, -3.7, -2.8, -0.7, 0.8, 1.5, 1.8, 1.9, 2.0, 2.2, 2.5, 3.0, 3.7, 5.7],
    [-9.7, -8.5, -7.2, -5.3, -3.5, -2.0, -1.0, -0.3, 0.0, 0.1, 0.2, 0.5, 0.8, 1.2, 1.9, 4.0],
    [-8.5, -7.0, -5.9, -5.1, -4.3, -3.6, -2.6, -1.8, -1.5, -1.4, -1.3, -1.0, -0.7, -0.3, 0.4, 2.5],
    [-10.2, -9.2, -8.5, -7.8, -7.1, -6.3, -5.3, -4.3, -3.9, -3.8, -3.6, -3.4, -3.0, -2.5, -1.6, 0.9],
    [-13.1, -11.7, -10.9, -10.2, -9.5, -8.8, -8.0, -7.2, -6.9, -6.8, -6.7, -6.5, -6.1, -5.7, -5.0, -2.4],
    [-14.2, -13.4, -12.5, -11.8, -11.0, -10.3, -9.6, -9.0, -8.8, -8.7, -8.6, -8.5, -8.3, -8.0, -7.7, -7.0]])
_LOG_TAU_I = np.array([
    [-2.6, -2.1, -1.7, -1.3, -0.9, -0.5, -0.1, 0.3, 0.5, 0.6, 0.8, 1.0, 1.3, 1.6, 2.1, 3.0],
    [-2.8, -2.5, -2.1, -1.7, -1.3, -0.9, -0.4, 0.2, 0.4, 0.5, 0.7, 0.9, 1.2, 1.6, 2.2, 3.2],
    [-1.2, -0.6, -0.1, 0.4, 0.9, 1.4, 2.0, 2.6, 2.9, 3.0, 3.2, 3.4, 3.7, 4.1, 4.7, 6.2],
    [-2.9, -2.5, -2.1, -1.7, -1.3, -0.8, -0.3, 0.3, 0.6, 0.7, 0.9, 1.1, 1.4, 1.8, 2.5, 4.2],
    [-4.1, -3.3, -2.7, -2.2, -1.6, -1.0, -0.3, 0.5, 0.9, 1.0, 1.2, 1.5, 1.9, 2.4, 3.2, 5.4]])
_FZERO_V = [0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.94]
_FZERO_I = [0.0] * 5


def _k_table(log_tau, rng):
    """k(Gauss, band, H2O, pressure, temperature): the wings of the lines grow
    with pressure, their centres fall; hot bands and water raise it."""
    nb = log_tau.shape[0]
    centre = np.linspace(0.0, 1.0, 16)
    logp = np.arange(-6.0, 5.0)
    temp = 50.0 * np.arange(1, 8)
    wref = np.array([1e-7, 1e-6, 1e-5, 1e-4, 1e-3, 1e-2, 1e-1, 0.2, 0.3, 0.4])
    logk = (log_tau.T - math.log10(3.51e22 * 6.5))[:, :, None, None, None]
    logk = logk + ((0.9 - 1.5 * centre)[:, None] * (logp - 0.5)[None, :])[:, None, None, :, None]
    hot = (0.25 + 0.15 * np.arange(nb))[None, :] * (1.0 - 0.8 * centre)[:, None]
    logk = logk + hot[:, :, None, None, None] * ((temp - 200.0) / 100.0)
    logk = logk + np.log10(1.0 + wref / 3e-3)[None, None, :, None, None] * 0.5
    k = np.zeros((NG, nb, 10, 11, 7))
    k[:16] = 10.0 ** (logk + 0.03 * rng.standard_normal(k[:16].shape))
    return k


def _mie(radius, wave, albedo):
    """Extinction, scattering and asymmetry of spheres, smooth in the size."""
    x = 2.0 * math.pi * radius / wave
    q = 2.1 * x * x / (1.5 + x * x) + 0.6 * x / (1.0 + x * x)
    return np.broadcast_arrays(q, albedo * q * x / (0.15 + x), 0.85 * x / (0.8 + x))


@functools.lru_cache(maxsize=None)
def _folder():
    """The synthetic data files; the folder lives as long as the process."""
    keep = tempfile.TemporaryDirectory(prefix="mgcm_rt_tables_")
    d = pathlib.Path(keep.name)
    rng = np.random.default_rng(20101)
    for name, tau, fz in ((data.KV_FILE, _LOG_TAU_V, _FZERO_V), (data.KI_FILE, _LOG_TAU_I, _FZERO_I)):
        with open(d / name, "wb") as f:
            for rec in (_k_table(tau, rng), np.asarray(fz)):
                raw = np.ascontiguousarray(rec, dtype="<f8").tobytes()
                mark = np.int32(len(raw)).tobytes()
                f.write(mark + raw + mark)
    radius = 1e-7 * (500.0 ** (np.arange(20) / 19.0))
    wave_v, wave_i = 1e-6 * np.array([3.8, 2.8, 2.1, 1.5, 1.0, 0.55, 0.3]), 1e-6 * np.array([113.0, 34.0, 16.0, 9.6, 5.8])
    core = np.array([0.1, 0.2, 0.25, 0.3, 0.35, 0.4, 0.45, 0.5, 0.55, 0.6, 0.65, 0.7, 0.8, 0.9, 0.99])
    alb_v, alb_i = np.array([0.75, 0.9, 0.97, 0.97, 0.97, 0.93, 0.75]), np.array([0.1, 0.15, 0.3, 0.35, 0.7])
    for name, wave, alb in ((data.ICE_VIS_FILE, wave_v, np.minimum(1.0, alb_v + 0.04)),
                            (data.ICE_IR_FILE, wave_i, alb_i)):
        t = np.stack(_mie(radius[None, :, None], wave, alb * (1.0 - 0.05 * core[:, None, None])), axis=2)
        (d / name).write_text("\n".join("%.6e" % v for v in t.ravel()))
    for name, wave, alb in (("Dust_vis_wolff2010_JD_12bands.dat", wave_v, alb_v),
                            ("Dust_ir_wolff2010_JD_12bands.dat", wave_i, alb_i)):
        t = np.stack(_mie(radius[:, None], wave, alb), axis=1)
        (d / name).write_text("\n".join("%.6e" % v for v in t.ravel()))
    return keep


# ------------------------------------------------------------------ inputs
def _grid_inputs(case, ncol, L, seed):
    """Host batch of min(ncol, BASE) columns and what differs per column."""
    base = min(ncol, BASE)
    kind, d = case["kind"], _folder().name
    if kind == "tracers":
        b = synth.make_tracer_batch(base, L=L, seed=seed, active_dust=case["active_dust"], cloudon=case["cloud"],
                                    data_dir=d)
    elif kind == "state":
        b = synth.make_state_batch(base, L=L, seed=seed, active_dust=case["active_dust"], cloudon=case["cloud"],
                                   vary_conr=True, data_dir=d)
    else:
        b = synth.make_batch(base, L=L, seed=seed, cloud=case["cloud"], data_dir=d)
    b.pop("meta")
    rng = np.random.default_rng(seed + 15485863)
    vary = None
    if ncol > base:
        day = rng.uniform(size=ncol) >= 0.5
        vary = dict(acosz=np.where(day, rng.uniform(0.0, 1.0, ncol), 0.0), als=rng.uniform(0.1, 0.4, ncol),
                    albi=1.0 - rng.uniform(0.9, 1.0, ncol), dust=np.exp(0.4 * rng.standard_normal(ncol)))
    b["ncol"] = ncol
    return b, vary


_SHARED = ("sigma", "sol")
_DUST = ("tauref", "tautot", "dust_mass", "dust_number")


def _to_device(b, vary, dev):
    """The batch as tensors on `dev`, repeated to its columns."""
    out, n = {}, int(b["ncol"])
    for k, v in b.items():
        if not isinstance(v, np.ndarray):
            out[k] = v
            continue
        t = torch.from_numpy(np.ascontiguousarray(v, dtype=np.float64)).to(dev)
        if vary is not None and k not in _SHARED:
            if k in vary:
                t = torch.from_numpy(vary[k]).to(dev)
            else:
                rep = -(-n // t.shape[0])
                t = t.repeat((rep,) + (1,) * (t.dim() - 1))[:n]
                if k in _DUST:
                    t = t * torch.from_numpy(vary["dust"]).to(dev).reshape((n,) + (1,) * (t.dim() - 1))
        out[k] = t.contiguous()
    return out


def _pinned(t):
    p = torch.empty(t.shape, dtype=torch.float64, pin_memory=True)
    p.copy_(t)
    return p.numpy()


def _batches(case, seed, where):
    """One input batch per grid: CUDA tensors, or numpy arrays in pinned host
    memory for the cases whose host program keeps its fields there."""
    dev = "cpu" if where == "cpu" else "cuda"
    res = []
    for i, (ncol, L) in enumerate(_grids(case)):
        b = _to_device(*_grid_inputs(case, ncol, L, seed + 101 * i), dev)
        if where == "host":
            b = {k: _pinned(v) if torch.is_tensor(v) else v for k, v in b.items()}
        res.append(b)
    return res


def _fields(ncol, L, dev):
    """Output arrays of one grid as slices of one block per kind of field,
    and the blocks."""
    lay, one = (ncol, L + 1), (ncol,)
    groups = dict(fluxes=[(k, lay) for k in abi.OUTPUT_LAY if k != "qrad"], heating=[("qrad", lay)],
                  column=[(k, one) for k in abi.OUTPUT_COL])
    outs, blocks = {}, {}
    for g, members in groups.items():
        blocks[g] = torch.zeros(sum(math.prod(s) for _, s in members), dtype=torch.float64, device=dev)
        at = 0
        for k, s in members:
            outs[k] = blocks[g][at:at + math.prod(s)].view(s)
            at += math.prod(s)
    return outs, blocks


def _partial_inputs(case, seed, dev):
    """What a full call left behind: DETAU of every system and the diffuse
    part, with the sun of this time step."""
    ncol = _grids(case)[0][0]
    rng = np.random.default_rng(seed)
    gas = 10.0 ** np.concatenate([_LOG_TAU_V.T, np.full((1, NV), -9.0)])           # [17][7]
    col = rng.uniform(0.6, 1.6, ncol)
    dust = 0.3 * np.exp(0.6 * rng.standard_normal(ncol))
    acosz = np.where(rng.uniform(size=ncol) < 0.5, 0.0, rng.uniform(0.0, 1.0, ncol))
    t = lambda a: torch.from_numpy(a).to(dev)  # noqa: E731
    detau = t(col)[:, None, None] * t(gas) + 0.5 * t(dust)[:, None, None]
    return dict(sol=t(synth.SOLARF / synth.RSDIST_TUTORIAL), acosz=t(acosz), detau=detau.contiguous(),
                dndiffv=t(rng.uniform(0.0, 80.0, ncol) * (acosz > 0.0)))


# ------------------------------------------------------------------ the calls
class State:
    """A handle with its batches and output buffers, as a host keeps them."""

    def __init__(self, case, seed):
        self.kind, self.where = case["kind"], case["where"]
        max_layers = max(L for _, L in _grids(case))
        self.rt = abi.Radiation(_folder().name, max_layers=max_layers,
                                precision=abi.MIXED if case["precision"] == MIXED else abi.FP64)
        if self.kind == "partial":
            self.args = _partial_inputs(case, seed, "cuda")
            return
        self.batches = _batches(case, seed, self.where)
        dev = "cuda" if self.where == "device" else None
        if self.kind in MANY:
            self.outs, self.blocks = zip(*(_fields(ncol, L, dev) for ncol, L in _grids(case)))
            self.blocks = [dict(g, detau=b["detau"], cumtauv=b["cumtauv"]) for g, b in zip(self.blocks, self.batches)]
        else:
            self.outs = [abi.alloc_outputs(ncol, L, device=dev) for ncol, L in _grids(case)]
        if self.where == "host":
            self.outs = [{k: _pinned(torch.from_numpy(v)) for k, v in o.items()} for o in self.outs]
        if self.kind == "graph":
            self.stream = torch.cuda.Stream()
            torch.cuda.synchronize()
            self.graph = self.rt.graph(self.batches, self.outs)

    def close(self):
        if getattr(self, "graph", None) is not None:
            torch.cuda.synchronize()
            self.graph.close()
            self.graph = None

    def __del__(self):
        self.close()


def prepare(case, seed):
    return State(case, seed)


def run(state):
    rt, kind = state.rt, state.kind
    if kind == "partial":
        a = state.args
        return rt.dsolflux(a["sol"], a["acosz"], a["detau"], a["dndiffv"])
    if kind == "tracers":
        return rt.run_tracers(state.batches[0], state.outs[0], inplace=True)
    if kind == "state":
        return rt.run_state(state.batches[0], state.outs[0], inplace=True)
    if kind == "run":
        return rt.run(state.batches[0], state.outs[0], inplace=True)
    if kind == "multi":
        rt.run_multi(state.batches, state.outs)
        return state.blocks
    if kind == "graph":
        state.stream.wait_stream(torch.cuda.current_stream())
        state.graph.launch(state.stream)
        torch.cuda.current_stream().wait_stream(state.stream)
        return state.blocks
    tickets = [rt.submit(b, o)[0] for b, o in zip(state.batches, state.outs)]
    for t in tickets:
        rt.wait(t, 60.0)
    return state.blocks


# ------------------------------------------------------------------ the values
# The radiation of COMP3 in plain torch, 64 bits: code/tpindex.f90, optcv.f90,
# optci.f90, getdetau.f90, gfluxv.f90, gfluxi.f90, dsolver.f90, dtridgl.f90,
# sfluxv.f90, sfluxi.f90 and code/comp3.f:637-771, every (band, Gauss) system
# of a chunk of columns at once.  Constants that the reference writes as
# single-precision literals are rounded as they are there.
_PI = 3.1415926535897932


def _f(x):
    return float(np.float32(x))


@functools.lru_cache(maxsize=None)
def _tables(dev):
    d = pathlib.Path(_folder().name)
    lp = np.log10(np.array([1e-6, 1e-5, 1e-4, 1e-3, 1e-2, 1e-1, 1.0, 1e1, 1e2, 1e3, 1e4], dtype=np.float32)
                  .astype(np.float64))
    pf = np.array([float("%.1f" % (-6.0 + 0.2 * i)) for i in range(51)])
    out = {}
    for name, nb, key in ((data.KV_FILE, NV, "kv"), (data.KI_FILE, NI, "ki")):
        raw = np.fromfile(d / name, dtype="<f8", offset=4, count=NG * nb * 10 * 11 * 7).reshape(NG, nb, 10, 11, 7)
        logk = np.where(raw > 1e-200, np.log10(np.maximum(raw, 1e-300)), -200.0)
        fine = np.empty((NG, nb, 10, 51, 7))
        for n in range(10):
            s = min(max(n - 1, 0), 7)
            for m in range(5):
                x = pf[5 * n + m]
                acc = 0.0
                for q in range(4):
                    w = 1.0
                    for r in range(4):
                        if r != q:
                            w = w * (x - lp[s + r]) / (lp[s + q] - lp[s + r])
                    acc = acc + w * logk[:, :, :, s + q]
                fine[:, :, :, 5 * n + m] = acc
        fine[:, :, :, 50] = logk[:, :, :, 10]
        # [temperature, pressure, water, band, Gauss 1..16]
        out[key] = torch.from_numpy(np.ascontiguousarray((10.0 ** fine[:16]).transpose(4, 3, 2, 1, 0))).to(dev)
    bv = np.array([2222.22, 3087.37, 4030.63, 5370.57, 7651.11, 12500.00, 25000.00, 41666.67])
    wl2 = (1.0e4 / (0.5 * (bv[1:] + bv[:-1]))) ** 2
    out["ray"] = (_f(8.7) / 3.72) * (_f(1.527) * (1.0 + _f(0.013) / wl2) / wl2 ** 2) * 100.0 / 9.423e6
    bi = np.array([10.0, 166.667, 416.667, 833.333, 1250.0, 2222.222])
    out["dwi"] = bi[1:] - bi[:-1]
    gx, gw = np.polynomial.legendre.leggauss(12)
    gx, gw = np.round(gx, 15), np.round(gw, 15)
    temp = (np.arange(8501) + 500) / 10.0
    planck = np.empty((8501, NI))
    for w in range(NI):
        a, b = 1.0e-2 / bi[w + 1], 1.0e-2 / bi[w]
        y = (b - a) / 2.0 * gx + (b + a) / 2.0
        f = 3.741832e-16 / (y ** 5 * (np.exp(1.438786e-2 / (y * temp[:, None])) - 1.0))
        planck[:, w] = (f * gw).sum(axis=1) * (b - a) / 2.0 / (_PI * out["dwi"][w])
    wt = np.array([4.8083554740e-02, 1.0563099137e-01, 1.4901065679e-01, 1.7227479710e-01, 1.7227479710e-01,
                   1.4901065679e-01, 1.0563099137e-01, 4.8083554740e-02, 2.5307134073e-03, 5.5595258613e-03,
                   7.8426661469e-03, 9.0670945845e-03, 9.0670945845e-03, 7.8426661469e-03, 5.5595258613e-03,
                   2.5307134073e-03])
    out.update(planck=planck, wt=wt, fzv=np.array(_FZERO_V), fzi=np.array(_FZERO_I), pf=pf,
               wref=np.array([1e-7, 1e-6, 1e-5, 1e-4, 1e-3, 1e-2, 1e-1, 0.2, 0.3, 0.4]))
    return {k: torch.from_numpy(v).to(dev) if isinstance(v, np.ndarray) else v for k, v in out.items()}


def _gas(T, tab, p, t, q, u):
    """Gas optical depth of one level: [column][band][16]."""
    mt = (torch.ceil(t / 50.0) - 2.0).clamp(0, 5).long()
    uu = (t - 50.0 * (mt + 1)) / 50.0
    lp = torch.log10(p)
    mp = (torch.searchsorted(T["pf"], lp.contiguous()) - 1).clamp(0, 49)
    tt = (lp - T["pf"][mp]) / (T["pf"][mp + 1] - T["pf"][mp])
    inside = (q > T["wref"][0]) & (q < T["wref"][9])
    nh = torch.where(q >= T["wref"][9], 9, (torch.searchsorted(T["wref"], q.contiguous(), right=True) - 1).clamp(0, 9))
    nh = torch.where(q <= T["wref"][0], 0, nh)
    nh1 = (nh + 1).clamp(max=9)
    wr = torch.where(inside, (q - T["wref"][nh]) / (T["wref"][nh1] - T["wref"][nh]).clamp(min=1e-300), 0.0)[:, None, None]

    def corner(a, b):
        c0 = tab[a, b, nh]
        return c0 + wr * (tab[a, b, nh1] - c0)
    w = lambda x: x[:, None, None]  # noqa: E731
    k = w((1 - tt) * (1 - uu)) * corner(mt, mp) + w(tt * (1 - uu)) * corner(mt, mp + 1) \
        + w(tt * uu) * corner(mt + 1, mp + 1) + w((1 - tt) * uu) * corner(mt + 1, mp)
    return w(u) * k


def _two_stream(lays, btop, bsurf, rsf):
    """DSOLVER rows, DTRIDGL and the unmixing: XK1, XK2 per layer.  A layer is
    (gama, e1, e2, e3, e4, cp, cm, cpm1, cmm1)."""
    rows = []
    hi = lays[-1]
    g, e1, e2, e3, e4, cp, cm, cpm1, cmm1 = hi
    bf = e2 - rsf * e4
    a, d = (e1 - rsf * e3) / bf, (bsurf - cp + rsf * cm) / bf
    rows.append((a, d))
    for lo in reversed(lays[:-1]):
        gl, a1, a2, a3, a4, lcp, lcm, _, _ = lo
        gh, hcpm1, hcmm1 = hi[0], hi[7], hi[8]
        for af, bf, cf, df in (
                (2.0 * (1.0 - gl * gl), (a1 - a3) * (1.0 + gh), (a1 + a3) * (gh - 1.0),
                 a3 * (hcpm1 - lcp) + a1 * (lcm - hcmm1)),
                ((a1 + a3) * (gh - 1.0), (a2 + a4) * (gh - 1.0), 2.0 * (1.0 - gh * gh),
                 (gh - 1.0) * (hcpm1 - lcp) + (1.0 - gh) * (lcm - hcmm1))):
            x = 1.0 / (bf - cf * a)
            a, d = af * x, (df - cf * d) * x
            rows.append((a, d))
        hi = lo
    x = 1.0 / (hi[0] + 1.0 - (hi[0] - 1.0) * a)
    rows.append((0.0 * x, (btop - hi[8] - (hi[0] - 1.0) * d) * x))
    rows.reverse()
    xs, prev = [], 0.0
    for a, d in rows:
        prev = d - a * prev
        xs.append(prev)
    res = []
    for n in range(len(lays)):
        xa, xb = xs[2 * n], xs[2 * n + 1]
        xk2 = xa - xb
        xk2 = torch.where((xk2 != 0.0) & ((xk2 / (xa + _f(1e-20))).abs() < _f(1e-30)), 0.0, xk2)
        res.append((xa + xb, xk2))
    return res


def _edge(g, ep, cp, cm, cpm1, cmm1):
    em = 1.0 / ep
    return (g, ep + g * em, ep - g * em, g * ep + em, g * ep - em, cp, cm, cpm1, cmm1)


def _band_sum(v, keep, wt, fz, scale):
    """Sum over the Gauss points and bands; a screened point's weight goes to
    the 17th.  v: [column][band][17]."""
    one = (1.0 - fz)[None, :, None]
    w16 = torch.where(keep[..., :16], wt * one, 0.0)
    w17 = fz[None, :] + torch.where(keep[..., :16], 0.0, wt * one).sum(-1)
    v16 = torch.where(keep[..., :16], v[..., :16], 0.0)
    return ((v16 * w16).sum(-1) * scale + v[..., 16] * w17 * scale).sum(-1)


def _radiation(b, dev):
    T = _tables(dev)
    L = int(b["L"])
    nl, lev = L + 1, 2 * L + 3
    n = b["plev"].shape[0]
    cld = "taurefcld" in b
    lv = lambda a, k: a[:, k - 1]  # noqa: E731  level k, 1-based
    bk = lambda a, k: a[:, :, k - 1]  # noqa: E731
    dpr = [None] * (lev + 1)
    gv, gi = [None] * (lev + 1), [None] * (lev + 1)
    for k in range(2, lev + 1):
        dpr[k] = lv(b["plev"], k) - lv(b["plev"], k - 1)
        args = (lv(b["pmid"], k), lv(b["tmid"], k), lv(b["qh2o"], k), 3.51e22 * dpr[k])
        gv[k], gi[k] = _gas(T, T["kv"], *args), _gas(T, T["ki"], *args)
    zero = torch.zeros(n, 1, device=dev, dtype=torch.float64)

    def dust(q, k, ref):
        return (lv(b["tauref"], k) / ref)[:, None] * bk(q, k)

    def ice(q, k):
        return (lv(b["taurefcld"], k) / lv(b["qextrefcld"], k))[:, None] * bk(q, k) if cld else zero
    full = lambda g, add: torch.cat([g, torch.zeros_like(g[..., :1])], -1) + add[..., None]  # noqa: E731

    # ---- visible
    ray, dtau, sca, asy = [None] * (lev + 1), [None] * (lev + 1), [None] * (lev + 1), [None] * (lev + 1)
    for k in range(2, lev + 1):
        ray[k] = T["ray"][None, :] * dpr[k][:, None]
        ref = b["qxvdst"][:, 5, k - 1]
        dtau[k] = full(gv[k], ray[k] + dust(b["qxvdst"], k, ref) + ice(b["qxvcld"] if cld else None, k))
        sd, sc = dust(b["qsvdst"], k, ref), ice(b["qsvcld"] if cld else None, k)
        sca[k] = sd + sc
        asy[k] = sd * bk(b["gvdst"], k) + (sc * bk(b["gvcld"], k) if cld else 0.0)
    tc = dtau[2]
    tau = torch.zeros_like(tc)
    w0s, cbs, dts, tops, mids, tc_e1 = [], [], [], [tau], [], None
    fprev = None
    for l in range(1, nl + 1):
        ks = [2 * l + 1, 2 * l + 2] if l <= L else [lev]
        ra, s, a = (sum(x[k] for k in ks) for x in (ray, sca, asy))
        cb = (a / (ra + s))[..., None]
        dt = sum(dtau[k] for k in ks)
        wb = (s + ra * _f(0.9999))[..., None] / dt
        f = 1.0 - wb * (cb * cb)
        if l == 1:
            tc_e1 = tc * f
            mids.append(tc_e1 + dtau[ks[0]] * f)
        elif l < nl:
            mids.append(tau + dtau[ks[0]] * fprev)
        w0s.append(wb * (1.0 - cb * cb) / f)
        cbs.append(cb / (1.0 + cb))
        dts.append(dt * f)
        tau = tau + dts[-1]
        tops.append(tau)
        fprev = f
        tc = tc + dt
    day = b["acosz"] >= _f(1e-5)
    detau = torch.where(day[:, None, None], tau.transpose(1, 2), b["detau"])
    cumtau = torch.where(day[:, None, None], tc.transpose(1, 2), b["cumtauv"])
    keep = torch.cat([sum(gv[2:]) >= 1.0e-3, torch.ones(n, NV, 1, device=dev, dtype=torch.bool)], -1)
    u0 = torch.where(day, b["acosz"], 0.5)[:, None, None]
    sol = b["sol"][None, :, None]
    rsf = b["als"][:, None, None]
    s3, s3h = float(np.sqrt(np.float32(3.0))), float(np.sqrt(np.float32(3.0)) * np.float32(0.5))
    beam = lambda x: torch.exp(-(x / u0).clamp(max=35.0))  # noqa: E731
    lays, keepc = [], []
    for l in range(nl):
        w0, cb = w0s[l], cbs[l]
        g1, g2 = s3h * (2.0 - w0 * (1.0 + cb)), s3 * w0 * 0.5 * (1.0 - cb)
        g3 = 0.5 * (1.0 - s3 * cb * u0)
        g4 = 1.0 - g3
        lam = torch.sqrt(g1 * g1 - g2 * g2)
        gam = (g1 - lam) / g2
        den = lam * lam - 1.0 / (u0 * u0)
        den = torch.where(den == 0.0, _f(1e-10), den)
        am = sol * w0 * (g4 * (g1 + 1.0 / u0) + g2 * g3) / den
        ap = sol * w0 * (g3 * (g1 - 1.0 / u0) + g2 * g4) / den
        et, eb = beam(tops[l]), beam(tops[l + 1])
        lays.append(_edge(gam, torch.exp((lam * dts[l]).clamp(max=35.0)), ap * eb, am * eb, ap * et, am * et))
        keepc.append((lam, gam, am, ap))
    bsurf = rsf * u0 * sol * beam(tau)
    xk = _two_stream(lays, 0.0, bsurf, rsf)
    up, dn = [], []
    for l in range(nl):
        (k1, k2), (lam, gam, am, ap) = xk[l], keepc[l]
        if l == 0:
            top = (k1 + gam * k2 + ap) - (k1 * gam + k2 + am + u0 * sol)
        if l < nl - 1:
            at = mids[l]
            ep, et = torch.exp((lam * (at - (tc_e1 if l == 0 else tops[l]))).clamp(max=35.0)), beam(at)
        else:
            ep, et = torch.exp((lam * (tops[nl] - tops[l])).clamp(max=35.0)), beam(tops[nl].clamp(max=35.0))
        em = 1.0 / ep
        up.append(k1 * ep + gam * k2 * em + ap * et)
        dn.append(k1 * ep * gam + k2 * em + am * et)
        if l == nl - 1:
            diff = dn[-1]
        dn[-1] = dn[-1] + u0 * sol * et
    vis = lambda v: torch.where(day, _band_sum(v, keep, T["wt"], T["fzv"], 1.0), 0.0)  # noqa: E731
    out = dict(detau=detau, cumtauv=cumtau, fluxupv=torch.stack([vis(x) for x in up], 1),
               fluxdnv=torch.stack([vis(x) for x in dn], 1),
               fmnetv=torch.stack([vis(x - y) for x, y in zip(up, dn)], 1), nfluxtopv=vis(top), diffvt=vis(diff))

    # ---- infrared
    ext, sca, asy, dtau = [None] * (lev + 2), [None] * (lev + 2), [None] * (lev + 2), [None] * (lev + 1)
    for k in range(2, lev + 2):
        ref = lv(b["qextrefdst"], k) if k <= lev else 1.0
        sd = dust(b["qsidst"], k, ref)
        if cld:
            sc = ice(b["qsicld"], k) if k <= lev else lv(b["taurefcld"], k)[:, None] * bk(b["qsicld"], k)
        else:
            sc = zero
        sca[k] = sd + sc
        asy[k] = sd * bk(b["gidst"], k) + (sc * bk(b["gicld"], k) if cld else 0.0)
        if k <= lev:
            dtau[k] = full(gi[k], dust(b["qxidst"], k, ref) + ice(b["qxicld"] if cld else None, k))
    planck = lambda k: T["planck"][(lv(b["tlev"], k) * 10.0 - 499.0).long().clamp(1, 8501) - 1][..., None]  # noqa: E731
    lays, mid = [], []
    for l in range(1, nl + 1):
        ks = [2 * l + 1, 2 * l + 2] if l <= L else [lev]
        dt = sum(dtau[k] for k in ks) + 1.0e-50
        s, a = sca[2 * l + 1] + sca[2 * l + 2], asy[2 * l + 1] + asy[2 * l + 2]
        cb = torch.where(s > 0.0, a / torch.where(s > 0.0, s, 1.0), 0.0)[..., None]
        thick = dt > _f(1e-9)
        w0 = torch.where(thick, s[..., None] / dt, 0.0)
        dt = torch.where(thick, dt, _f(1e-9))
        alpha = torch.sqrt((1.0 - w0) / (1.0 - w0 * cb))
        lam = alpha * (1.0 - w0 * cb) / 0.5
        gam = (1.0 - alpha) / (1.0 + alpha)
        term = 0.5 / (1.0 - w0 * cb)
        if l < nl:
            b0 = planck(2 * l)
            b1 = (planck(2 * l + 2) - b0) / dt
        else:
            b0 = planck(2 * l)
            b1 = (planck(2 * l + 1) - b0) / dt
        dtk = dtau[2 * l + 1] if l < nl else dt
        if l == 1:
            dt1 = dt
        lays.append(_edge(gam, torch.exp((lam * dt).clamp(max=35.0)), b0 + b1 * dt + b1 * term,
                          b0 + b1 * dt - b1 * term, b0 + b1 * term, b0 - b1 * term))
        mid.append((lam, gam, b0, b1, term, dtk))
    rsf = b["albi"][:, None, None]
    ptop = (lv(b["plev"], 2) / (lv(b["plev"], 4) - lv(b["plev"], 2)))[:, None, None]
    btop = (1.0 - torch.exp(-(dt1 * ptop) / 0.5)) * planck(2)
    bsurf = (1.0 - rsf) * planck(lev)
    xk = _two_stream(lays, btop, bsurf, rsf)
    up, dn = [], []
    for l in range(nl):
        (k1, k2), (lam, gam, b0, b1, term, dtk) = xk[l], mid[l]
        if l == 0:
            top = ((k1 + gam * k2 + b0 + b1 * term) - (k1 * gam + k2 + b0 - b1 * term)) * _PI
        ep = torch.exp((lam * dtk).clamp(max=35.0))
        em = 1.0 / ep
        up.append((k1 * ep + gam * k2 * em + b0 + b1 * dtk + b1 * term) * _PI)
        dn.append((k1 * ep * gam + k2 * em + b0 + b1 * dtk - b1 * term) * _PI)
    keep = torch.cat([sum(gi[2:]) >= 5.0e-3, torch.ones(n, NI, 1, device=dev, dtype=torch.bool)], -1)
    ir = lambda v: _band_sum(v, keep, T["wt"], T["fzi"], T["dwi"])  # noqa: E731
    out.update(fluxupi=torch.stack([ir(x) for x in up], 1), fluxdni=torch.stack([ir(x) for x in dn], 1),
               fmneti=torch.stack([ir(x - y) for x, y in zip(up, dn)], 1), nfluxtopi=ir(top))

    # ---- divergences, heating and the surface
    out["suntot"] = torch.diff(out["fmnetv"], dim=1, prepend=out["nfluxtopv"][:, None])
    out["irtotal"] = torch.diff(out["fmneti"], dim=1, prepend=out["nfluxtopi"][:, None])
    even = torch.arange(2, lev, 2, device=dev)
    ym = (b["plev"][:, even] - b["plev"][:, even - 2]) * 100.0 / 3.72
    ym[:, 0] = float(b["ptrop"]) * 100.0 / 3.72
    om = (b["plev"][:, even - 1] / b["plev"][:, lev - 1:lev]) ** 0.25684
    pn = b["sigma"][even - 1] * (b["pcol"][:, None] - float(b["ptrop"])) + float(b["ptrop"])
    out["qrad"] = (out["suntot"] * 2.2e4 * pn / (1.0 + 2.2e4 * pn) + out["irtotal"]) / (735.94 * ym * om)
    out["dnvflux"], out["dndiffv"], out["dnirflux"] = out["fluxdnv"][:, -1], out["diffvt"], out["fluxdni"][:, -1]
    out["fluxsurf"] = (1.0 - b["als"]) * out["dnvflux"]
    return out


def _state_levels(st):
    """Column prep of COMP3 (code/potemp1.f, fillpt.f90, dustprofile.f,
    filltaucum.f): the level arrays and, for prescribed dust, TAUREF."""
    L, ptrop = int(st["L"]), float(st["ptrop"])
    lev = 2 * L + 3
    p, sig, t = st["pcol"][:, None], st["sigma"], st["t"]
    n, dev = p.shape[0], p.device
    plev = ptrop + sig[None, :] * p
    plev[:, :2] = ptrop / 2.0
    plev[:, lev - 1] = ptrop + p[:, 0]
    tlev = torch.empty_like(plev)
    tlev[:, :3] = st["tstrat"][:, None]
    tlev[:, 3:lev - 1:2] = t
    lo, mi, hi = plev[:, 3:lev - 3:2], plev[:, 4:lev - 2:2], plev[:, 5:lev - 1:2]
    tlev[:, 4:lev - 2:2] = t[:, 1:] + (t[:, :-1] - t[:, 1:]) * torch.log(mi / hi) / torch.log(lo / hi)
    tlev[:, lev - 1] = st["gt"]
    tmid, pmid = tlev.clone(), plev.clone()
    tmid[:, 0] = tlev[:, 1]
    tmid[:, 3:lev - 1:2], pmid[:, 3:lev - 1:2] = tlev[:, 2:lev - 2:2], plev[:, 2:lev - 2:2]
    q = torch.zeros_like(plev)
    q[:, 3:lev - 1:2] = q[:, 4:lev:2] = float(st["mwratio"]) * st["vapour"]
    b = dict(st, plev=plev, tlev=tlev, pmid=pmid, tmid=tmid, qh2o=q)
    if st["active_dust"]:
        return b
    rptau, conr = float(st["rptau"]), st["conr"][:, None]
    step = (5.0 * float(st["psf"]) / ptrop) ** float(np.float32(1.0) / np.float32(99.0))
    pr = ptrop * step ** torch.arange(100, device=dev, dtype=torch.float64)
    shape = lambda x: torch.exp(conr * (1.0 - rptau / x[None, :]))  # noqa: E731
    mid, dp = 0.5 * (pr[1:] + pr[:-1]), pr[1:] - pr[:-1]
    m = int((pr < rptau).sum())                        # pr[m - 1] < rptau <= pr[m]
    last = shape(torch.stack([0.5 * (rptau + pr[m - 1])]))
    total = (shape(mid[:m - 1]) * dp[:m - 1]).sum(1, keepdim=True) + last * (rptau - pr[m - 1])
    rate = torch.ones(n, 99, device=dev, dtype=torch.float64)
    rate[:, :m - 1] = shape(mid[:m - 1])
    rate[:, m - 1:m] = (last * (rptau - pr[m - 1]) + (pr[m] - rptau)) / dp[m - 1]
    cum = torch.cat([torch.zeros(n, 1, device=dev, dtype=torch.float64), torch.cumsum(rate * dp, 1)], 1)
    cum = cum * (st["tautot"][:, None] / total)
    ps = torch.clamp(p * sig[None, 3:] + ptrop, min=ptrop)
    at = (torch.searchsorted(pr[:99], ps.contiguous(), right=True) - 1).clamp(0, 98)
    c0, c1 = cum.gather(1, at), cum.gather(1, at + 1)
    tc = c0 + (ps - pr[at]) * (c1 - c0) / (pr[at + 1] - pr[at])
    b["tauref"] = torch.zeros(n, lev + 1, device=dev, dtype=torch.float64)
    b["tauref"][:, 3:lev] = torch.diff(tc, dim=1, prepend=torch.zeros(n, 1, device=dev, dtype=torch.float64))
    return b


@functools.lru_cache(maxsize=None)
def _mie_tables(dev):
    d = pathlib.Path(_folder().name)

    def read(name, *shape):
        v = np.array([np.float32(x) for x in (d / name).read_text().split()], dtype=np.float64)
        return torch.from_numpy(v.reshape(shape)).to(dev)
    third = float(np.float32(1.0) / np.float32(3.0))
    r0, r1 = _f(1e-7), _f(50e-6)
    vrat = math.exp(math.log(r1 / r0) / 19.0 * 3.0)
    edges = [_f(0.0001e-6)]
    for i in range(19):
        edges.append((2.0 * vrat / (vrat + 1.0)) ** third * r0 * vrat ** (third * i))
    edges.append(_f(1e-2))
    return (torch.tensor(edges, device=dev, dtype=torch.float64), third, read(data.ICE_VIS_FILE, 15, 20, 3, NV),
            read(data.ICE_IR_FILE, 15, 20, 3, NI), read("Dust_vis_wolff2010_JD_12bands.dat", 20, 3, NV),
            read("Dust_ir_wolff2010_JD_12bands.dat", 20, 3, NI))


def _optics(b, dev, ice):
    """OPT_DST / OPT_CLD (code/opt_dst.f, code/opt_cld.f) of a chunk."""
    edges, third, cv, ci, dv, di = _mie_tables(dev)
    L = int(b["L"])
    n, lev1 = b["plev"].shape[0], 2 * L + 4
    if ice:
        ma, mc, nb = b["ice_mass"], b["ice_core_mass"], b["ice_number"]
        on = (ma + mc > _f(1e-7)) & (nb > 1.0)
        mo, no = torch.where(on, ma + mc, 1.0), torch.where(on, nb, 1.0)
        core = (mc / 2500.0 / torch.where(on, ma / 917.0 + mc / 2500.0, 1.0)).float()
        core = (core.double() ** third).float()
        cr = torch.tensor([0.1, 0.2, 0.25, 0.3, 0.35, 0.4, 0.45, 0.5, 0.55, 0.6, 0.65, 0.7, 0.8, 0.9, 0.99],
                          device=dev, dtype=torch.float32)
        row = (torch.searchsorted(cr, core.contiguous(), right=True) - 1).clamp(0, 14)
        tv, ti = cv[row], ci[row]
        dens = ma / mo * 917.0 + mc / mo * 2500.0
        dens = torch.where(on, dens, 1.0)
        dev_, big = _f(0.3087), _f(100e-6)
    else:
        ma, nb = b["dust_mass"], b["dust_number"]
        on = (ma > _f(1e-8)) & (nb > 1.0)
        mo, no, dens = torch.where(on, ma, 1.0), nb + 1.0, 2500.0
        tv, ti = dv, di
        dev_, big = _f(0.63676), _f(50e-6)
    rs = (mo / no * (0.75 / (_PI * dens))) ** third * math.exp(-0.5 * dev_ * dev_)
    area = no * _PI * rs * rs
    rs = (rs * math.exp(1.5 * dev_ * dev_)).clamp(min=_f(1e-7), max=big)
    e = torch.erf(torch.log(edges / rs[..., None]) / (float(np.sqrt(np.float32(2.0))) * dev_))
    surf = 0.5 * (e[..., 1:] - e[..., :-1])
    eq = "nli,nlimw->nlmw" if ice else "nli,imw->nlmw"
    res = {}
    for fam, tab, nbd in (("v", tv, NV), ("i", ti, NI)):
        m = torch.einsum(eq, surf, tab)
        q, s, g = m[:, :, 0], torch.minimum(m[:, :, 1], _f(0.99999) * m[:, :, 0]), m[:, :, 2]
        for key, v, fill in (("qx", q, 1.0), ("qs", s, _f(0.99)), ("g", g, 0.0)):
            a = torch.full((n, nbd, lev1), fill, device=dev, dtype=torch.float64)
            v = torch.where(on[..., None], v, fill).transpose(1, 2)
            a[:, :, 3:lev1 - 2:2] = v
            a[:, :, 4:lev1 - 1:2] = v
            res[key + fam] = a
    suffix = "cld" if ice else "dst"
    out = {k + suffix: v for k, v in res.items()}
    ref = out["qxv" + suffix][:, 5].clone()
    ref[:, :3] = 1.0
    ref[:, lev1 - 1] = 1.0
    mass = 100.0 * torch.diff(b["plev"], dim=1) / 3.72
    tau = torch.zeros(n, lev1, device=dev, dtype=torch.float64)
    act = torch.where(on, area, 0.0)
    for o in (3, 4):
        tau[:, o:lev1 - 2 + o - 3:2] = act * ref[:, o:lev1 - 2 + o - 3:2] * mass[:, o - 1::2][:, :L]
    out["tauref" + ("cld" if ice else "")] = tau
    out["qextref" + suffix] = ref
    return out


def _aerosols(b, dev):
    """The per-level aerosol arrays of a tracer batch (code/comp3.f:592-630)."""
    b = dict(b)
    if b["active_dust"]:
        b.update(_optics(b, dev, False))
    else:
        n, lev1 = b["plev"].shape[0], 2 * int(b["L"]) + 4
        r = _f(0.99999)
        qv, qi = synth.QEV1, synth.QEI1
        sv, si = np.where(synth.QSV1 >= qv, r * qv, synth.QSV1), np.where(synth.QSI1 >= qi, r * qi, synth.QSI1)
        for key, v in (("qxvdst", qv), ("qsvdst", sv), ("gvdst", synth.GV1), ("qxidst", qi), ("qsidst", si),
                       ("gidst", synth.GI1)):
            b[key] = torch.from_numpy(np.asarray(v, dtype=np.float64)).to(dev)[None, :, None].expand(n, -1, lev1)
        b["qextrefdst"] = b["qxvdst"][:, 5]
        b["tauref"] = b["tauref"].clone()
        b["tauref"][:, lev1 - 1] = 0.0
    if b["cloudon"]:
        b.update(_optics(b, dev, True))
    return b


def _exact_grid(case, b, dev):
    n = int(b["ncol"])
    parts = []
    size = 2048 if dev == "cuda" else 512
    for c in range(0, n, size):
        s = {k: v[c:c + size] if torch.is_tensor(v) and k not in _SHARED else v for k, v in b.items()}
        if case["kind"] == "state":
            s = _state_levels(s)
        if case["kind"] in ("state", "tracers"):
            s = _aerosols(s, dev)
        parts.append({k: v.cpu() for k, v in _radiation(s, dev).items()})
    return {k: torch.cat([p[k] for p in parts]).numpy() for k in parts[0]}


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "partial":
        a = _partial_inputs(case, seed, dev)
        T = _tables(dev)
        u0 = torch.where(a["acosz"] >= _f(1e-5), a["acosz"], 1.0)[:, None, None]
        w = torch.cat([T["wt"][:, None] * (1.0 - T["fzv"]), T["fzv"][None, :]])
        d = a["detau"]
        term = torch.where(d <= 5.0, u0 * a["sol"] * torch.exp(-d / u0) * w, 0.0).sum((1, 2))
        return (a["dndiffv"] + torch.where(a["acosz"] >= _f(1e-5), term, 0.0)).cpu().numpy()
    cells = sum(n * L for n, L in _grids(case))
    if cells > (7_000_000 if dev == "cuda" else 60_000):
        return None
    outs = [_exact_grid(case, b, dev) for b in _batches(case, seed, dev)]
    if case["kind"] not in MANY:
        return outs[0]
    join = lambda o, names: np.concatenate([o[k].ravel() for k in names])  # noqa: E731
    return [dict(fluxes=join(o, [k for k in abi.OUTPUT_LAY if k != "qrad"]), heating=o["qrad"].ravel(),
                 column=join(o, abi.OUTPUT_COL), detau=o["detau"], cumtauv=o["cumtauv"]) for o in outs]
