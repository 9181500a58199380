"""Performance cases: the calls a simulator makes through this package, over
the sizes it makes them at.

A FIM time step runs, per Newton iteration, the flash with its derivatives
over every bulk (warm-started from the last iterate), KrPc, the upstream
choice and the Jacobian's bulk part. Beside it stand the fresh flash of a
block (initial states, screening studies), the IMPEC and FIMn formulations,
several PVT regions in one call, the host-buffer call of an application that
keeps its Bulk arrays on the host, and a training step of the learned
initialiser.

``listed()`` holds one case of each, ``draw(rng)`` gives more over the same
ranges. Inputs are made on the GPU from the seed alone.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from opencaeporo_b200 import _lib, learn, synth, workload
from opencaeporo_b200.fim_jacobian import ConnGraph
from opencaeporo_b200.flash import MixtureCompBatch, copy_arrays, flash_fim_regions
from opencaeporo_b200.fluid import synthetic_fluid
from opencaeporo_b200.krpc import FlowUnitBatch

DEV = "cuda:0"
F64 = torch.float64
PSI = 145.0377          # psia per MPa
NC_ALL = (3, 6, 9, 12)  # component counts the library is built for
JAC_FROM_FLASH = ("phaseExist", "pSderExist", "pVnumCom", "S", "rho", "xi", "mu", "muP", "xiP", "rhoP", "xij",
                  "rhox", "xix", "mux", "dSec_dPri", "vfP", "vfi")


def listed():
    return [
        # a whole Newton iteration of a small sector model: launches and latency
        {"name": "newton_300", "kind": "newton", "nc": 6, "nx": 10, "ny": 10, "nz": 3, "form": "batched"},
        # the same on a mid-size model with a detailed fluid, odd in every direction
        {"name": "newton_nc9_17k", "kind": "newton", "nc": 9, "nx": 31, "ny": 29, "nz": 19, "form": "batched"},
        # the plain FP64 drop-in (the default form) on 4096 independent fresh states
        {"name": "flash_plain_4096", "kind": "fresh", "nc": 6, "n": 4096, "form": "plain", "near": False},
        # the fresh flash of a 128 x 128 x 64 block, 30 % of it near the phase envelope
        {"name": "flash_fast_1m", "kind": "fresh", "nc": 6, "n": 1 << 20, "form": "fast", "near": True},
        # the flash of one Newton iteration of the 60 x 220 x 85 model, warm-started
        {"name": "flash_warm_1122k", "kind": "warm", "nc": 6, "nx": 60, "ny": 220, "nz": 85, "form": "fast",
         "entry": "fim"},
        # an IMPEC step's flash with 9 components, ragged size
        {"name": "impec_nc9_100k", "kind": "warm", "nc": 9, "nx": 47, "ny": 43, "nz": 49, "form": "mixed",
         "entry": "impec"},
        # the FIMn formulation's flash of a Newton iteration
        {"name": "fimn_50k", "kind": "warm", "nc": 6, "nx": 41, "ny": 61, "nz": 20, "form": "batched",
         "entry": "fimn"},
        # four PVT regions of 3, 6, 9 and 12 components in one call, wide ranges of P and T
        {"name": "regions4_8k", "kind": "regions", "n": 8192, "form": "mixed"},
        # the host-buffer call of an application whose Bulk arrays live on the host
        {"name": "host_300k", "kind": "host", "nc": 6, "n": 300_000, "form": "fast"},
        # relative permeability and capillary pressure with derivatives, full model
        {"name": "krpc_1122k", "kind": "krpc", "n": 1_122_000, "tables": "swof", "deriv": True},
        # upstream choice and the Jacobian's bulk part, full model (3.3M connections)
        {"name": "jacobian_1122k", "kind": "jacobian", "nc": 6, "nx": 60, "ny": 220, "nz": 85},
        # one training step of the learned initialiser at its default batch
        {"name": "train_8192", "kind": "train", "n": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi):
    """A grid of about lo..hi cells with ragged extents."""
    n = _log_int(rng, lo, hi)
    nz = max(1, min(85, int(round(n ** (1 / 3) * rng.uniform(0.3, 1.2)))))
    nx = max(1, int(round(math.sqrt(n / nz) * rng.uniform(0.6, 1.0))))
    return {"nx": nx, "ny": max(1, n // (nx * nz)), "nz": nz}


def draw(rng):
    kind = rng.choice(("newton", "fresh", "warm", "regions", "host", "krpc", "jacobian", "train"))
    form = rng.choice(("batched", "mixed", "fast"))
    if kind == "newton":
        return {"kind": kind, "nc": rng.choice(NC_ALL), "form": rng.choice(("plain", "batched", "mixed")),
                **_grid(rng, 100, 30_000)}
    if kind == "fresh":
        if rng.random() < 0.3:
            return {"kind": kind, "nc": 6, "n": _log_int(rng, 64, 20_000), "form": "plain", "near": False}
        return {"kind": kind, "nc": 6, "n": _log_int(rng, 1000, 500_000), "form": form, "near": rng.random() < 0.6}
    if kind == "warm":
        return {"kind": kind, "nc": rng.choice(NC_ALL), "form": form, "entry": rng.choice(("fim", "impec", "fimn")),
                **_grid(rng, 1000, 200_000)}
    if kind == "regions":
        return {"kind": kind, "n": _log_int(rng, 500, 8000), "form": rng.choice(("batched", "mixed"))}
    if kind == "host":
        return {"kind": kind, "nc": 6, "n": _log_int(rng, 1000, 250_000), "form": form}
    if kind == "krpc":
        return {"kind": kind, "n": _log_int(rng, 500, 1_100_000), "tables": rng.choice(("swof", "sof3")),
                "deriv": rng.random() < 0.7}
    if kind == "jacobian":
        nc = rng.choice(NC_ALL)
        return {"kind": kind, "nc": nc, **_grid(rng, 200, 700_000 if nc <= 6 else 200_000)}
    return {"kind": kind, "n": _log_int(rng, 500, 60_000)}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uni(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, dtype=F64, device=DEV, generator=g)


@functools.lru_cache(maxsize=None)
def _fluid(nc):
    return workload.bench_fluid() if nc == 6 else synthetic_fluid(nc, 1234 + nc)


@functools.lru_cache(maxsize=None)
def _block():
    """The benchmark's 1,048,576 states of the 6-component fluid, recorded:
    (P, T, Ni, near), near marking the 30 % within 5 % of the envelope."""
    w = workload.make_workload(_fluid(6), workload.NCELL, workload.SEED, 0)
    return [torch.as_tensor(np.ascontiguousarray(a), device=DEV) for a in (w["P"], w["T"], w["Ni"].T, w["near_mask"])]


def _block_states(g, n, near):
    """The block's first n cells, or with near False the first n of its
    uniform 70 %, in a random order (restart chains differ a hundredfold
    between cells: so every seed's cells hold the same ones)."""
    P, T, Ni, mask = _block()
    cells = torch.arange(P.numel(), device=DEV) if near else torch.nonzero(~mask).reshape(-1)
    cells = cells[:n][torch.randperm(min(n, cells.numel()), device=DEV, generator=g)]
    return P[cells], T[cells], Ni[:, cells]


@functools.lru_cache(maxsize=None)
def _wide_block(nc):
    """8192 independent states over wide ranges: P 2-60 MPa, T 300-450 K,
    z ~ Dirichlet(1/2) (Gamma(1/2): half a squared normal)."""
    g, n = _gen(workload.SEED + nc), 8192
    P = _uni(g, 2.0 * PSI, 60.0 * PSI, n)
    T = _uni(g, 300.0 * 1.8 - 459.67, 450.0 * 1.8 - 459.67, n)
    gam = 0.5 * torch.randn(nc, n, dtype=F64, device=DEV, generator=g) ** 2 + 1e-30
    nt = _uni(g, 1e3, 1e4, n)
    return P, T, torch.cat([gam / gam.sum(dim=0, keepdim=True) * nt, (_uni(g, 0.5, 2.0, n) * nt)[None, :]])


def _wide_states(g, nc, n):
    """The first n states of the wide block in a random order."""
    order = torch.randperm(n, device=DEV, generator=g)
    return [t[..., order] for t in _wide_block(nc)]


class _Reservoir:
    """A block with one injector and two producers; inputs(t) are its cells'
    (P, T, Ni) at time t: a gas front spreading, pressure drawn down."""

    def __init__(self, g, nc, nx, ny, nz):
        n = nx * ny * nz
        i = torch.arange(n, device=DEV)
        x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
        self.nc, self.n = nc, n
        self.lnk = 3.0 + 2.0 * torch.randn(n, dtype=F64, device=DEV, generator=g)
        self.poro = _uni(g, 0.05, 0.35, n)
        self.noise = torch.randn(n, dtype=F64, device=DEV, generator=g)
        self.depth = 8000.0 + 2.0 * z.to(F64)
        kfac = torch.exp(0.25 * (self.lnk - 3.0))
        dist = lambda wx, wy: torch.hypot((x - wx).to(F64), (y - wy).to(F64)) / kfac  # noqa: E731
        self.d_inj = dist(2, ny // 2)
        self.d_prod = torch.minimum(dist(nx - 3, 5), dist(nx - 3, ny - 6))
        u = np.linspace(0, 1, nc)
        mk = lambda v: torch.as_tensor(v / v.sum(), device=DEV)[:, None]  # noqa: E731
        self.z_res = mk(np.interp(u, np.linspace(0, 1, 6), [0.30, 0.10, 0.12, 0.15, 0.18, 0.15]))
        self.z_inj = mk(np.interp(u, np.linspace(0, 1, 6), [0.80, 0.12, 0.05, 0.02, 0.005, 0.005]))
        self.shape = (nz, ny, nx)

    def inputs(self, t):
        P = 3000.0 + 0.35 * (self.depth - 8000.0) + 1500.0 * (1 - math.exp(-t / 6.0)) * torch.exp(-self.d_inj / 25.0) \
            - 1200.0 * (1 - math.exp(-t / 4.0)) * torch.exp(-self.d_prod / 18.0) + 3.0 * self.noise
        phi = torch.sigmoid((8.0 * t - self.d_inj) / 3.0)
        z = (1 - phi) * self.z_res + phi * self.z_inj
        pv = 1000.0 * self.poro
        T = torch.full_like(P, 160.0)
        return P, T, torch.cat([z * (pv * P / (10.73 * (T + 459.67)) * 1.2), (0.68 * pv)[None, :]])

    def connections(self):
        """7-point connections (begin, end, harmonic mean permeability)."""
        idx = torch.arange(self.n, device=DEV).reshape(self.shape)
        k = torch.exp(self.lnk).reshape(self.shape)
        b, e, a = [], [], []
        for d in (2, 1, 0):
            m = self.shape[d] - 1
            lo, hi = idx.narrow(d, 0, m), idx.narrow(d, 1, m)
            kl, kh = k.narrow(d, 0, m), k.narrow(d, 1, m)
            b.append(lo.reshape(-1)), e.append(hi.reshape(-1)), a.append((2 * kl * kh / (kl + kh)).reshape(-1))
        return torch.cat(b), torch.cat(e), torch.cat(a)


def _context(nc, form):
    m = MixtureCompBatch(_fluid(nc), 0)
    if form == "fast" and nc == 6:
        learn.Initializer.load(learn.DEFAULT_MODEL).attach(m)
    return m


def _put(st, inputs):
    for dst, src in zip((st.P, st.T, st.Ni), inputs):
        dst.copy_(src)


def _warm_state(m, res):
    """The state a Newton iteration starts from: every cell flashed at an
    earlier iterate, then the next iterate's P and Ni. Returns the state and
    the (current, saved) pairs that put its warm-start arrays back."""
    st = m.new_state(res.n)
    _put(st, res.inputs(2.0))
    m.flash_fim(st, form="plain")
    _put(st, res.inputs(2.25))
    cur = [st.out[k] for k in ("S", "phaseNum", "xij")] + [st.skip[k] for k in ("flag", "minEig", "P", "T", "z")]
    return st, [(t, t.clone()) for t in cur]


def _saturations(g, n):
    """Saturations of a flooded block: connate to swept water, a gas zone."""
    sw = 0.1 + 0.75 * _uni(g, 0.0, 1.0, n) ** 2
    sg = torch.where(_uni(g, 0.0, 1.0, n) < 0.5, (1 - sw) * _uni(g, 0.0, 0.9, n), torch.zeros_like(sw))
    return torch.stack([1 - sw - sg, sg, sw])


def _tables(kind):
    return [synth.corey_tables(501), synth.corey_tables(502, swc=0.2, nrow=17)] if kind == "swof" else \
        [synth.corey_fn_tables(501), synth.corey_fn_tables(502, swc=0.2, nrow=17)]


def _krpc_inputs(case, seed):
    g, n = _gen(seed), case["n"]
    P, S = _uni(g, 1500.0, 6000.0, n), _saturations(g, n)
    return P, S, torch.randint(0, 2, (n,), device=DEV, generator=g, dtype=torch.int32)


def _jac_inputs(case, seed):
    """Bulk arrays as the flash and KrPc leave them: an oil zone, a gas zone
    and a two-phase zone between them, mobile water everywhere."""
    g, nc = _gen(seed), case["nc"]
    res = _Reservoir(g, nc, case["nx"], case["ny"], case["nz"])
    n, ncom, ncol = res.n, nc + 1, nc + 2
    sec = 3 * ncol * ncol
    zone = res.d_inj + 0.5 * res.noise
    q = torch.quantile(zone[:: max(1, n // 100_000)], torch.tensor([0.25, 0.6], dtype=F64, device=DEV))
    gas, oil = zone < q[1], zone > q[0]
    i32 = lambda *t: torch.stack(t).to(torch.int32)  # noqa: E731
    one, zero = torch.ones_like(gas), torch.zeros_like(gas)
    sw = _uni(g, 0.1, 0.85, n)
    sg = (1 - sw) * torch.where(gas, torch.where(oil, _uni(g, 0.05, 0.9, n), 1.0), 0.0)
    S = torch.stack([1 - sw - sg, sg, sw])
    vn = i32(oil, gas, zero) * nc
    nrow = (i32(oil, gas, one) + vn).sum(dim=0)
    x = -torch.log(_uni(g, 1e-6, 1.0, 3, ncom, n))
    x[:, nc] = 0
    x = x / x.sum(dim=1, keepdim=True)
    x[2, :nc], x[2, nc] = 0, 1
    dsec = torch.empty(sec, n, dtype=F64, device=DEV)
    for r in range(3 * ncol):  # compact rows; those a bulk does not have are zero
        dsec[r * ncol:(r + 1) * ncol] = torch.where(r < nrow, 1e-3 * torch.randn(ncol, n, dtype=F64, device=DEV, generator=g), 0.0)
    part = lambda s: (s * torch.randn(3, ncom, n, dtype=F64, device=DEV, generator=g)).reshape(3 * ncom, n)  # noqa: E731
    P = res.inputs(2.0)[0]
    bulk = {"phaseExist": i32(oil, gas, one), "pSderExist": i32(oil, gas, one), "pVnumCom": vn, "S": S,
            "rho": _uni(g, 5.0, 60.0, 3, n), "xi": _uni(g, 0.2, 3.0, 3, n), "mu": _uni(g, 0.02, 1.0, 3, n),
            "muP": 1e-5 * _uni(g, 0.1, 1.0, 3, n), "xiP": 1e-5 * _uni(g, 0.1, 1.0, 3, n),
            "rhoP": 1e-4 * _uni(g, 0.1, 1.0, 3, n), "xij": x.reshape(3 * ncom, n), "rhox": part(5.0), "xix": part(0.1),
            "mux": part(0.1), "dSec_dPri": dsec, "vfP": -_uni(g, 0.01, 0.2, n), "vfi": _uni(g, 0.3, 5.0, ncom, n),
            "kr": _uni(g, 0.0, 1.0, 3, n), "Pj": P + torch.stack([torch.zeros_like(P), _uni(g, 0.0, 1.5, n),
                                                                 -_uni(g, 0.0, 4.0, n)]),
            "dKr_dS": torch.randn(9, n, dtype=F64, device=DEV, generator=g),
            "dPcj_dS": torch.randn(9, n, dtype=F64, device=DEV, generator=g),
            "v": torch.full_like(P, 1000.0), "poroP": 3e-6 * res.poro, "depth": res.depth}
    return bulk, res.connections(), n


def _jac_out(nc, n, nconn):
    mk = lambda m: torch.zeros((nc + 2) ** 2, m, dtype=F64, device=DEV)  # noqa: E731
    return {"diag": mk(n), "offEB": mk(nconn), "offBE": mk(nconn)}


def _train_inputs(case, seed):
    """A batch of normalised features and labels, and a network with Adam
    moments from earlier steps."""
    g, n, nin, nout = _gen(seed), case["n"], 8, 7
    f32 = torch.float32
    x = torch.randn(nin, n, dtype=f32, device=DEV, generator=g)
    two = (torch.rand(n, device=DEV, generator=g) < 0.3).to(f32)
    t = torch.cat([two[None, :], torch.randn(nout - 1, n, dtype=f32, device=DEV, generator=g) * two])
    p = torch.as_tensor(learn.init_params(nin, nout, seed % 65536), device=DEV)
    m1 = 1e-3 * torch.randn(p.numel(), dtype=f32, device=DEV, generator=g)
    m2 = 1e-5 * (1.0 + torch.rand(p.numel(), dtype=f32, device=DEV, generator=g))
    return x, t, two, p, m1, m2


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("newton", "warm"):
        res = _Reservoir(_gen(seed), case["nc"], case["nx"], case["ny"], case["nz"])
        s["m"] = _context(case["nc"], case["form"])
        s["st"], s["pairs"] = _warm_state(s["m"], res)
        if kind == "newton":
            s["fu"] = FlowUnitBatch([synth.corey_tables(501)], 0)
            s["kr"] = s["fu"].new_outputs(res.n)
            b, e, a = (t.cpu().numpy() for t in res.connections())
            s["graph"] = ConnGraph(res.n, b, e, a, 0)
            s["bulk"] = {k: s["st"].out[k] for k in JAC_FROM_FLASH}
            s["bulk"].update({k: s["kr"][k] for k in ("kr", "Pj", "dKr_dS", "dPcj_dS")})
            s["bulk"].update(v=torch.full_like(res.depth, 1000.0), poroP=3e-6 * res.poro, depth=res.depth)
            s["jac"] = _jac_out(case["nc"], res.n, len(b))
    elif kind == "fresh":
        s["m"] = _context(case["nc"], case["form"])
        s["st"] = s["m"].new_state(case["n"])
        _put(s["st"], _block_states(_gen(seed), case["n"], case["near"]))
    elif kind == "regions":
        g, s["regions"] = _gen(seed), []
        for nc in NC_ALL:
            m = _context(nc, case["form"])
            st = m.new_state(case["n"])
            _put(st, _wide_states(g, nc, case["n"]))
            s["regions"].append((m, st))
    elif kind == "host":
        s["m"] = _context(case["nc"], case["form"])
        s["hs"] = s["m"].new_host_state(case["n"])
        for k, v in zip(("P", "T", "Ni"), _block_states(_gen(seed), case["n"], True)):
            s["hs"][k].copy_(v)
    elif kind == "krpc":
        s["P"], s["S"], s["satnum"] = _krpc_inputs(case, seed)
        s["fu"] = FlowUnitBatch(_tables(case["tables"]), 0)
        s["out"] = s["fu"].new_outputs(case["n"], case["deriv"])
    elif kind == "jacobian":
        s["bulk"], (b, e, a), n = _jac_inputs(case, seed)
        s["graph"] = ConnGraph(n, b.cpu().numpy(), e.cpu().numpy(), a.cpu().numpy(), 0)
        s["jac"] = _jac_out(case["nc"], n, b.numel())
    else:
        s["x"], s["t"], s["w"], s["p"], s["m1"], s["m2"] = _train_inputs(case, seed)
        s["g"], s["loss"], s["step"] = torch.zeros_like(s["p"]), torch.zeros(2, device=DEV), 100
    return s


# ---------------------------------------------------------------------- run
def _flash_again(s):
    """One Newton iteration's flash, from the same warm-start arrays each time."""
    case, m, st = s["case"], s["m"], s["st"]
    copy_arrays(s["pairs"])
    entry = case.get("entry", "fim")
    f = {"fim": m.flash_fim, "impec": m.flash_impec, "fimn": m.flash_fimn}[entry]
    f(st, form=case["form"], diagnostics=False)
    # what the call does not write stays out
    if entry == "impec":
        return {k: st.out[k] for k in _lib.IMPEC_OUT_FIELDS if k not in _lib.OPTIONAL_OUT}
    drop = {"ePEC", "ftype", "iters", "status"} | (set() if entry == "fimn" else {"nj"})
    return {k: v for k, v in st.out.items() if k not in drop}


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "warm":
        return _flash_again(s)
    if kind == "newton":
        out = _flash_again(s)
        st, g = s["st"], s["graph"]
        s["fu"].cal_krpc(st.P, st.out["S"], None, out=s["kr"])
        up, rho = g.upwind(s["bulk"])
        g.jacobian(case["nc"], 1.0, s["bulk"], up, rho, out=s["jac"])
        return {"flash": out, "krpc": s["kr"], "up": up, "rho": rho, "jac": s["jac"]}
    if kind == "fresh":
        s["st"].skip["flag"].zero_()  # new bulks: no cached stability result
        s["m"].flash_fim(s["st"], form=case["form"], fresh=True)
        return s["st"].out
    if kind == "regions":
        for _, st in s["regions"]:
            st.skip["flag"].zero_()
        flash_fim_regions(s["regions"], form=case["form"], fresh=True, diagnostics=False)
        keep = ("phaseNum", "S", "vf", "vfP", "vfi", "rho", "xi", "mu", "xij", "dSec_dPri")
        return [{k: st.out[k] for k in keep} for _, st in s["regions"]]
    if kind == "host":
        s["hs"]["out"]["phaseNum"].zero_()
        s["hs"]["skip"]["flag"].zero_()
        s["m"].flash_fim_host(s["hs"], form=case["form"])
        return s["hs"]["out"]
    if kind == "krpc":
        return s["fu"].cal_krpc(s["P"], s["S"], s["satnum"], out=s["out"], deriv=case["deriv"])
    if kind == "jacobian":
        up, rho = s["graph"].upwind(s["bulk"])
        return {"up": up, "rho": rho, **s["graph"].jacobian(case["nc"], 1.0, s["bulk"], up, rho, out=s["jac"])}
    learn.grad(s["p"], s["x"], s["t"], s["w"], 1.0, s["g"], s["loss"])
    s["step"] += 1
    _lib.check(_lib.lib().ocpf_mlp_adam(s["p"].data_ptr(), s["g"].data_ptr(), s["m1"].data_ptr(), s["m2"].data_ptr(),
                                        s["step"], 1e-3, None), "ocpf_mlp_adam")
    return {"params": s["p"], "m": s["m1"], "v": s["m2"], "loss": s["loss"]}


# --------------------------------------------------------------------- work
def _bytes_of(shapes):
    size = {"f64": 8, "u32": 4, "i32": 4, "u16": 2, "u8": 1}
    return sum(nf * size[dt] for nf, dt in shapes.values())


def _flash_work(nc, n, evals):
    """Bytes of one flash (inputs and outputs once; the derivative rows of a
    one-phase or two-phase cell are about half of dSec_dPri's space) and the
    arithmetic of `evals` fugacity evaluations per cell."""
    out = _lib.out_shapes(nc)
    rows = out["dSec_dPri"][0] * 8 // 2
    b = _bytes_of(_lib.in_shapes(nc)) + _bytes_of(out) - rows + 2 * _bytes_of(_lib.skip_shapes(nc))
    return n * b, n * evals * (2 * nc * nc + 10 * nc + 40)


def _jac_work(nc, n, nconn):
    ncom, ncol = nc + 1, nc + 2
    bulk = 8 * (3 * 9 + 12 * ncom + (nc + 3) * ncol + ncom + 18 + 6)
    conn = 20 + 2 * 36 + 2 * 8 * ncol * ncol
    return n * (bulk + 8 * ncol * ncol) + nconn * conn, nconn * 4.0 * ncom * ncol * (nc + 3)


def _size(case):
    if "n" in case:
        return case["n"], 0
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return nx * ny * nz, (nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1)


def work(case):
    kind = case["kind"]
    n, nconn = _size(case)
    if kind == "krpc":
        b, f = n * (36 + 72 + (144 if case["deriv"] else 0)), 60.0 * n
    elif kind == "train":
        b, f = n * 64 + 6288 * 32, 6.0 * n * (16 * 64 + 64 * 64 + 64 * 16)
    elif kind == "jacobian":
        b, f = _jac_work(case["nc"], n, nconn)
    elif kind == "regions":
        w = [_flash_work(nc, n, 100) for nc in NC_ALL]
        b, f = sum(v[0] for v in w), sum(v[1] for v in w)
    else:
        b, f = _flash_work(case["nc"], n, 60 if kind in ("fresh", "host") else 10)
        if kind == "newton":
            jb, jf = _jac_work(case["nc"], n, nconn)
            b, f = b + jb + 252 * n, f + jf + 60 * n
    return {"bytes": float(b), "flops": float(f)}


# -------------------------------------------------------------------- exact
def _lookup(tab, val):
    """Linear interpolation in a table's first column with the end rows'
    values and no slope outside it: (values, slopes) of the other columns."""
    t = torch.as_tensor(np.ascontiguousarray(tab), dtype=F64, device=DEV)
    k = (torch.searchsorted(t[:, 0].contiguous(), val, right=True) - 1).clamp(0, len(t) - 2)
    slope = (t[k + 1, 1:] - t[k, 1:]) / (t[k + 1, :1] - t[k, :1])
    v = t[k, 1:] + slope * (val - t[k, 0])[:, None]
    lo, hi = (val < t[0, 0])[:, None], (val >= t[-1, 0])[:, None]
    zero = torch.zeros_like(v)
    return torch.where(lo, t[0, 1:], torch.where(hi, t[-1, 1:], v)).T, torch.where(lo | hi, zero, slope).T


def _exact_krpc(case, seed):
    P, S, satnum = _krpc_inputs(case, seed)
    n = case["n"]
    kr, pc = torch.zeros(3, n, dtype=F64, device=DEV), torch.zeros(3, n, dtype=F64, device=DEV)
    dk, dp = torch.zeros(9, n, dtype=F64, device=DEV), torch.zeros(9, n, dtype=F64, device=DEV)
    for r, tabs in enumerate(_tables(case["tables"])):
        m = satnum == r
        w, dw = _lookup(tabs[0], S[2, m])
        g, dg = _lookup(tabs[1], S[1, m])
        krw, krg, dkrw, dkrg = w[0], g[0], dw[0], dg[0]
        pc[1, m], pc[2, m], dp[4, m], dp[8, m] = g[-1], -w[-1], dg[-1], -dw[-1]
        kr[1, m], kr[2, m], dk[4, m], dk[8, m] = krg, krw, dkrg, dkrw
        if case["tables"] == "swof":
            krow, krog, km = w[1], g[1], float(tabs[0][0, 2])
        else:
            o, do = _lookup(tabs[2], S[0, m])
            krow, krog, km = o[0], o[1], float(tabs[2][-1, 1])
        a1, a2 = krow / km + krw, krog / km + krg
        kro = km * (a1 * a2 - (krw + krg))
        if case["tables"] == "swof":
            neg = kro < 0
            dk[2, m] = torch.where(neg, 0.0, km * ((dw[1] / km + dkrw) * a2 - dkrw))
            dk[1, m] = torch.where(neg, 0.0, km * (a1 * (dg[1] / km + dkrg) - dkrg))
        elif case["deriv"]:
            neg = kro < 0
            dk[0, m] = torch.where(neg, 0.0, do[0] * a2 + do[1] * a1)
        else:  # without derivatives the reference weights krog and krow by saturation
            swc = float(tabs[0][0, 0])
            den = S[1, m] + S[2, m] - swc
            kro = torch.where(den <= 1e-8, km, (S[1, m] * krog + (S[2, m] - swc) * krow) / den)
        kr[0, m] = kro.clamp_min(0.0) if case["tables"] == "swof" or case["deriv"] else kro
    out = {"kr": kr, "Pc": pc, "Pj": P + pc}
    if case["deriv"]:
        out.update(dKr_dS=dk, dPcj_dS=dp)
    return out


def _exact_jacobian(case, seed):
    """The assembly as dense products: flux derivatives of both ends in the
    full set of secondary variables (3 saturations, nc mole fractions of each
    hydrocarbon phase), times the full dSec_dPri."""
    bulk, (b, e, area), n = _jac_inputs(case, seed)
    nc = case["nc"]
    ncom, ncol, grav, darcy = nc + 1, nc + 2, 0.00694444, 5.61458 * 1.12712e-3
    ex = bulk["phaseExist"] > 0
    # rows of the compact dSec_dPri in the full set's order (-1: none)
    sd, nsat = ex.long(), ex.long().sum(dim=0)
    sat = torch.where(ex, torch.cumsum(sd, dim=0) - 1, -1)
    k = torch.arange(nc, device=DEV)[:, None]
    xo = torch.where(ex[0], nsat + k, -1)
    xg = torch.where(ex[1], nsat + sd[0] * nc + k, -1)
    rows = torch.cat([sat, xo, xg])
    P3 = lambda name: bulk[name].reshape(3, -1, n)  # noqa: E731
    up = torch.empty(3, b.numel(), dtype=torch.int64, device=DEV)
    rho = torch.empty(3, b.numel(), dtype=F64, device=DEV)
    dd = bulk["depth"][b] - bulk["depth"][e]
    for j in range(3):
        xb, xe = ex[j, b], ex[j, e]
        rb, re, sb, se = bulk["rho"][j, b], bulk["rho"][j, e], bulk["S"][j, b], bulk["S"][j, e]
        r = torch.where(xb & xe, (rb * sb + re * se) / (sb + se), torch.where(xb, rb, torch.where(xe, re, 0.0)))
        dphi = bulk["Pj"][j, b] - grav * r * bulk["depth"][b] - (bulk["Pj"][j, e] - grav * r * bulk["depth"][e])
        up[j], rho[j] = torch.where((dphi < 0) & (xb | xe), e, b), r
    out = _jac_out(nc, n, b.numel())
    diag = out["diag"].reshape(ncol, ncol, n)
    for i in range(1, ncol):
        diag[i, i] = 1
    diag[0, 0] = bulk["v"] * bulk["poroP"] - bulk["vfP"]
    diag[0, 1:] = -bulk["vfi"]
    for c0 in range(0, b.numel(), 1 << 17):
        c = slice(c0, min(b.numel(), c0 + (1 << 17)))
        m = c.stop - c.start
        B, E = b[c], e[c]
        Fp = torch.zeros(2, ncom, m, dtype=F64, device=DEV)                 # dF/dP of (begin, end)
        Fs = torch.zeros(2, ncom, 3 + 2 * nc, m, dtype=F64, device=DEV)     # dF/d(secondary)
        akd, dg = darcy * area[c], grav * dd[c]
        for j in range(3):
            u = up[j, c]
            at_b, xb, xe = u == B, ex[j, B], ex[j, E]
            live = torch.where(at_b, xb, xe).to(F64)
            at = [at_b.to(F64), 1.0 - at_b.to(F64)]
            q = lambda name: bulk[name][j, u]  # noqa: E731
            both = (xb & xe).to(F64)
            dP = bulk["Pj"][j, B] - bulk["Pj"][j, E] - rho[j, c] * dg
            x, xi, mu, kr = P3("xij")[j][:, u], q("xi"), q("mu"), q("kr")
            tr = live * akd * kr / mu
            tx = x * xi * tr
            common = x * tr * q("xiP") * dP - tx * q("muP") / mu * dP
            for end, sign, N in ((0, 1.0, B), (1, -1.0, E)):
                own = (at[end] * (common - (1 - both) * tx * q("rhoP") * dg))
                Fp[end] += sign * tx + own - 0.5 * both * tx * bulk["rhoP"][j, N] * dg
                for j1 in range(3):
                    f = 3 * j + j1
                    Fs[end, :, j1] += sign * tx * bulk["dPcj_dS"][f, N] \
                        + live * akd * x * xi / mu * at[end] * bulk["dKr_dS"][f, u] * dP
                if j < 2:
                    o = 3 + j * nc
                    for kk in range(nc):
                        rx = P3("rhox")[j][kk]
                        v = -tx * (both * 0.5 * rx[N] + (1 - both) * at[end] * rx[u]) * dg
                        v += at[end] * (x * tr * P3("xix")[j][kk, u] - tx * P3("mux")[j][kk, u] / mu) * dP
                        Fs[end, :, o + kk] += v
                        Fs[end, kk, o + kk] += at[end] * xi * tr * dP
        for end, N, dst, sign in ((0, B, "offEB", -1.0), (1, E, "offBE", 1.0)):
            rr = rows[:, N]
            sec = torch.gather(bulk["dSec_dPri"].reshape(-1, ncol, n)[:, :, N].permute(1, 0, 2), 1,
                               rr.clamp_min(0).expand(ncol, -1, -1)) * (rr >= 0)
            blk = torch.einsum("isc,psc->ipc", Fs[end], sec)
            blk[:, 0] += Fp[end]
            out[dst].reshape(ncol, ncol, -1)[1:, :, c] = sign * blk
            diag[1:].index_add_(2, N, -sign * blk)
    return {"up": None, "rho": rho, **out}


def _exact_train(case, seed):
    x, t, w, p, m1, m2 = (v.double() for v in _train_inputs(case, seed))
    n, nout = case["n"], t.shape[0]
    p = p.clone().requires_grad_(True)
    o = 0
    sizes = (64 * 16, 64, 64 * 64, 64, 16 * 64, 16)
    part = [p[sum(sizes[:i]):sum(sizes[:i + 1])] for i in range(6)]
    silu = torch.nn.functional.silu
    X = torch.cat([x, torch.zeros(16 - x.shape[0], n, dtype=F64, device=DEV)])
    h = silu(part[0].reshape(64, 16) @ X + part[1][:, None])
    h = silu(part[2].reshape(64, 64) @ h + part[3][:, None])
    o = part[4].reshape(16, 64) @ h + part[5][:, None]
    bce = (torch.nn.functional.softplus(o[0]) - t[0] * o[0]).sum()
    mse = (w * ((o[1:nout] - t[1:]) ** 2).sum(dim=0)).sum() / (nout - 1)
    gr, = torch.autograd.grad((bce + mse) / n, p)
    a, c = 0.9 * m1 + 0.1 * gr, 0.999 * m2 + 0.001 * gr * gr
    new = p.detach() - 1e-3 * (a / (1 - 0.9 ** 101)) / (torch.sqrt(c / (1 - 0.999 ** 101)) + 1e-8)
    return {"params": new, "m": a, "v": c, "loss": torch.stack([bce, mse]).detach()}


def exact(case, seed):
    """The flash kinds have none: their iterations in plain array operations
    over a block take minutes."""
    f = {"krpc": _exact_krpc, "jacobian": _exact_jacobian, "train": _exact_train}.get(case["kind"])
    return f(case, seed) if f else None
