"""The work that a user of relxill_gb300 has it do, as cases that can be timed one by one.

Every case goes through the package's public entry points, in one of four ways:

* ``call``   one local-model call (``relxill_gb300.relxilllp(energy, params)`` and its siblings), the
  way XSPEC, ISIS and a simple fit evaluate a spectrum: host arrays in, host array out;
* ``host``   ``relxill_gb300.eval_batch``, many parameter sets with their own grids in host arrays;
* ``device`` ``relx_eval_batch_device`` of the C ABI, the same with buffers on the GPU, on the
  caller's stream (a sampler that keeps its walkers there);
* ``serve``  ``relxill_gb300.Server``, single requests from many walkers.

Parameters are drawn over the ranges that fits move in (the ranges of ``bench.py`` and of the public
model list), grids are logarithmic with 300 to 5000 bins, tables are the synthetic full-size ones.
The output cache of the local-model calls is off: a fit that moves its parameters misses it.
"""
import ctypes
import math
import os

import numpy as np
import torch

import relxill_gb300 as R

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RELATIVISTIC = ("relxill", "relxilllp", "relxillCp", "relxilllpCp")
LINES = ("relline", "relline_lp")
CONVS = ("relconv", "relconv_lp")
CP = ("xillverCp", "relxillCp", "relxilllpCp")


def _case(name, how, model, sets, bins, emin=0.3, emax=80.0, returnrad=0, gradient=0, limb=0):
    """bins: the mean number of bins of a set's grid (a batch's grids spread from a third to twice
    of it); returnrad: $switch_returnrad of the lamp-post models; gradient: the ionisation-gradient
    switch (2: alpha disk, 25 zones); limb: the limb-darkening law of the line models."""
    return {"name": name, "how": how, "model": model, "sets": sets, "bins": bins, "emin": emin, "emax": emax,
            "returnrad": returnrad, "gradient": gradient, "limb": limb}


def listed():
    return [
        # the smallest call: the non-relativistic reflection model on a CCD-like grid
        _case("xillver call", "call", "xillver", 1, 400),
        # a single broad line, the classical relline fit (3000 bins, 0.1-20 keV)
        _case("relline call", "call", "relline", 1, 3000, emin=0.1, emax=20.0),
        # one spectrum of the lamp-post model, what an XSPEC fit does thousands of times
        _case("relxilllp call", "call", "relxilllp", 1, 2847),
        # the same with the model's default switches (returning radiation) and the nthcomp continuum
        _case("relxilllpCp call", "call", "relxilllpCp", 1, 1201, returnrad=1),
        # a user's continuum blurred for a few spectra at once, host arrays
        _case("relconv host 11", "host", "relconv", 11, 1000, emin=0.1, emax=100.0),
        # walkers of an ensemble sampler
        _case("relxill device 64", "device", "relxill", 64, 1500),
        # lines of many epochs or models with a limb law and returning radiation
        _case("relline_lp device 333", "device", "relline_lp", 333, 900, emin=0.5, emax=12.0, returnrad=1, limb=1),
        # the alpha-disk ionisation gradient: 25 zones per set
        _case("relxilllp gradient device 500", "device", "relxilllp", 500, 1200, gradient=2),
        # the nthcomp flavour with its default switches, a nested sampler's batch
        _case("relxilllpCp device 1000", "device", "relxilllpCp", 1000, 2000, returnrad=1),
        # 256 walkers, one request each, through the serving engine
        _case("relxilllp serve 256", "serve", "relxilllp", 256, 2650),
        # a parameter scan from host arrays, default switches
        _case("relxilllp host 2048", "host", "relxilllp", 2048, 2000, returnrad=1),
        # the headline batch: 4096 sets of 300-5000 bins, resident on the GPU
        _case("relxilllp device 4096", "device", "relxilllp", 4096, 2650),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    how = rng.choice(("call", "call", "host", "device", "device", "device", "serve"))
    bins = _log_int(rng, 300, 2600)
    emin, emax = rng.choice(((0.3, 80.0), (0.1, 20.0), (0.5, 12.0), (0.2, 150.0), (3.0, 79.0)))
    if how == "call":
        model, sets, bins = rng.choice(sorted(R.MODELS)), 1, _log_int(rng, 200, 5000)
    elif how == "serve":
        model, sets = rng.choice(("relxilllp", "relxill")), _log_int(rng, 8, 256)
    else:
        model = rng.choice(("relline", "relconv", "relxill", "relxilllp", "relxilllp", "relxilllp", "relline_lp",
                            "relconv_lp", "xillver", "relxillCp", "relxilllpCp"))
        top = 2048 if how == "host" else 4096
        top = 1000 if model in CP else 1000 if model in LINES else top
        sets = _log_int(rng, 2, top)
    returnrad = rng.choice((0, 1)) if "lp" in model else 0
    gradient = 2 if model == "relxilllp" and how != "serve" and rng.random() < 0.2 else 0
    sets = min(sets, 700 if gradient else 2048 if returnrad else sets)
    c = _case("", how, model, sets, bins, emin, emax, returnrad=returnrad, gradient=gradient,
              limb=rng.choice((0, 0, 1, 2)) if model in LINES + CONVS else 0)
    del c["name"]
    return c


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
_ready = {}


def _tables():
    from relxill_gb300 import synth_tables

    d = os.path.join(ROOT, "_tables", "full")
    written = os.path.join(d, ".complete_full_1234")  # the tables are written once per checkout
    if not os.path.exists(written):
        synth_tables.ensure_tables(d, xill="full")
        with open(written, "w") as f:
            f.write("ok\n")
    return d


def _program():
    """What a program sets up once: the tables, its stream, the output cache off."""
    if not _ready:
        d = _tables()
        os.environ["RELXILL_TABLE_PATH"] = d
        R.init(d)
        R.output_cache_config(0)
        _ready["stream"] = torch.cuda.Stream()
    return _ready


def _server():
    if "server" not in _program():
        _ready["server"] = R.Server(hbm_budget_bytes=4 << 30, max_batch=1024)
    return _ready["server"]


def _params(case, seed):
    rng = np.random.default_rng([seed, 1])
    n, model = case["sets"], case["model"]
    names = [k for k, _ in R.PARAMS[model]]
    p = np.tile(R.default_params(model), (n, 1))

    def put(name, v):
        if name in names:
            p[:, names.index(name)] = v

    put("a", rng.uniform(0.0, 0.998, n))
    put("Incl", rng.uniform(5.0, 85.0, n))
    put("h", rng.uniform(3.0, 100.0, n))
    put("Index1", rng.uniform(2.0, 5.0, n))
    put("Index2", rng.uniform(2.0, 4.0, n))
    put("Rbr", rng.uniform(6.0, 40.0, n))
    put("gamma", rng.uniform(1.4, 2.8, n))
    put("logxi", rng.uniform(0.0, 4.5, n))
    put("Afe", rng.choice([1.0, 2.3], n))
    put("Ecut", rng.uniform(50.0, 500.0, n))
    put("kTe", rng.uniform(20.0, 300.0, n))
    put("logN", rng.uniform(15.0, 19.0, n))
    put("lineE", rng.uniform(6.3, 7.0, n))
    put("z", rng.choice([0.0, 0.03], n))
    put("refl_frac", rng.uniform(0.3, 3.0, n))
    put("limb", case["limb"])
    put("switch_returnrad", case["returnrad"])
    return p


def _grids(case):
    """The instruments' grids: they belong to the case and stay when the parameters move."""
    n, bins = case["sets"], case["bins"]
    rng = np.random.default_rng([n, bins, 2])
    nb = np.full(n, bins) if n == 1 else rng.integers(max(50, bins // 3), max(51, 2 * bins - bins // 3), n)
    lo, hi = math.log(case["emin"]), math.log(case["emax"])
    return [np.exp(np.linspace(lo, hi, int(k) + 1)) for k in nb]


def _continua(case, grids, seed):
    """The spectra that a convolution model blurs: a power law with a narrow iron line."""
    rng = np.random.default_rng([seed, 3])
    out = []
    for e in grids:
        m, w = 0.5 * (e[1:] + e[:-1]), np.diff(e)
        gam, norm = rng.uniform(1.5, 2.5), rng.uniform(0.05, 0.5)
        out.append(w * (m ** -gam + norm * np.exp(-0.5 * ((m - 6.4) / 0.05) ** 2)))
    return out


def _host_inputs(case, seed):
    params, grids = _params(case, seed), _grids(case)
    flux = _continua(case, grids, seed) if case["model"] in CONVS else None
    return params, grids, flux


def prepare(case, seed):
    prog = _program()
    params, grids, flux = _host_inputs(case, seed)
    n = case["sets"]
    s = {"how": case["how"], "model": case["model"], "n": n, "params": params, "grids": grids, "flux": flux}
    gradient = case["gradient"] if case["model"] == "relxilllp" else 0
    s["igt"] = np.full(n, gradient, dtype=np.int32) if gradient else None
    if s["how"] == "serve":
        s["server"] = _server()
        s["out"] = [np.zeros(len(e) - 1) for e in grids]
    if s["how"] == "device":
        edges, offs = R.pack_grids(grids)
        s["offs"] = offs
        s["d_params"], s["d_edges"], s["d_offs"] = (torch.from_numpy(x).cuda() for x in (params, edges, offs))
        s["d_flux"] = torch.zeros(int(offs[-1]) - n, dtype=torch.float64, device="cuda")
        s["d_status"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        s["d_in"] = None
        if flux is not None:  # the device call takes input spectra in the layout of the edges
            spread = np.zeros(int(offs[-1]))
            for i, f in enumerate(flux):
                spread[offs[i]:offs[i] + len(f)] = f
            s["d_in"] = torch.from_numpy(spread).cuda()
        s["d_igt"] = torch.from_numpy(s["igt"]).cuda() if gradient else None
        s["d_igi"] = torch.zeros(n, dtype=torch.float64, device="cuda") if gradient else None
        s["stream"] = prog["stream"]
    return s


# ----------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------
def _at(t):
    return None if t is None else t.data_ptr()


def _run_device(s):
    igt = s["igt"].ctypes.data_as(ctypes.POINTER(ctypes.c_int)) if s["igt"] is not None else None
    st = R.lib().relx_eval_batch_device(
        R.MODELS[s["model"]], s["n"], _at(s["d_params"]), _at(s["d_edges"]), _at(s["d_offs"]),
        s["offs"].ctypes.data_as(ctypes.POINTER(ctypes.c_int64)), _at(s["d_in"]), _at(s["d_flux"]), _at(s["d_status"]),
        _at(s["d_igt"]), igt, _at(s["d_igi"]), s["stream"].cuda_stream)
    if st:
        raise RuntimeError(f"relx_eval_batch_device: {st} {R.last_error()}")
    return {"flux": s["d_flux"], "status": s["d_status"]}


def _run_serve(s):
    srv, left = s["server"], {}
    for i in range(s["n"]):
        left[srv.submit(s["model"], s["params"][i], s["grids"][i], s["out"][i])] = i
    status = np.zeros(s["n"], dtype=np.int32)
    while left:
        for rid, st, _ in srv.poll():
            status[left.pop(rid)] = st
    return {"flux": np.concatenate(s["out"]), "status": status}


def run(s):
    if s["how"] == "call":
        args = (s["grids"][0], s["params"][0]) + ((s["flux"][0],) if s["flux"] is not None else ())
        return {"flux": getattr(R, s["model"])(*args)}
    if s["how"] == "host":
        flux, status = R.eval_batch(s["model"], s["params"], s["grids"], s["flux"], ion_grad_type=s["igt"])
        # the sets' fluxes are consecutive views of one array
        return {"flux": flux[0].base, "status": status}
    return _run_serve(s) if s["how"] == "serve" else _run_device(s)


# ----------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------
def work(case):
    """bytes: parameters, grids and fluxes, and the table rows that the sets reach, each row once.
    flops: the integrand of the line profile (25 per evaluation; on average 1.5 evaluations of both
    branches per pair of a radius and a bin it reaches), the products of the convolution over the
    zones' profile windows and the weighted sum of the table rows."""
    n, model, bins = case["sets"], case["model"], case["bins"]
    npar = len(R.PARAMS[model])
    io = n * 8.0 * (npar + 2 * bins + 1 + (bins if model in CONVS else 0))
    zones = 25 if case["gradient"] else 10 if "lp" in model and model in RELATIVISTIC else 1
    per_fold = bins / math.log(case["emax"] / case["emin"]) if model in LINES else 4096 / math.log(2000 / 0.00035)
    table = flops = 0.0
    if model not in ("xillver", "xillverCp"):
        flops += n * 1000 * 0.42 * per_fold * 1.5 * 2 * 25
        table += min(48.9e6, n * 4 * 64e3)
    if model in RELATIVISTIC + CONVS:
        out = 263 * math.log(case["emax"] / case["emin"])
        flops += n * 2 * out * (700 if zones == 1 else 200 * zones)
    if model in RELATIVISTIC:
        rows = 10 * (24 if model in CP else 12) * (2 if case["gradient"] else 1)
        flops += n * 2 * rows * 2520 * zones * (0.3 if zones > 10 else 0.7)
        table += min((58e6 if model in CP else 838e6), n * rows * 2520 * 4)
    elif model in ("xillver", "xillverCp"):
        flops += n * 2 * 32 * 3000
        table += min((69e6 if model in CP else 998e6), n * 32 * 3000 * 4)
    return {"bytes": io + table, "flops": flops}


# ----------------------------------------------------------------------------
# the same numbers in 64 bits
# ----------------------------------------------------------------------------
def exact(case, seed):
    """The models' definition in numpy, FP64: line profiles (broken power law and lamp post, limb
    laws), relconv, relxill and relxilllp without gradient, xillver; up to 64 sets.  None for the
    nthcomp continuum, returning radiation and the ionisation gradient, and for larger batches."""
    model = case["model"]
    if model in CP or case["returnrad"] or case["gradient"] or case["sets"] > 64:
        return None
    params, grids, flux = _host_inputs(case, seed)
    T = _Exact(_tables())
    out = [T.model(model, params[i], grids[i], None if flux is None else flux[i]) for i in range(case["sets"])]
    got = {"flux": np.concatenate(out)}
    return got if case["how"] == "call" else {**got, "status": None}


def _hdus(path):
    """(name, rows, {column: dtype and repeat}, data offset, row bytes) of a FITS file's binary tables."""
    kinds = {"E": ">f4", "D": ">f8", "J": ">i4", "I": ">i2", "K": ">i8"}
    out, pos = [], 0
    with open(path, "rb") as f:
        size = os.path.getsize(path)
        while pos < size:
            f.seek(pos)
            cards = {}
            while True:
                block = f.read(2880).decode("latin1")
                for k in range(0, 2880, 80):
                    c = block[k:k + 80]
                    if c[8:10] == "= ":
                        v = c[10:].strip()
                        cards[c[:8].strip()] = v[1:v.index("'", 1)].strip() if v[0] == "'" else v.split("/")[0].strip()
                    if c.startswith("END "):
                        break
                else:
                    continue
                break
            data = f.tell()
            cols = []
            for k in range(1, int(cards.get("TFIELDS", 0)) + 1):
                form = cards[f"TFORM{k}"]
                rep = int(form[:-1] or 1)
                dt = f"S{rep}" if form[-1] == "A" else (kinds[form[-1]], (rep,))
                cols.append((cards[f"TTYPE{k}"], dt))
            n = 1 if int(cards["NAXIS"]) else 0
            for k in range(1, int(cards["NAXIS"]) + 1):
                n *= int(cards[f"NAXIS{k}"])
            rows = int(cards.get("NAXIS2", 0))
            out.append((cards.get("EXTNAME", ""), rows, np.dtype(cols) if cols else None, data))
            pos = data + (n + 2879) // 2880 * 2880
    return out


def _rows(path, hdu):
    return np.memmap(path, dtype=hdu[2], mode="r", offset=hdu[3], shape=(hdu[1],))


def _last_le(arr, v):
    """The last index k of an ascending array with arr[k] <= v, within [0, len - 2]."""
    return np.clip(np.searchsorted(arr, v, side="right") - 1, 0, len(arr) - 2)


def _rebin(en, e0, f0):
    """The spectrum f0 on the grid e0, on the grid en (constant within a bin)."""
    cum = np.concatenate([[0.0], np.cumsum(f0)])
    return np.diff(np.interp(en, e0, cum))


class _Exact:
    NR = 1000
    H = 5e-3

    def __init__(self, d):
        self.d = d
        self.rel = os.path.join(d, "rel_table_v0.5a.fits")
        self.rel_h = _hdus(self.rel)
        by = {h[0]: h for h in self.rel_h}
        self.rel_a = _rows(self.rel, by["a"])["a"].astype("f4").ravel()
        self.rel_mu = _rows(self.rel, by["mu0"])["mu0"].astype("f4").ravel()
        self.conv = np.exp(np.linspace(0, 1, 4097) * (math.log(2000.0) - math.log(0.00035)) + math.log(0.00035))

    # ---- radii, transfer functions, emissivity
    @staticmethod
    def _factor(arr, v):
        """Bracket and interpolation factor; parameters meet the tables in the tables' own type."""
        k = int(_last_le(arr, np.float32(v)))
        return k, float((np.float32(v) - arr[k]) / (arr[k + 1] - arr[k]))

    @staticmethod
    def _rms(a):
        z1 = 1 + (1 - a * a) ** (1 / 3) * ((1 + a) ** (1 / 3) + (1 - a) ** (1 / 3))
        z2 = math.sqrt(3 * a * a + z1 * z1)
        return 3 + z2 - math.copysign(1, a) * math.sqrt((3 - z1) * (3 + z1 + 2 * z2))

    def system(self, q):
        ia, fa = self._factor(self.rel_a, q["a"])
        im, fm = self._factor(self.rel_mu, math.cos(q["incl"]))
        nm = len(self.rel_mu)
        t = [_rows(self.rel, self.rel_h[3 + i * nm + m]) for m in (im, im + 1) for i in (ia, ia + 1)]
        w = [(1 - fa) * (1 - fm), fa * (1 - fm), (1 - fa) * fm, fa * fm]

        def plane(col):
            return sum(wi * ti[col].astype("f8") for wi, ti in zip(w, t))

        r = ((1 - fa) * t[0]["r"].astype("f8") + fa * t[1]["r"].astype("f8")).ravel()
        if r[-1] > q["rms"] and (r[-1] - q["rms"]) / r[-1] < 1e-3:
            r[-1] = q["rms"]
        top = int(np.clip(np.searchsorted(-r, -q["rout"], side="right") - 1, 0, len(r) - 2))
        if r[top] < 1000 < r[top] * 1.01:
            r[top] = 1000.0
        u = np.arange(self.NR) * (1 / math.sqrt(q["rin"]) - 1 / math.sqrt(q["rout"])) / (self.NR - 1)
        re = (1 / (u + 1 / math.sqrt(q["rout"]))) ** 2
        k = np.clip(np.searchsorted(-r, -re, side="left") - 1, 0, len(r) - 2)
        f = ((re - r[k + 1]) / (r[k] - r[k + 1]))[:, None]
        S = {"re": re}
        for name, cols in (("g", ("gmin", "gmax")), ("trf", ("trff1", "trff2")), ("mu", ("cosne1", "cosne2"))):
            S[name] = [f * v[k] + (1 - f) * v[k + 1] for v in (plane(c).reshape(len(r), -1) for c in cols)]
        S["gmin"], S["gmax"] = (v.ravel() for v in S.pop("g"))
        dr = np.empty(self.NR)
        dr[1:-1], dr[0], dr[-1] = 0.5 * (re[:-2] - re[2:]), 0.5 * (re[0] - re[1]), 0.5 * (re[-2] - re[-1])
        S["wt"] = re * dr * math.pi / 2
        if q["emis"] == "bkn":
            e = (re / q["rbr"]) ** -np.where(re > q["rbr"], q["i2"], q["i1"])
            S["emis"] = e / np.sum(e * 4 * S["wt"])
        else:
            self.lamp_post(q, S)
        return S

    def lamp_post(self, q, S):
        path = os.path.join(self.d, "rel_lp_table_v0.5b.fits")
        h = next(x for x in _hdus(path) if x[0] == "I_h")
        t = _rows(path, h)
        a = t["a"].astype("f4").ravel()
        ia, fa = self._factor(a, q["a"])
        rad = (1 - fa) * t["r"][ia].astype("f8") + fa * t["r"][ia + 1].astype("f8")

        def column(name):
            v = 0.0
            for i, w in ((ia, 1 - fa), (ia + 1, fa)):
                k, f = self._factor(t["hgrid"][i].astype("f4"), q["h"])
                lo, hi = (np.abs(t[f"{name}{n}"][i].astype("f8")) for n in (k + 1, k + 2))
                v = v + w * ((1 - f) * lo + f * hi)
            return v

        inten, de = column("h"), column("del")
        re = S["re"]
        k = _last_le(rad, re)
        lin = (re - rad[k]) / (rad[k + 1] - rad[k])
        log = np.log(re / rad[k]) / np.log(rad[k + 1] / rad[k])
        f = np.where(de[k] / math.pi * 180 <= 75, lin, log)
        S["del"] = f * de[k + 1] + (1 - f) * de[k]
        gi = self.shift(re, q)
        S["emis"] = np.exp(f * np.log(inten[k + 1]) + (1 - f) * np.log(inten[k])) * gi ** q["gamma"]
        at = [S["del"][int(np.clip(np.searchsorted(-re, -x, side="right") - 1, 0, self.NR - 2))]
              for x in (q["rin"], q["rout"])]
        q["f_inf"] = 0.5 * (1 + math.cos(max(de[-1], math.pi / 2)))
        q["rf"] = 0.5 * (math.cos(at[0]) - math.cos(at[1])) / q["f_inf"]

    @staticmethod
    def shift(r, q):
        a, h, s = q["a"], q["h"], np.sqrt(r)
        ud = (r * s + a) / (s * np.sqrt(r * r - 3 * r + 2 * a * s))
        return ud / math.sqrt((h * h + a * a) / (h * h - 2 * h + a * a))

    # ---- line profile
    def profile(self, q, S, e, rgrid, n_incl=0):
        nz, n, H = len(rgrid) - 1, len(e) - 1, self.H
        gmin, gmax, ng = S["gmin"], S["gmax"], S["trf"][0].shape[1]
        gs = H + (1 - 2 * H) / (ng - 1) * np.arange(ng)
        hit = (gmax > e[0]) & (gmin < e[-1])
        lo = np.clip(np.searchsorted(e, np.maximum(gmin, e[0]), side="right") - 1, 0, n - 1)
        hi = np.clip(np.searchsorted(e, np.minimum(gmax, e[-1]), side="right") - 1, 0, n - 1)
        cnt = np.where(hit, hi - lo + 1, 0)
        rad = np.repeat(np.arange(self.NR), cnt)
        b = np.arange(cnt.sum()) - np.repeat(np.cumsum(cnt) - cnt, cnt) + np.repeat(lo, cnt)
        dg = gmax - gmin

        def F(x, i, k):
            g = (x - gmin[i]) / dg[i]
            j = _last_le(gs, g)
            f = (g - gs[j]) / (gs[j + 1] - gs[j])
            v = x ** 3 / (dg[i] * np.sqrt(g - g * g)) * (f * S["trf"][k][i, j] + (1 - f) * S["trf"][k][i, j + 1])
            if q["limb"]:
                m = f * S["mu"][k][i, j] + (1 - f) * S["mu"][k][i, j + 1]
                v = v * (1 + 2.06 * m if q["limb"] == 1 else np.log(1 + 1 / m))
            return v

        glo, ghi = (np.clip((e[b + o] - gmin[rad]) / dg[rad], 0, 1) for o in (0, 1))
        v = np.zeros(len(rad))
        every = np.arange(self.NR)
        eH, e1H = H * dg + gmin, (1 - H) * dg + gmin
        edge = [sum(F(x, every, k) for k in (0, 1)) * math.sqrt(H) * 2 * dg for x in (eH, e1H)]
        live = ghi > 0
        m = live & (glo <= H)
        v[m] += edge[0][rad[m]] * (np.sqrt(np.minimum(ghi[m], H)) - np.sqrt(glo[m]))
        m = live & (ghi >= 1 - H)
        v[m] += edge[1][rad[m]] * (np.sqrt(1 - np.maximum(glo[m], 1 - H)) - np.sqrt(1 - ghi[m]))
        a = np.where(glo <= H, eH[rad], e[b])
        c = np.where(ghi >= 1 - H, e1H[rad], e[b + 1])
        inner = live & ~((glo <= H) & (ghi <= H)) & ~((ghi >= 1 - H) & (glo >= 1 - H))
        m = np.flatnonzero(inner & (a < 0.95))
        for k in (0, 1):
            v[m] += F(0.5 * (a[m] + c[m]), rad[m], k) * (c[m] - a[m])
        m = np.flatnonzero(inner & (a >= 0.95))
        for k in (0, 1):
            v[m] += self.romberg(lambda x, i, k=k: F(x, i, k), a[m], c[m], rad[m])
        w = v * (S["emis"] * S["wt"])[rad]
        zone = _last_le(rgrid, S["re"])
        flux = np.bincount(zone[rad] * n + b, w, nz * n).reshape(nz, n) / (0.5 * (e[1:] + e[:-1]))
        if q["renorm"]:
            flux *= q["renorm"] / flux.sum()
        if not n_incl:
            return flux, None
        dgs = np.full(ng, gs[1] - gs[0])
        dgs[0] = dgs[-1] = 0.5 * (gs[1] - gs[0]) + H
        dist = np.zeros((nz, n_incl))
        re = S["re"][:, None]
        g = gs * dg[:, None] + gmin[:, None]
        for k in (0, 1):
            im = np.clip((n_incl * (1 - S["mu"][k]) + 1).astype(int) - 1, 0, n_incl - 1)
            t = re * (2 * math.pi * g * re) ** 2 / np.sqrt(gs - gs * gs) * S["trf"][k] * (S["emis"] * S["wt"])[:, None] * dgs
            t = np.where(hit[:, None], t, 0.0)
            np.add.at(dist, (np.broadcast_to(zone[:, None], im.shape), im), t)
        return flux, dist / dist.sum(1, keepdims=True)

    @staticmethod
    def romberg(F, a, b, rad):
        """The reference's Romberg rule: at most 6 refinements, until the last one moved by under 2%."""
        ta = 0.5 * (F(a, rad) + F(b, rad))
        out = np.zeros(len(a))
        at = np.arange(len(a))
        table, s, n = [ta * (b - a)], np.zeros(len(a)), 0
        while len(at) and n < 6:
            n += 1
            h = (b - a) / 2 ** n
            s = s + sum(F(a + h * i, rad) for i in range(1, 2 ** n, 2))
            row, r = [(ta + s) * h], 1.0
            for j in range(n):
                r *= 4
                row.append((r * row[j] - table[j]) / (r - 1))
            out[at] = row[n]
            go = np.abs(row[n] - table[n - 1]) / row[n] > 0.02
            at, a, b, rad, ta, s = at[go], a[go], b[go], rad[go], ta[go], s[go]
            table = [x[go] for x in row]
        return out

    # ---- reflection spectra
    def xillver_table(self):
        path = os.path.join(self.d, "xillver-a-Ec5.fits")
        h = {x[0]: x for x in _hdus(path)}
        p = _rows(path, h["PARAMETERS"])
        vals = [p[q][p.dtype.names[9]][:int(np.ravel(p[q][p.dtype.names[8]])[0])].astype("f4") for q in range(len(p))]
        names = [bytes(p[q][p.dtype.names[0]]).decode().strip() for q in range(len(p))]
        en = _rows(path, h["ENERGIES"])
        lo, hi = (en[en.dtype.names[k]].astype("f8").ravel() for k in (0, 1))
        spec = _rows(path, h["SPECTRA"])
        return names, vals, np.append(lo, hi[-1]), spec[spec.dtype.names[1]]

    def corners(self, tab, q, ecut, n_free):
        """(row, weight) of the brackets' corners over the first n_free parameters."""
        names, vals, _, _ = tab
        want = {"Gamma": q["gamma"], "A_Fe": q["afe"], "logXi": q["logxi"], "Ecut": ecut, "Incl": q["incl_deg"]}
        row, out = [], [(0, 1.0)]
        for k, (name, v) in enumerate(zip(names, vals)):
            if k >= n_free:
                break
            x = min(max(np.float32(want[name]), v[0]), v[-1])
            i = int(_last_le(v, np.float32(want[name])))
            f = float((x - v[i]) / (v[i + 1] - v[i]))
            row = out
            lx = (lambda j: 10.0 ** -float(v[j])) if name == "logXi" else (lambda j: 1.0)
            out = [(r * len(v) + i + u, w * (f if u else 1 - f) * lx(i + u)) for r, w in row for u in (0, 1)]
        return [(r, w) for r, w in out if w]

    @staticmethod
    def cutoff(e, gam, ecut):
        m = 0.5 * (e[1:] + e[:-1])
        return math.exp(1 / ecut) * m ** -gam * np.exp(-m / ecut) * np.diff(e)

    def norm(self, gam, ecut):
        e = np.exp(np.linspace(0, 1, 501) * (math.log(1000.0) - math.log(0.1)) + math.log(0.1))
        return (1e15 / 4 / math.pi) / (np.sum(self.cutoff(e, gam, ecut) * 0.5 * (e[1:] + e[:-1])) * 1e20 * 1.602177e-09)

    def convolve(self, x, rel):
        e = self.conv
        cf = 0.5 * (e[1:] + e[:-1]) / np.diff(e)
        r = np.roll(rel * cf, -int(_last_le(e, 1.0)))
        # the products are non-negative: a direct sum over the profile's window, no FFT rounding
        c, xs = np.zeros(4096), x * cf
        for i in np.flatnonzero(r):
            c += r[i] * np.roll(xs, i)
        c /= cf
        band = (e[:-1] >= 0.01) & (e[1:] < 1000)
        return c * (rel[band].sum() * x[band].sum() / c[band].sum())

    def zones(self, q):
        nz, h, rin, rout = q["nz"], q["h"], q["rin"], q["rout"]
        if nz == 1:
            return np.array([rin, rout])
        g = np.exp(np.linspace(0, 1, nz + 1) * (math.log(rout) - math.log(rin)) + math.log(rin))
        k = int(_last_le(g, h)) if h > rin else 0
        lo = g[k] if h > rin else rin
        f = np.arange(nz + 1 - k) / (nz - k)
        g[k:] = 1 / (f * (1 / rout - 1 / lo) + 1 / lo)
        return g

    # ---- the models
    def parameters(self, model, p):
        v = dict(zip([k for k, _ in R.PARAMS[model]], p))
        q = {"a": v.get("a", 0.0), "incl_deg": v["Incl"], "incl": v["Incl"] * math.pi / 180, "z": v.get("z", 0.0),
             "lineE": v.get("lineE", 1.0), "limb": int(v.get("limb", 0)), "gamma": v.get("gamma", 2.0),
             "logxi": v.get("logxi"), "afe": v.get("Afe"), "ecut": v.get("Ecut"), "refl": v.get("refl_frac"),
             "emis": "lp" if "lp" in model else "bkn", "nz": 10 if model == "relxilllp" else 1, "h": 0.0}
        if model == "xillver":
            return q
        q["rms"] = self._rms(q["a"])
        q["rin"], q["rout"] = q["rms"] * -v["Rin"], v["Rout"]
        if q["emis"] == "bkn":
            q["i1"], q["i2"], q["rbr"] = v["Index1"], v["Index2"], min(max(v["Rbr"], q["rin"]), q["rout"])
            q["renorm"] = 0.5 * math.cos(q["incl"]) if model == "relxill" else 1.0
        else:
            q["h"] = max(v["h"], 1.1 * (1 + math.sqrt(1 - q["a"] ** 2)))
            q["renorm"] = 0.0 if model == "relxilllp" else 1.0
        return q

    def model(self, model, p, energy, flux):
        q = self.parameters(model, p)
        e = energy * (1 + q["z"])
        if model == "xillver":
            return self.xillver(q, e)
        S = self.system(q)
        if model in LINES:
            return self.profile(q, S, e / q["lineE"], np.array([q["rin"], q["rout"]]))[0][0]
        if model in CONVS:
            prof = self.profile(q, S, self.conv, np.array([q["rin"], q["rout"]]))[0][0]
            out = _rebin(e, self.conv, self.convolve(_rebin(self.conv, e, flux), prof))
            out[(e[1:] < 0.01) | (e[:-1] > 1000)] = 0.0
            return out
        return self.relxill(q, S, e)

    def xillver(self, q, e):
        tab = self.xillver_table()
        spec = sum(w * tab[3][r].astype("f8") for r, w in self.corners(tab, q, q["ecut"], 5))
        out = _rebin(e, tab[2], spec * 0.5 * math.cos(q["incl"])) * abs(q["refl"])
        return out + self.cutoff(e, q["gamma"], q["ecut"]) * self.norm(q["gamma"], q["ecut"])

    def relxill(self, q, S, e):
        lamp = q["emis"] == "lp"
        tab = self.xillver_table()
        n_incl = len(tab[1][4])
        rgrid = self.zones(q)
        rmean = 0.5 * (rgrid[1:] + rgrid[:-1])
        rel, dist = self.profile(q, S, self.conv, rgrid, n_incl)
        g_inf = math.sqrt(1 - 2 * q["h"] / (q["h"] ** 2 + q["a"] ** 2)) if lamp else 1.0
        ecut = q["ecut"] / g_inf
        src = self.norm(q["gamma"], ecut)
        rows, total = {}, np.zeros(4096)
        for z in range(q["nz"]):
            if rel[z].sum() < 1e-12:
                continue
            shift = float(self.shift(rmean[z], q)) if lamp else 1.0
            spec = 0.0
            for r, w in self.corners(tab, q, ecut * shift, 4):
                if r not in rows:
                    rows[r] = np.array(tab[3][r * n_incl:(r + 1) * n_incl], dtype="f8")
                spec = spec + w * (dist[z] @ rows[r])
            spec = spec / (self.norm(q["gamma"], ecut * shift) / src)
            total += self.convolve(_rebin(self.conv, tab[2], spec), rel[z])
        prim = self.cutoff(self.conv, q["gamma"], ecut * g_inf) * src
        if lamp:
            total *= abs(q["refl"]) / q["rf"]
            prim = prim * (q["f_inf"] / 0.5 * g_inf ** q["gamma"])
        else:
            total *= abs(q["refl"])
        return _rebin(e, self.conv, total + prim)
