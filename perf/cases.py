"""The work that users of this framework have it do, as cases that can be timed and compared.

The framework synthesises Stokes spectra of stellar-atmosphere pixels and inverts them.  Its users
come with (a) column records (the state their own code holds per depth) and ask for spectra, chi2
gradients or node responses; (b) node vectors (temperature, velocity and field nodes) and ask for the
same with the hydrostatic and chemistry build on the GPU, or for whole Levenberg-Marquardt fits;
(c) atmosphere columns, which they want as records, or as NLTE level populations of Ca II.

Inputs are seeded draws around the columns, node vectors and spectra of the repository's fixtures
(quiet to active solar pixels, 80 or 100 depths, Fe I 6301.5/6302.5 or Ca II 8542).  Nothing in the
inputs comes from the framework's own kernels.  Wavelength counts and, where the caller's records
set it, depth counts vary around the fixtures' (201 wavelengths, 80 depths).
"""
import math
import os

import numpy as np
import torch

import snapi_b200 as sb
from snapi_b200.eos_tables import EosTables

GOLDEN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(sb.__file__))), "tests", "golden")
_LOADED = {}


def listed():
    return [
        # one atmosphere, one spectrum: an interactive call or a serial host program (latency)
        {"name": "synth_one", "do": "synth", "npix": 1, "nl": 201, "nd": 80},
        # a forward-modelled cube from a simulation's records (a 128 x 128 tile per call)
        {"name": "synth_cube", "do": "synth", "npix": 16384, "nl": 201, "nd": 80},
        # chi2 gradient for a gradient-based inversion that keeps its own model -> record map, a
        # ragged batch with an odd wavelength grid, per-pixel masks and dense node tangents
        {"name": "adjoint_records", "do": "adjoint", "npix": 1021, "nl": 187, "nd": 73},
        # the spectra's Jacobian for a caller's own least-squares step (forward mode)
        {"name": "responses", "do": "responses", "npix": 301, "nl": 201, "nd": 80},
        # spectra + chi2 gradient from node vectors, a handful of pixels (one slit position)
        {"name": "nodes_gradient_slit", "do": "nodes", "npix": 61, "nl": 201},
        # the same for a 64 x 64 map: the headline workload
        {"name": "nodes_gradient_map", "do": "nodes", "npix": 4096, "nl": 201},
        # spectra from models with a temperature node at every depth (85 nodes)
        {"name": "synth_from_nodes", "do": "fine", "npix": 1500, "nl": 201},
        # a Levenberg-Marquardt fit of a small map, forward-mode Jacobian, uneven wavelength masks
        {"name": "fit_map", "do": "fit", "npix": 1000, "iters": 4, "tangent": True, "width": 0.0},
        # a fit with the default (central-difference) Jacobian and the instrument's broadening
        {"name": "fit_broadened", "do": "fit", "npix": 77, "iters": 3, "tangent": False, "width": 45.0},
        # a simulation's atmosphere columns to records (the synthesis job's first half)
        {"name": "records_of_columns", "do": "columns", "npix": 4096},
        # Ca II populations of a batch of columns, two rays, to a relative change of 1e-2
        {"name": "nlte_two_rays", "do": "nlte", "npix": 512, "rays": 2, "tol": 1e-2},
        # the same with the ten directions of the five-point angle set, 100 depths, to 1e-4
        {"name": "nlte_ten_rays", "do": "nlte", "npix": 40, "rays": 10, "tol": 1e-4},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    do = rng.choice(["synth", "synth", "adjoint", "responses", "nodes", "nodes", "fine", "fit", "columns", "nlte"])
    if do == "synth":
        return {"do": do, "npix": size(1, 16000), "nl": rng.randint(90, 260), "nd": rng.randint(50, 100)}
    if do == "adjoint":
        return {"do": do, "npix": size(2, 3500), "nl": rng.randint(90, 260), "nd": rng.randint(50, 100)}
    if do == "responses":
        return {"do": do, "npix": size(2, 500), "nl": rng.randint(90, 220), "nd": rng.randint(50, 90)}
    if do == "nodes":
        return {"do": do, "npix": size(1, 4000), "nl": rng.randint(101, 201)}
    if do == "fine":
        return {"do": do, "npix": size(3, 3000), "nl": rng.randint(101, 201)}
    if do == "fit":
        tangent = rng.random() < 0.5
        return {"do": do, "npix": size(5, 900 if tangent else 400), "iters": rng.randint(2, 4), "tangent": tangent,
                "width": rng.choice([0.0, 45.0, 150.0])}
    if do == "columns":
        return {"do": do, "npix": size(4, 6000)}
    rays = rng.choice([2, 10])
    return {"do": do, "npix": size(3, 500 if rays == 2 else 38), "rays": rays, "tol": 1e-2 if rays == 2 else 1e-4}


def work(case):
    """Inputs once and outputs once; arithmetic per the repository's operation counts (per wavelength
    and depth 1196 for a synthesis and 3915 for a synthesis with its reverse sweep; 1.2e7 per column
    build, 9 builds per column where tangents of 4 temperature nodes are wanted)."""
    n, do, npar = case["npix"], case["do"], 10
    if do == "synth":
        nd, nl = case["nd"], case["nl"]
        return {"bytes": n * (nd * 27 * 4 + nl * 16), "flops": n * nd * nl * 1196.0}
    if do == "adjoint":
        nd, nl = case["nd"], case["nl"]
        return {"bytes": n * (nd * 27 * 4 * (1 + npar) + nl * (16 + 16 + 4) + 8 * (1 + npar)),
                "flops": n * nd * nl * 3915.0}
    if do == "responses":
        nd, nl = case["nd"], case["nl"]
        return {"bytes": n * (nd * 27 * 4 * (1 + npar) + nl * 16 * (1 + npar)),
                "flops": n * nd * nl * 1196.0 * (1 + npar)}
    if do == "nodes":
        return {"bytes": n * (8 * npar + case["nl"] * 32 + 8 * (1 + npar) + 4),
                "flops": n * (1.08e8 + 80 * case["nl"] * 3915.0)}
    if do == "fine":
        return {"bytes": n * (8 * 85 + case["nl"] * 16 + 4), "flops": n * (1.2e7 + 80 * case["nl"] * 1196.0)}
    if do == "fit":
        per = 1.08e8 + 80 * 201 * 1196.0 * (1 + npar)
        return {"bytes": n * (2 * 8 * npar + 201 * (16 + 4 + 16) + 12), "flops": n * per * (case["iters"] + 1)}
    if do == "columns":
        return {"bytes": n * 80 * (12 * 8 + 27 * 4), "flops": n * 80 * 1.5e5}
    nd, it = (80, 12) if case["rays"] == 2 else (100, 60)
    return {"bytes": n * nd * (12 * 8 + 2 * 6 * 8), "flops": n * nd * 444.0 * case["rays"] * it * 700.0}


# ---- inputs ---------------------------------------------------------------------------------------
def fixture(name):
    if name not in _LOADED:
        with np.load(os.path.join(GOLDEN, name + ".npz")) as z:
            _LOADED[name] = {k: z[k] for k in z.files}
    return _LOADED[name]


def cuda(a, dtype=None):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype).cuda()


def window(pool, nl):
    """nl of the fixture's wavelengths around the lines (all of them for 201), or a grid of nl over
    the same window."""
    lam = pool["lambda_air"]
    return lam if nl == lam.size else np.linspace(lam[0], lam[-1], nl)


def spectra(pool, col, nl, rng, noise):
    """Observed spectra: the fixture's, on the window's grid, with photon noise."""
    lam, st = pool["lambda_air"], pool["stokes"][col]
    if nl != lam.size:
        x = np.linspace(0.0, lam.size - 1.0, nl)
        i = np.minimum(x.astype(int), lam.size - 2)
        w = (x - i)[None, :, None]
        st = st[:, i] * (1.0 - w) + st[:, i + 1] * w
    return (st + rng.normal(0.0, noise, st.shape)).astype(np.float32)


def masks(npix, nl, rng):
    """Per-pixel wavelength masks: a contiguous window of 60 to 100 % with some single points off."""
    keep = rng.integers(int(0.6 * nl), nl + 1, npix)
    start = (rng.random(npix) * (nl - keep + 1)).astype(int)
    l = np.arange(nl)[None, :]
    m = (l >= start[:, None]) & (l < (start + keep)[:, None]) & (rng.random((npix, nl)) > 0.02)
    return m.astype(np.float32)


def on_depths(a, nd):
    """Columns [..., depth, field] on nd depths of the same log tau range."""
    n = a.shape[-2]
    if nd == n:
        return a
    x = np.linspace(0.0, n - 1.0, nd)
    i = np.minimum(x.astype(int), n - 2)
    w = (x - i)[:, None]
    return a[..., i, :] * (1.0 - w) + a[..., i + 1, :] * w


def truth(npix, rng):
    return {"vt": rng.uniform(0.5e5, 2.0e5, npix), "v1": rng.normal(0.0, 1e5, npix), "v2": rng.normal(0.0, 1e5, npix),
            "B": 10.0 ** rng.uniform(2.0, math.log10(2500.0), npix),
            "th": rng.uniform(math.radians(20.0), math.radians(160.0), npix),
            "ph": rng.uniform(math.radians(10.0), math.radians(170.0), npix)}


def records(pool, npix, nd, rng):
    """Column records [npix, nd, 27] (float32) on the GPU and the fixture column of each."""
    col = rng.integers(0, pool["record"].shape[0], npix)
    rec = cuda(on_depths(pool["record"], nd), torch.float32)[torch.from_numpy(col).cuda()]
    w = on_depths(pool["tangent"][0, 5:7, :, 3].T.astype(np.float64)[None], nd)[0]
    p = truth(npix, rng)
    rec[:, :, 1] = cuda(p["vt"], torch.float32)[:, None]
    rec[:, :, 3] = cuda(p["v1"][:, None] * w[None, :, 0] + p["v2"][:, None] * w[None, :, 1], torch.float32)
    rec[:, :, 4] = cuda(p["B"], torch.float32)[:, None]
    rec[:, :, 5] = cuda(np.rad2deg(p["th"]), torch.float32)[:, None]
    az = np.rad2deg(p["ph"])
    rec[:, :, 6] = cuda(np.where(az > 90.0, az - 180.0, az), torch.float32)[:, None]
    return rec.contiguous(), col


def context(pool, nl, nd, npix, scale):
    f = dict(pool, lambda_air=window(pool, nl), tau500=10.0 ** np.linspace(-6.0, 1.0, nd))
    return sb.Context.from_fixture(f, stokes_scale=scale, max_batch=min(npix, 4096))


def node_vectors(pool, npix, rng):
    """Models of an inversion under way: fixture nodes with offsets of the size a fit starts from."""
    col = rng.integers(0, pool["nodes"].shape[0], npix)
    sig = np.array([100.0, 100.0, 100.0, 100.0, 1e4, 2e4, 2e4, 50.0, 0.05, 0.05])
    off = np.array([0.0, 0.0, 0.0, 0.0, 0.3e5, 0.3e5, -0.3e5, 200.0, 0.1, 0.1])
    return pool["nodes"][col] + off + rng.normal(0.0, 1.0, (npix, 10)) * sig, col


def smooth(npix, nd, rng):
    """Smooth random depth profiles of unit size [npix, nd]."""
    x = np.linspace(0.0, math.pi, nd)[None, :]
    return sum(rng.normal(0.0, 0.7, (npix, 1)) * np.cos(k * x) for k in range(3))


def prepare(case, seed):
    rng = np.random.default_rng([seed, 17])
    do, n = case["do"], case["npix"]
    pool = fixture("bench_pool")
    ic = float(pool["stokes"][:, :, 0].max())
    s = {"do": do, "n": n}
    if do in ("synth", "adjoint", "responses"):
        nl, nd = case["nl"], case["nd"]
        s["rec"], col = records(pool, n, nd, rng)
        s["ctx"] = context(pool, nl, nd, n, ic)
        s["stokes"] = torch.empty(n, nl, 4, device="cuda")
        if do != "synth":
            s["tan"] = cuda(on_depths(pool["tangent"], nd), torch.float32)[torch.from_numpy(col).cuda()].contiguous()
        if do == "adjoint":
            s["obs"] = cuda(spectra(pool, col, nl, rng, 1e-3 * ic))
            s["mask"] = cuda(masks(n, nl, rng))
            s["chi2"] = torch.empty(n, dtype=torch.float64, device="cuda")
            s["grad"] = torch.empty(n, 10, dtype=torch.float64, device="cuda")
        if do == "responses":  # this entry point's arrays are the host's
            s["ctx"].jacobian_mode(sb.api.JACOBIAN_TANGENT)
            s["rec"], s["tan"] = s["rec"].cpu().numpy(), s["tan"].cpu().numpy()
            s["step"] = 1e-2 * np.array([5e3] * 4 + [1e5] * 3 + [1e3, 1.0, 1.0])
    elif do == "nodes":
        nl = case["nl"]
        nodes, col = node_vectors(pool, n, rng)
        s["ctx"] = context(pool, nl, 80, n, ic)
        s["ctx"].eos_set(EosTables(fixture("eos_c3")))
        s["nodes"] = cuda(nodes)
        s["obs"] = cuda(spectra(pool, col, nl, rng, 1e-3 * ic))
        s["stokes"] = torch.empty(n, nl, 4, device="cuda")
        s["chi2"] = torch.empty(n, dtype=torch.float64, device="cuda")
        s["grad"] = torch.empty(n, 10, dtype=torch.float64, device="cuda")
        s["status"] = torch.empty(n, dtype=torch.int32, device="cuda")
    elif do == "fine":
        nl = case["nl"]
        eos = fixture("eos_c1")
        nodes = eos["nodes"][rng.integers(0, eos["nodes"].shape[0], n)].copy()
        nodes[:, :80] += 80.0 * smooth(n, 80, rng)
        p = truth(n, rng)
        nodes[:, 80:] = np.stack([p["vt"], p["v1"], p["B"], p["th"], p["ph"]], axis=1)
        s["ctx"] = context(pool, nl, 80, n, ic)
        s["ctx"].eos_set(EosTables(eos))
        s["nodes"] = cuda(nodes)
        s["rec"] = torch.empty(n, 80, 27, device="cuda")
        s["status"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["stokes"] = torch.empty(n, nl, 4, device="cuda")
    elif do == "fit":
        s["nodes"], col = node_vectors(pool, n, rng)
        s["ctx"] = context(pool, 201, 80, n, ic)
        s["ctx"].eos_set(EosTables(fixture("eos_c3")))
        s["ctx"].jacobian_mode(sb.api.JACOBIAN_TANGENT if case["tangent"] else sb.api.JACOBIAN_FD)
        s["obs"] = spectra(pool, col, 201, rng, 1e-3 * ic)
        s["mask"] = masks(n, 201, rng)
        s["kinds"] = pool["node_kind"].astype(np.int32)
        s["step"] = 1e-2 * np.array([{1: 5e3, 2: 1e5, 3: 1e5, 4: 1e3}.get(int(k), 1.0) for k in s["kinds"]])
        s["kw"] = {"lm_start": 1e3, "max_iter": case["iters"], "delta": 1e-4,
                   "spectral_broadening": case["width"] * 1e-11 / 2.3548}  # FWHM in mA to sigma in cm
    elif do == "columns":
        c = fixture("eos_c3")["atm_arr"]
        a = c[rng.integers(0, c.shape[0], n)].copy()
        jitter(a, rng)
        s["ctx"] = context(pool, 201, 80, n, ic)
        s["ctx"].eos_set(EosTables(fixture("eos_c3")))
        s["cols"] = a
    else:
        fx = fixture("config5" if case["rays"] == 2 else "config5_spec")
        a = fx["alis_atm"][rng.integers(0, fx["alis_atm"].shape[0], n)].copy()
        jitter(a, rng)
        s["ctx"] = sb.Context.from_fixture(fx)
        s["ctx"].eos_set(EosTables({k[4:]: v for k, v in fx.items() if k.startswith("eos_")}))
        s["ali"] = sb.api.AliContext.from_fixture(fx)
        s["tables"] = sb.api.AliSetupTables.from_fixture(fx)
        s["cols"] = cuda(a)
        s["out"] = {k: torch.empty(v, dtype=torch.float64, device="cuda") for k, v in s["ali"].column_shapes(n).items()}
        s["rel"] = torch.empty(n, dtype=torch.float64, device="cuda")
        s["iters"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["status"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["tol"] = case["tol"]
    torch.cuda.synchronize()
    return s


def jitter(a, rng):
    """Columns in the 12-row layout with other temperatures, pressures and velocities."""
    n, _, nd = a.shape
    a[:, 2] *= 1.0 + 0.01 * smooth(n, nd, rng)
    a[:, 3] *= 10.0 ** (0.02 * smooth(n, nd, rng))
    a[:, 8] = rng.uniform(0.5e5, 2e5, (n, 1))
    a[:, 9] += 1e5 * smooth(n, nd, rng)


# ---- one pass -------------------------------------------------------------------------------------
def run(s):
    do, n, ctx = s["do"], s["n"], s["ctx"]
    if do == "synth":
        ctx.synth_device(n, s["rec"].data_ptr(), s["stokes"].data_ptr())
        return s["stokes"]
    if do == "adjoint":
        ctx.adjoint_device(n, s["rec"].data_ptr(), s["obs"].data_ptr(), 10, s["tan"].data_ptr(), s["chi2"].data_ptr(),
                           s["grad"].data_ptr(), stokes_ptr=s["stokes"].data_ptr(), mask_ptr=s["mask"].data_ptr())
        return {"stokes": s["stokes"], "chi2": s["chi2"], "grad": s["grad"]}
    if do == "responses":
        st, ds = ctx.responses(s["rec"], s["tan"], s["step"])
        return {"stokes": st, "responses": ds}
    if do == "nodes":
        ctx.adjoint_nodes_device(n, s["nodes"].data_ptr(), s["obs"].data_ptr(), s["chi2"].data_ptr(),
                                 s["grad"].data_ptr(), stokes_ptr=s["stokes"].data_ptr(),
                                 status_ptr=s["status"].data_ptr())
        return {"stokes": s["stokes"], "chi2": s["chi2"], "grad": s["grad"], "status": s["status"]}
    if do == "fine":
        ctx.build_records_device(n, s["nodes"].data_ptr(), s["rec"].data_ptr(), status_ptr=s["status"].data_ptr())
        ctx.synth_device(n, s["rec"].data_ptr(), s["stokes"].data_ptr())
        return {"records": s["rec"], "status": s["status"], "stokes": s["stokes"]}
    if do == "fit":
        r = ctx.lm_fit_device(s["nodes"], s["obs"], s["kinds"], s["step"], mask=s["mask"], **s["kw"])
        return {k: r[k] for k in ("nodes", "chi2", "iters", "stokes")}
    if do == "columns":
        rec, status = ctx.records_from_columns(s["cols"])
        return {"records": rec, "status": status}
    o = s["out"]
    p = {k: v.data_ptr() for k, v in o.items()}
    s["ali"].setup_device(ctx, s["tables"], n, s["cols"].data_ptr(), {k: v for k, v in p.items() if k != "pops"},
                          p["pops"], s["status"].data_ptr())
    s["ali"].iterate_device(n, p, p["pops"], max_iter=200, tol=s["tol"], rel_ptr=s["rel"].data_ptr(),
                            iters_ptr=s["iters"].data_ptr(), status_ptr=s["status"].data_ptr())
    return {"pops": o["pops"], "rel": s["rel"], "iters": s["iters"], "status": s["status"], "ne": o["ne"],
            "kappa": o["kappa"]}


# ---- the same in 64 bits --------------------------------------------------------------------------
# Spectra from column records, with their derivatives by automatic differentiation.  What starts from
# node vectors or atmosphere columns has no such value: its records, fits and populations are the
# iterates at which stop rules (1e-4 in the chemistry, 1e-2 in the hydrostatic steps, the fit's and
# the populations' own) end, computed in 64 bits already.
C, H, K = 2.99792458e10, 6.6260687652e-27, 1.3806503e-16


def to_vacuum(lam):
    s2 = (1e4 / (lam * 1e8)) ** 2
    return lam * (1.0 + 0.00008336624212083 + 0.02408926869968 / (130.1065924522 - s2) +
                  0.0001599740894897 / (38.92568793293 - s2))


def horner(z, coef):
    r = torch.full_like(z, coef[-1])
    for c in reversed(coef[:-1]):
        r = c + z * r
    return r


def voigt_faraday(x, a):
    """Humlicek's four-region rational approximation (1982): H and F over sqrt(pi)."""
    s = x.abs() + a
    far, mid = s >= 15.0, (s > 5.5) & (s < 15.0)
    near = (s <= 5.5) & (a > 0.195 * x.abs() - 0.176)
    core = ~(far | mid | near)
    out = torch.zeros(torch.broadcast_shapes(x.shape, a.shape), dtype=torch.complex128, device=x.device)
    x, a = x.expand(out.shape), a.expand(out.shape)
    for k, m in enumerate((far, mid, near, core)):
        if not bool(m.any()):
            continue
        t = torch.complex(torch.where(m, a, torch.ones_like(a) * (1.0 if k != 3 else 1e-2)),
                          -torch.where(m, x, torch.ones_like(x) * (20.0, 8.0, 1.0, 2.0)[k]))
        u = t * t
        if k == 0:
            w = t * 0.5641896 / (0.5 + u)
        elif k == 1:
            w = t * (1.410474 + u * 0.5641896) / (0.75 + u * (3.0 + u))
        elif k == 2:
            w = horner(t, [16.4955, 20.20933, 11.96482, 3.778987, 0.5642236]) / \
                horner(t, [16.4955, 38.82363, 39.27121, 21.69274, 6.699398, 1.0])
        else:
            num = t * horner(-u, [36183.31, 3321.9905, 1540.787, 219.0313, 35.76683, 1.320522, 0.56419])
            den = horner(-u, [32066.6, 24322.84, 9022.228, 2186.181, 364.2191, 61.57037, 1.841439, 1.0])
            si, e = torch.sin(u.imag), torch.exp(u.real)
            w = torch.complex(e * torch.sqrt(1.0 - si * si), e * si) - num / den
        out = torch.where(m, w, out)
    return out.real / 1.77245386399759, out.imag / 1.77245386399759


def planck(lam, T):
    return 2.0 * 6.62606957 * 8.9875517e-7 / lam ** 5 / (torch.exp(1.4387769 / lam / T) - 1.0)


def opacity(rec, f, lam, mid):
    """eta_I, eta_Q, eta_U, eta_V, rho_Q, rho_U, rho_V and the four emissivities over kappa_500,
    each [npix, nd, nl], of records [npix, nd, nfield]."""
    r = [rec[:, :, i, None] for i in range(rec.shape[2])]
    T, vt, ne, vlos, B = r[:5]
    la, lA = lam[None, None, :], lam * 1e8
    thomson = ne * 6.65e-25
    th, ph = (torch.where(B < 1e-3, torch.zeros_like(q), q * math.pi / 180.0) for q in (r[5], r[6]))
    st2, ct = torch.sin(th) ** 2, torch.cos(th)
    c2, s2 = torch.cos(2.0 * ph), torch.sin(2.0 * ph)
    fudge = torch.where(lA > 4500.0, 0.0, 2.1177 * torch.exp(-(lA - 2087.7) ** 2 / 2.421e6) + 0.68738)
    fudge = 1.0 + 0.666667 * fudge
    alpha = sum(c * lA ** i for i, c in enumerate((1.99654, -1.18267e-5, 2.64243e-6, -4.40524e-10, 3.23992e-14,
                                                   -1.39568e-18, 2.78701e-23)))
    lg = torch.log10(lA)
    f0 = -2.2763 - 1.6850 * lg + 0.76661 * lg ** 2 - 0.053346 * lg ** 3
    f1 = 15.2827 - 9.2846 * lg + 1.99381 * lg ** 2 - 0.142631 * lg ** 3
    f2 = -197.789 + 190.266 * lg - 67.9775 * lg ** 2 + 10.6913 * lg ** 3 - 0.625151 * lg ** 4
    lt = torch.log10(5040.0 / T)
    hminus = fudge * (alpha * r[8] * (1.0 - torch.exp(-H * C / la / K / T)) + r[9] * 10.0 ** (f0 + f1 * lt + f2 * lt ** 2))
    eta = [thomson + r[10] + hminus, 0.0, 0.0, 0.0]
    em = [thomson * planck(mid, T) + r[11] + hminus * planck(la, T), 0.0, 0.0, 0.0]
    rho = [0.0, 0.0, 0.0]
    for j in range(f["line_const"].shape[0]):
        lam0, sf, ar, mass = (float(v) for v in f["line_const"][j, :4])
        op, emi, gc = r[12 + 3 * j], r[13 + 3 * j], r[14 + 3 * j]
        width = torch.sqrt(2.0 * K * T / mass + vt ** 2) * lam0 / C
        a = sf * (ar + gc) / width
        shifted = la * (1.0 + vlos / C)
        if not int(f["line_const"][j, 5]):
            h = voigt_faraday((lam0 - shifted) / width, a)[0] / width
            eta[0] = eta[0] + op * h
            em[0] = em[0] + emi * h
            continue
        hs, fs = [], []
        for g in range(3):
            h = v = 0.0
            for i in range(int(f["line_ncomp"][j, g])):
                strength, shift = (float(q) for q in f["line_pattern"][j, g, :, i])
                x = (lam0 + shift * 4.67e-5 * lam0 * lam0 * B - shifted) / width
                p, q = voigt_faraday(x, a)
                h, v = h + strength * p / width, v + strength * q / width
            hs.append(h)
            fs.append(v)

        def vector(p, b, red):
            lin = 0.5 * (p - 0.5 * (red + b)) * st2
            return lin * c2, lin * s2, 0.5 * (red - b) * ct

        e = (0.5 * (hs[0] * st2 + 0.5 * (hs[2] + hs[1]) * (1.0 + ct * ct)),) + vector(*hs)
        for k in range(4):
            eta[k] = eta[k] + op * e[k]
            em[k] = em[k] + emi * e[k]
        for k, q in enumerate(vector(*fs)):
            rho[k] = rho[k] + op * q
    return [q / r[7] for q in eta], [q / r[7] for q in rho], [q / r[7] for q in em]


def spectrum(rec, f, lam_air, tau, mu=1.0):
    """Emergent Stokes vectors [npix, nl, 4]: linear DELO along the ray, optical depths by monotone
    Bezier increments, the top point copied from the one below."""
    lam = to_vacuum(lam_air)
    eta, rho, em = opacity(rec, f, lam, 0.5 * (lam[-1] + lam[0]))
    one = torch.ones_like(eta[0])
    eta, rho, em = ([q * one for q in v] for v in (eta, rho, em))
    z0 = torch.zeros_like(one)
    q, u, v = (eta[k] / eta[0] for k in (1, 2, 3))
    a, b, c = (rho[k] / eta[0] for k in range(3))
    kp = torch.stack([torch.stack(row, -1) for row in
                      ((z0, q, u, v), (q, z0, c, -b), (u, -c, z0, a), (v, b, -a, z0))], -2)
    src = torch.stack([e / eta[0] for e in em], -1)
    nd, oo = rec.shape[1], eta[0]
    step = lambda i: (tau[i + 1] - tau[i]) / mu  # noqa: E731
    slope = [(oo[:, i] - oo[:, i + 1]) / step(i) for i in range(nd - 1)]  # upwards, from i + 1 to i
    der = [None] * nd
    der[nd - 1], der[0] = slope[nd - 2], slope[0]
    for i in range(1, nd - 1):
        h1, h2, d1, d2 = step(i), step(i - 1), slope[i], slope[i - 1]
        al = (1.0 + h1 / (h1 + h2)) / 3.0
        same = d1 * d2 > 0.0
        den = torch.where(same, al * d1 + (1.0 - al) * d2, torch.ones_like(d1))
        der[i] = torch.where(same, d1 * d2 / den, torch.zeros_like(d1))
    I = torch.stack([src[:, nd - 1, :, 0]] + [z0[:, 0]] * 3, -1)
    eye = torch.eye(4, dtype=rec.dtype, device=rec.device)
    for i in range(nd - 2, 0, -1):
        h = step(i)
        ctrl = 0.5 * (oo[:, i] - 0.5 * h * der[i] + oo[:, i + 1] + 0.5 * h * der[i + 1])
        t = h / 3.0 * (oo[:, i] + oo[:, i + 1] + ctrl)
        small, big = torch.where(t < 1e-2, t, 0.0 * t), torch.where(t < 1e-2, 1.0 + 0.0 * t, t)
        e = torch.where(t < 1e-2, 1.0 - small + small ** 2 / 2.0 - small ** 3 / 6.0, torch.exp(-big))
        w0 = torch.where(t < 1e-2, small * (0.5 - small * (1.0 / 3.0 - small / 8.0)),
                         1.0 / big - torch.exp(-big) * (1.0 + 1.0 / big))
        w1 = torch.where(t < 1e-2, 0.5 * small * (1.0 - small / 3.0 * (1.0 - small / 4.0)),
                         1.0 - 1.0 / big + torch.exp(-big) / big)
        w0, w1, e = w0[..., None], w1[..., None], e[..., None]
        rhs = e * I + w0 * (src[:, i + 1] - (kp[:, i + 1] @ I[..., None])[..., 0]) + w1 * src[:, i]
        I = torch.linalg.solve(eye + w1[..., None] * kp[:, i], rhs)
    return I


def exact(case, seed):
    do = case["do"]
    if do not in ("synth", "adjoint", "responses"):
        return None
    s = prepare(case, seed)
    s.pop("ctx").close()
    f = fixture("bench_pool")
    lam = cuda(window(f, case["nl"]))
    tau = cuda(10.0 ** np.linspace(-6.0, 1.0, case["nd"]))
    chunk = {"synth": 256, "adjoint": 48, "responses": 32}[do]
    if case["npix"] * case["nl"] * case["nd"] > {"synth": 6e7, "adjoint": 3e7, "responses": 7e6}[do]:
        return None  # over 20 seconds
    got = {"stokes": [], "chi2": [], "grad": [], "responses": []}
    for i in range(0, case["npix"], chunk):
        rec = torch.as_tensor(s["rec"][i:i + chunk]).cuda().double()
        if do == "synth":
            with torch.no_grad():
                got["stokes"].append(spectrum(rec, f, lam, tau))
            continue
        tan = torch.as_tensor(s["tan"][i:i + chunk]).cuda().double()
        if do == "adjoint":
            rec.requires_grad_(True)
            st = spectrum(rec, f, lam, tau)
            chi2 = ((s["obs"][i:i + chunk].double() - st) * s["mask"][i:i + chunk, :, None].double()).square().sum((1, 2))
            g, = torch.autograd.grad(chi2.sum(), rec)
            got["grad"].append(torch.einsum("pdf,pqdf->pq", g, tan))
            got["chi2"].append(chi2.detach())
            got["stokes"].append(st.detach())
            del st, chi2, g
        else:
            fn = lambda r: spectrum(r, f, lam, tau)  # noqa: E731
            d = [torch.func.jvp(fn, (rec,), (tan[:, q].contiguous(),)) for q in range(tan.shape[1])]
            got["stokes"].append(d[0][0])
            got["responses"].append(torch.stack([v[1] for v in d], 1))
    got = {k: torch.cat(v) for k, v in got.items() if v}
    return got["stokes"] if do == "synth" else got
