"""Forms of the population iteration that the fixtures do not have (snapi_ali_iter): few and odd numbers of
wavelengths (the work arrays hold them in groups of 16, 8 or 4), every depth range of the sums (four, two
and one slice of wavelengths), the fewest depths, and more columns than one batch of work buffers holds."""
import sys

import numpy as np
import pytest

from conftest import ROOT, load_fixture

sys.path.insert(0, ROOT + "/oracle")
import ali_oracle  # noqa: E402

pytestmark = pytest.mark.gpu

DEPTH = ("T", "ne", "na", "kap", "vray", "dld", "adamp", "bfratio", "bgop", "bgem", "grid")


def _form(every, drop, nd):
    """The two-ray fixture on every `every`-th wavelength less the last `drop`, its columns on nd depths."""
    fx = dict(load_fixture("config5"))
    lam = slice(0, len(fx["ali_lambda"]) - drop, every)
    for k in ("lambda", "lw", "fudge"):
        fx["ali_" + k] = fx["ali_" + k][lam]
    fx["ali_sigma"] = fx["ali_sigma"][:, lam]
    fx["ali_bgop"], fx["ali_bgem"] = fx["ali_bgop"][:, :, lam], fx["ali_bgem"][:, :, lam]
    n0 = len(fx["ali_grid"])
    at = np.linspace(0, n0 - 1, nd)
    i = np.minimum(at.astype(int), n0 - 2)
    w = at - i
    for k in DEPTH:
        a = np.asarray(fx["ali_" + k])
        fx["ali_" + k] = a[..., i] * (1.0 - w) + a[..., i + 1] * w
    for k in ("coll", "pop0"):
        a = np.asarray(fx["ali_" + k])
        ww = w.reshape((-1,) + (1,) * (a.ndim - 2))
        fx["ali_" + k] = a[:, i] * (1.0 - ww) + a[:, i + 1] * ww
    return fx


@pytest.mark.parametrize("every,drop,nd", [(1, 1, 80), (30, 0, 80), (3, 0, 3), (7, 0, 257), (30, 1, 513)])
def test_one_iteration_against_the_oracle(every, drop, nd):
    import snapi_b200 as sb
    fx = _form(every, drop, nd)
    ctx = sb.api.AliContext.from_fixture(fx)
    pops, rel, iters, st = ctx.iterate(ctx.columns_from_fixture(fx), fx["ali_pop0"], max_iter=1, tol=1e-30)
    P = ali_oracle.Problem(fx)
    for c in range(len(pops)):
        ref, r, neg = ali_oracle.iterate(P, fx, c, np.asarray(fx["ali_pop0"][c]))
        assert bool(neg) == (st[c] != 0)
        if neg:
            continue
        # FP32 profiles (relative 1e-6) against FP64 ones; the step gains up to 20 on the full grid and may
        # gain more on a thinned one.  A wavelength lost or taken twice is of order one over their number.
        assert np.abs(pops[c] / ref - 1.0).max() < 1e-3
        np.testing.assert_allclose(rel[c], r, rtol=1e-3)
    # a column alone, and in a batch of another size: the same bits
    one = {k: np.asarray(v)[1:2] for k, v in ctx.columns_from_fixture(fx).items()}
    alone, _, _, st1 = ctx.iterate(one, fx["ali_pop0"][1:2], max_iter=1, tol=1e-30)
    assert st1[0] == st[1] and np.array_equal(alone[0], pops[1])
    ctx.close()


def test_more_columns_than_a_batch_holds():
    import torch

    import snapi_b200 as sb
    fx = load_fixture("config5")
    ctx = sb.api.AliContext.from_fixture(fx)
    cols = ctx.columns_from_fixture(fx)
    want, rel, iters, st = ctx.iterate(cols, fx["ali_pop0"], max_iter=3, tol=1e-30)
    # 7 MB of work a column against 24 GiB a batch
    reps = 1400
    dev = {k: torch.tensor(np.asarray(v, np.float64)).cuda().repeat((reps,) + (1,) * (np.ndim(v) - 1)) for k, v in cols.items()}
    names = {"kap": "kappa", "bgop": "bg_op", "bgem": "bg_em"}
    n = 3 * reps
    pops = torch.tensor(np.asarray(fx["ali_pop0"], np.float64)).cuda().repeat(reps, 1, 1)
    r = torch.zeros(n, dtype=torch.float64, device="cuda")
    it, s = (torch.full((n,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    ctx.iterate_device(n, {names.get(k, k): v.data_ptr() for k, v in dev.items()}, pops.data_ptr(), max_iter=3, tol=1e-30,
                       rel_ptr=r.data_ptr(), iters_ptr=it.data_ptr(), status_ptr=s.data_ptr())
    assert torch.equal(pops.cpu(), torch.tensor(want).repeat(reps, 1, 1))
    assert torch.equal(r.cpu(), torch.tensor(rel).repeat(reps)) and bool((it == 3).all()) and bool((s == 0).all())
    ctx.close()


def _levels(fx, keep):
    """The fixture's atom on the levels `keep` alone (the last one the continuum), their populations its total."""
    fx = dict(fx)
    lv = list(keep)
    tr = np.asarray(fx["ali_tr"]).astype(int)
    on = [t for t in range(len(tr)) if tr[t, 1] in lv and tr[t, 2] in lv]
    of = {t: k for c in (0, 1) for k, t in enumerate(np.flatnonzero(tr[:, 0] == c))}  # among its kind
    ln, bf = ([of[t] for t in on if tr[t, 0] == c] for c in (0, 1))
    fx["ali_trc"] = np.asarray(fx["ali_trc"])[on]
    tr = tr[on]
    tr[:, 1:3] = [[lv.index(i) for i in row] for row in tr[:, 1:3]]
    fx["ali_tr"] = tr
    for k in ("A", "B"):
        fx["ali_" + k] = np.asarray(fx["ali_" + k])[np.ix_(lv, lv)]
    for k in ("dld", "adamp"):
        fx["ali_" + k] = np.asarray(fx["ali_" + k])[:, ln]
    fx["ali_bfratio"], fx["ali_sigma"] = np.asarray(fx["ali_bfratio"])[:, bf], np.asarray(fx["ali_sigma"])[bf]
    fx["ali_coll"] = np.asarray(fx["ali_coll"])[:, :, lv][:, :, :, lv]
    fx["ali_pop0"] = np.asarray(fx["ali_pop0"])[:, :, lv]
    fx["ali_na"] = fx["ali_pop0"].sum(-1)
    return fx


def _compare_one_iteration(fx):
    """FP32 profiles against FP64 ones: of 1e-6 each (W4, and a Doppler shift of up to 3 widths rounded to
    FP32), and a step of the oracle from profiles moved by 1e-6 differs by 1e-6: 1e-4 as in test_ali.py."""
    import snapi_b200 as sb
    ctx = sb.api.AliContext.from_fixture(fx)
    pops, rel, iters, st = ctx.iterate(ctx.columns_from_fixture(fx), fx["ali_pop0"], max_iter=1, tol=1e-30)
    ctx.close()
    P = ali_oracle.Problem(fx)
    for c in range(len(pops)):
        ref, r, neg = ali_oracle.iterate(P, fx, c, np.asarray(fx["ali_pop0"][c]))
        assert not neg and st[c] == 0
        assert np.abs(pops[c] / ref - 1.0).max() < 1e-4
        np.testing.assert_allclose(rel[c], r, rtol=1e-4)


@pytest.mark.parametrize("nd", [897, 1024])
def test_deepest_grids(nd):
    """The rate equations are one thread per depth of one CTA, up to 1024: 29 warps and more."""
    _compare_one_iteration(_levels(_form(7, 1, nd), (0, 3, 4, 5)))


def _on_device(fx, cols, reps):
    import torch
    names = {"kap": "kappa", "bgop": "bg_op", "bgem": "bg_em"}
    dev = {names.get(k, k): torch.tensor(np.asarray(v, np.float64)).cuda().repeat((reps,) + (1,) * (np.ndim(v) - 1))
           for k, v in cols.items()}
    pops = torch.tensor(np.asarray(fx["ali_pop0"], np.float64)).cuda().repeat(reps, 1, 1)
    torch.cuda.synchronize()
    return dev, pops


def test_work_buffers_leave_half_of_the_free_memory():
    """300 columns want 2 GiB of work buffers where 1 GiB is free: they run in batches of what half of that holds,
    with the same bits, and the next calls keep those buffers."""
    import torch

    import snapi_b200 as sb
    fx = load_fixture("config5")
    ctx = sb.api.AliContext.from_fixture(fx)
    cols = ctx.columns_from_fixture(fx)
    want, _, _, _ = ctx.iterate(cols, fx["ali_pop0"], max_iter=2, tol=1e-30)
    dev, pops = _on_device(fx, cols, 100)
    torch.cuda.empty_cache()
    rest = torch.empty(torch.cuda.mem_get_info()[0] - (1 << 30), dtype=torch.uint8, device="cuda")
    free = [torch.cuda.mem_get_info()[0]]
    for _ in range(3):
        p = pops.clone()
        torch.cuda.synchronize()
        ctx.iterate_device(300, {k: v.data_ptr() for k, v in dev.items()}, p.data_ptr(), max_iter=2, tol=1e-30)
        free.append(torch.cuda.mem_get_info()[0])
        assert torch.equal(p.cpu(), torch.tensor(want).repeat(100, 1, 1))
    del rest
    torch.cuda.empty_cache()
    assert free[0] > 0.8 * 2**30 and free[1] > 0.4 * free[0] and free[3] == free[1], free
    ctx.close()


def test_a_host_call_keeps_the_work_buffers():
    import torch

    import snapi_b200 as sb
    fx = load_fixture("config5")
    ctx = sb.api.AliContext.from_fixture(fx)
    cols = ctx.columns_from_fixture(fx)
    dev, pops = _on_device(fx, cols, 100)
    ctx.iterate_device(300, {k: v.data_ptr() for k, v in dev.items()}, pops.data_ptr(), max_iter=2, tol=1e-30)
    free = torch.cuda.mem_get_info()[0]
    got, _, _, _ = ctx.iterate(cols, fx["ali_pop0"], max_iter=2, tol=1e-30)
    assert torch.cuda.mem_get_info()[0] <= free
    assert np.array_equal(got, pops[:3].cpu().numpy())
    ctx.close()


@pytest.mark.parametrize("memory", ["device", "pinned", "pageable"])
def test_inputs_of_a_device_call_that_lie_elsewhere(memory):
    """Device inputs are read in place; memory that the kernels of this GPU cannot or should not read there is copied
    first (another GPU's, pinned host memory), and what is no CUDA memory is an error of the call, not of the GPU."""
    import torch

    import snapi_b200 as sb
    fx = load_fixture("config5")
    ctx = sb.api.AliContext.from_fixture(fx)
    cols = ctx.columns_from_fixture(fx)
    want, _, _, _ = ctx.iterate(cols, fx["ali_pop0"], max_iter=2, tol=1e-30)
    dev, pops = _on_device(fx, cols, 1)
    if memory != "device":  # one of the inputs
        host = dev["bg_op"].cpu()
        dev["bg_op"] = host.pin_memory() if memory == "pinned" else host

    def call():
        ctx.iterate_device(3, {k: v.data_ptr() for k, v in dev.items()}, pops.data_ptr(), max_iter=2, tol=1e-30)
    try:
        call()
    except RuntimeError as e:
        assert memory == "pageable" and "not a device array" in str(e)
    else:
        assert np.array_equal(pops.cpu().numpy(), want)
    got, _, _, _ = ctx.iterate(cols, fx["ali_pop0"], max_iter=2, tol=1e-30)
    assert np.array_equal(got, want)
    ctx.close()


@pytest.mark.parametrize("every,drop,nd,group", [(1, 1, 80, 16), (6, 0, 80, 16), (7, 3, 257, 8), (9, 2, 513, 4), (30, 1, 513, 4)])
def test_the_last_wavelengths_of_an_uneven_grid(every, drop, nd, group):
    """The wavelengths beyond the last whole group of slots (16, 8, 4 by the number of slices) are the ones that matter
    most, next to the line centres (their order is free): leaving any one of them out of the oracle moves the populations by
    more than the tolerance.  (On the grid in its own order the last ones move them by 1e-8 to 1e-4 only.)"""
    import snapi_b200 as sb
    tol = 1e-3  # as in test_one_iteration_against_the_oracle
    fx = _form(every, drop, nd)
    pop0 = np.asarray(fx["ali_pop0"])
    want = ali_oracle.iterate(ali_oracle.Problem(fx), fx, 0, pop0[0])[0]

    def without(i):
        fy = dict(fx)
        fy["ali_lw"] = np.array(fx["ali_lw"])
        fy["ali_lw"][i] = 0.0
        return np.abs(ali_oracle.iterate(ali_oracle.Problem(fy), fy, 0, pop0[0])[0] / want - 1.0).max()
    lam = np.asarray(fx["ali_lambda"])
    lines = np.asarray(fx["ali_trc"])[np.asarray(fx["ali_tr"])[:, 0] == 0, 0]
    near = sorted({int(i) for c in lines for i in np.argsort(np.abs(lam - c))[:4]}, key=without)
    rest = len(lam) % group
    last = near[len(near) - rest:]
    assert rest and min(without(i) for i in last) > 2 * tol
    order = np.concatenate([np.delete(np.arange(len(lam)), last), last])
    for k in ("lambda", "lw", "fudge"):
        fx["ali_" + k] = np.asarray(fx["ali_" + k])[order]
    fx["ali_sigma"] = np.asarray(fx["ali_sigma"])[:, order]
    for k in ("bgop", "bgem"):
        fx["ali_" + k] = np.asarray(fx["ali_" + k])[:, :, order]
    ctx = sb.api.AliContext.from_fixture(fx)
    pops, rel, iters, st = ctx.iterate(ctx.columns_from_fixture(fx), pop0, max_iter=1, tol=1e-30)
    ctx.close()
    P = ali_oracle.Problem(fx)
    for c in range(len(pops)):
        ref, r, neg = ali_oracle.iterate(P, fx, c, pop0[c])
        assert bool(neg) == (st[c] != 0)
        if not neg:
            assert np.abs(pops[c] / ref - 1.0).max() < tol
            np.testing.assert_allclose(rel[c], r, rtol=tol)
