"""The node build's march on table sets that take its other branches, against the FP64 oracle: the
reduced Newton system with 6 unknowns (the widest that a group of lanes takes; the Fe I 6300 set has 5)
and with 9, and more bound-free edges at the hydrostatic wavelength than the compact opacity holds (one
thread per march both), and partition functions whose asymptotic terms change form within a column;
and batches around the sizes where the march's launch shape and the order of launches change.

Tolerances as for the Fe I 6300 set (tests/test_eos.py): Nt 1e-10 (FP64, the same path of iterates),
records 3e-7 (their float32 rounding and the H- factors' products of rounded n_e and n_H), tangents
2e-5 of each field's scale (5 K differences of solutions stopped at 1e-4)."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark_gpu = pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")
pytestmark = [pytest.mark.gpu, pytestmark_gpu]


def _forms(eos, form):
    d = {k: np.array(v) for k, v in eos.items()}
    if form.startswith("unknowns"):  # further diatomic molecules of atoms that are in none
        extra = {"unknowns6": [6], "unknowns9": [5, 6, 7, 8]}[form]  # Si; Ca, Si, Al, Fe with oxygen
        mi, mc = d["mol_i"], d["mol_coef"]
        co = next(i for i in range(len(mi)) if mi[i, 0] == 2 and set(mi[i, 1:3]) == {2, 4})
        for a in extra:
            row, coef = mi[co].copy(), mc[co].copy()
            row[1:3] = (a, 4)
            coef[0] += 1.0  # a tenth of CO's binding
            mi, mc = np.vstack([mi, row]), np.vstack([mc, coef])
        d["mol_i"], d["mol_coef"] = mi, mc
        d["meta"] = d["meta"].copy()
        d["meta"][1] = len(mi)
    elif form == "far_terms":  # l above z f n_e^(-1/6) in the deep layers only, and for some terms only
        d["pf_ll"] = d["pf_ll"] * np.where(d["pf_ll"] > 5.5, 14.0, 1.0)
    else:  # many_edges: ten neutral iron levels with edges at the hydrostatic wavelength
        fe = 8
        for l in range(4, 10):
            d["lev"][fe, 0, l] = d["lev"][fe, 0, l - 4]
            d["lev"][fe, 0, l, 1] += 1e-13 * (l + 1)
        d["lev_n"][fe, 0] = 10
        d["lev"][fe, 0, :10, 2] = 1e-18 * (1.0 + np.arange(10))
    return d


@pytest.mark.gpu
@pytestmark_gpu
@pytest.mark.parametrize("start", ["cold", "continue"])
@pytest.mark.parametrize("form", ["unknowns6", "unknowns9", "far_terms", "many_edges"])
def test_gpu_build_other_table_forms_vs_oracle(oracle_lib, eos3, config3, form, start):
    import eos_oracle as eo
    import snapi_b200 as sb
    from snapi_b200.eos_tables import EosTables
    d = _forms(eos3, form)
    t, base = EosTables(d), EosTables(eos3)
    lam0, mass = config3["line_const"][:, 0].copy(), config3["line_const"][:, 3].copy()
    ctx = sb.Context.from_fixture(config3)
    ctx.eos_set(EosTables(d))
    ctx.eos_chem_start(sb.api.CHEM_START_COLD if start == "cold" else sb.api.CHEM_START_CONTINUE)
    nodes = config3["nodes"][:3]
    rec, tan, nt, status = ctx.build_records(nodes, tangents=True, want_nt=True)
    old = eo.set_chem_start(eo.CHEM_START_COLD if start == "cold" else eo.CHEM_START_CONTINUE)
    try:
        for p in range(nodes.shape[0]):
            _, Nt, ro, st = eo.build(t, lam0, mass, nodes[p])
            assert st == status[p]
            _, Nt0, _, _ = eo.build(base, lam0, mass, nodes[p])
            assert np.abs(Nt / Nt0 - 1).max() > 1e-9  # the form does change the column
            np.testing.assert_allclose(nt[p], Nt, rtol=1e-10)
            np.testing.assert_allclose(rec[p], ro, rtol=3e-7, atol=0)
            if start == "cold":
                to, _ = eo.tangents(t, lam0, mass, nodes[p])
                scale = np.maximum(np.abs(to).max(axis=1, keepdims=True), 1e-6 * np.abs(ro).max(axis=0))
                assert (np.abs(tan[p] - to) / scale).max() < 2e-5
    finally:
        eo.set_chem_start(old)
    ctx.close()


@pytest.mark.gpu
@pytestmark_gpu
@pytest.mark.parametrize("npix", [1, 3, 5, 33, 789, 790])
def test_gpu_build_is_the_same_in_every_batch(eos3, config3, npix):
    """A pixel's records, tangents and densities do not depend on the batch it is in: 1 to 33 pixels leave
    warps and CTAs partly empty, 789 x 9 marches are the last that are all resident (other registers and
    one record launch), and with inactive pixels among them."""
    import snapi_b200 as sb
    from snapi_b200.eos_tables import EosTables
    ctx = sb.Context.from_fixture(config3, max_batch=800)
    ctx.eos_set(EosTables(eos3))
    nodes = config3["nodes"]
    rec0, tan0, nt0, st0 = ctx.build_records(nodes, want_nt=True)
    idx = np.arange(npix) % nodes.shape[0]
    active = (np.arange(npix) % 7 != 3).astype(np.int32)
    rec, tan, nt, st = ctx.build_records(nodes[idx], active=active, want_nt=True)
    on = active != 0
    np.testing.assert_array_equal(rec[on], rec0[idx][on])
    np.testing.assert_array_equal(tan[on], tan0[idx][on])
    np.testing.assert_array_equal(nt[on], nt0[idx][on])
    assert not rec[~on].any() and not tan[~on].any()
    ctx.close()


@pytest.mark.parametrize("start,npix", [("cold", 2440), ("cold", 2450), ("continue", 4440), ("continue", 4450)])
def test_gpu_build_is_the_same_on_both_sides_of_the_march_rule(eos3, config3, start, npix):
    """Around the batch sizes (marches = 9 per pixel; 22000 and 40000) from which a march is one thread's."""
    import snapi_b200 as sb
    from snapi_b200.eos_tables import EosTables
    ctx = sb.Context.from_fixture(config3, max_batch=800)
    ctx.eos_set(EosTables(eos3))
    ctx.eos_chem_start(sb.api.CHEM_START_COLD if start == "cold" else sb.api.CHEM_START_CONTINUE)
    nodes = config3["nodes"]
    rec0, tan0, nt0, st0 = ctx.build_records(nodes, want_nt=True)
    idx = np.arange(npix) % nodes.shape[0]
    rec, tan, nt, st = ctx.build_records(nodes[idx], want_nt=True)
    np.testing.assert_array_equal(rec, rec0[idx])
    np.testing.assert_array_equal(tan, tan0[idx])
    np.testing.assert_array_equal(nt, nt0[idx])
    np.testing.assert_array_equal(st, st0[idx])
    ctx.close()


@pytest.mark.gpu
@pytestmark_gpu
@pytest.mark.parametrize("start,npix,tangents", [("cold", 13000, False), ("cold", 13001, False), ("continue", 6000, True)])
def test_gpu_build_of_large_batches_is_that_of_small_ones(eos3, config3, start, npix, tangents):
    """Records only from the cold start on both sides of 13000 marches; 54000 marches, more than are resident at once,
    from the continued start."""
    import snapi_b200 as sb
    from snapi_b200.eos_tables import EosTables
    ctx = sb.Context.from_fixture(config3, max_batch=800)
    ctx.eos_set(EosTables(eos3))
    ctx.eos_chem_start(sb.api.CHEM_START_COLD if start == "cold" else sb.api.CHEM_START_CONTINUE)
    nodes = config3["nodes"]
    idx = np.arange(npix) % nodes.shape[0]
    for got, want in zip(ctx.build_records(nodes[idx], tangents=tangents, want_nt=True),
                         ctx.build_records(nodes, tangents=tangents, want_nt=True)):
        if got is not None:
            np.testing.assert_array_equal(got, want[idx])
    ctx.close()
