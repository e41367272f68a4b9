"""GPU parity of the fused FP64 rates + Jacobian kernel against the oracle.

Tolerances (FP64):
  * net production rates: |gpu - oracle| <= 1e-12 * (create + destroy)
    (the magnitude net = create - destroy cancels from; 1e-12 relative when
    there is no cancellation);
  * Jacobian entries: |gpu - oracle| <= 1e-12 * (sum of |terms| of the entry);
    for the forward-difference temperature column the terms are those of both
    right-hand sides divided by the temperature step;
  * the sparsity pattern is compared bit-exactly (tests/test_loader.py).
Also against the reference library's own outputs (tests/golden, generated by
tests/golden/make_golden.py from oracle/_ref).
"""
import numpy as np
import pytest

from conftest import golden, have_gpu, oracle_tables, scaled_err, synth

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.fixture(scope="module")
def torch():
    if not have_gpu():
        pytest.skip("no CUDA device")
    import torch
    return torch


def _run(torch, pm, T, P, Y, ld=None, want_ydot=False):
    """Species-major device call; returns reactor-major numpy (wdot, jac, ydot)."""
    n = T.shape[0]
    ld = ld or n
    dev = torch.device("cuda")
    Tt = torch.zeros(ld, dtype=torch.float64, device=dev)
    Pt = torch.zeros(ld, dtype=torch.float64, device=dev)
    Yt = torch.zeros((pm.nsp, ld), dtype=torch.float64, device=dev)
    Tt[:n] = torch.from_numpy(T)
    Pt[:n] = torch.from_numpy(P)
    Yt[:, :n] = torch.from_numpy(np.ascontiguousarray(Y.T))
    sentinel = -7.25
    W = torch.full((pm.nsp, ld), sentinel, dtype=torch.float64, device=dev)
    J = torch.full((pm.nnz, ld), sentinel, dtype=torch.float64, device=dev)
    D = torch.full((pm.nsp + 1, ld), sentinel, dtype=torch.float64, device=dev) if want_ydot else None
    pm.rates_jac(Tt, Pt, Yt, W, J, D, n=n)
    torch.cuda.synchronize()
    if ld > n:  # padding columns untouched
        assert torch.all(W[:, n:] == sentinel) and torch.all(J[:, n:] == sentinel)
    out = (W[:, :n].T.cpu().numpy(), J[:, :n].T.cpu().numpy())
    return out + ((D[:, :n].T.cpu().numpy(),) if want_ydot else (None,))


def _check(pm, ot, T, P, Y, w, j):
    wo, jo, ws, js = ot.batch_rates_jac_scaled(T, P, Y)
    ew, ej = scaled_err(w, wo, ws), scaled_err(j, jo, js)
    assert ew < TOL, f"wdot scaled error {ew:.3e}"
    assert ej < TOL, f"jacobian scaled error {ej:.3e}"
    return ew, ej


@pytest.mark.parametrize("name", ["c1_h2", "c2_53"])
def test_rates_jac_vs_oracle(torch, name, mech_dir):
    import zerork_b200 as zb
    from zerork_b200 import mechgen
    g, (m, t) = synth(name, mech_dir)
    pm = zb.Mechanism(m, t)
    ot = oracle_tables(pm)
    T, P, Y = mechgen.rate_states(g, 300, seed=13)
    w, j, _ = _run(torch, pm, T, P, Y)
    _check(pm, ot, T, P, Y, w, j)


@pytest.mark.parametrize("ts,v,warps,gws,stage", [
    (8, 1, 4, False, False), (8, 2, 8, False, False), (8, 4, 16, False, False),
    (16, 1, 8, False, False), (16, 2, 8, False, False), (16, 4, 4, False, False),
    (32, 1, 8, False, False), (32, 2, 4, False, False), (32, 4, 8, False, False),
    (16, 2, 8, True, False), (8, 1, 16, True, False), (32, 4, 1, True, False),
    (16, 2, 16, False, True), (16, 1, 16, False, True), (8, 2, 8, False, True),
    (16, 2, 8, True, True), (16, 2, 8, False, "two"), (8, 1, 8, False, "two"), (16, 4, 4, True, "two"),
    (32, 1, 32, False, False), (16, 1, 32, True, False), (8, 1, 32, False, True), (16, 1, 32, True, True),
    (16, 2, 16, True, True), (8, 1, 2, True, "two")])
def test_launch_mappings(torch, ts, v, warps, gws, stage, mech_dir):
    """Every tile/CTA mapping (shared or global workspace, mechanism tables
    staged in shared memory or read from global memory, one or two resident
    CTAs per SM) gives the same answer."""
    import zerork_b200 as zb
    from zerork_b200 import mechgen
    g, (m, t) = synth("c2_53", mech_dir)
    pm = zb.Mechanism(m, t)
    try:
        pm.set_launch(ts, v, warps, gws, grid=7 if gws else 0, stage=stage is True,
                      two_ctas=stage == "two")
    except zb.ZeroRKError:
        pytest.skip("mapping does not fit in shared memory")
    ot = oracle_tables(pm)
    T, P, Y = mechgen.rate_states(g, 77, seed=3)
    w, j, _ = _run(torch, pm, T, P, Y, ld=80)
    _check(pm, ot, T, P, Y, w, j)


def test_launch_flags_are_not_ignored(torch, mech_dir):
    """Staged tables that cannot be staged are refused: with tiles of 32 states
    at the call, with tables larger than shared memory when they are asked for,
    whatever the workspace."""
    import zerork_b200 as zb
    from zerork_b200 import mechgen
    g, (m, t) = synth("c1_h2", mech_dir)
    pm = zb.Mechanism(m, t)
    T, P, Y = mechgen.rate_states(g, 40, seed=3)
    for gws in (False, True):
        pm.set_launch(32, 1, 8, gws, grid=3 if gws else 0, stage=True)
        with pytest.raises(zb.ZeroRKError):
            _run(torch, pm, T, P, Y)
    pm.set_launch(32, 1, 8)
    w, j, _ = _run(torch, pm, T, P, Y)
    _check(pm, oracle_tables(pm), T, P, Y, w, j)
    _, (m, t) = synth("c3_160", mech_dir)
    with pytest.raises(zb.ZeroRKError):
        zb.Mechanism(m, t).set_launch(16, 2, 8, True, grid=7, stage=True)


@pytest.mark.parametrize("name", ["c1_h2", "c2_53"])
def test_rates_jac_vs_reference_golden(torch, name, mech_dir):
    """Against the reference library's own rates (committed fixture)."""
    import zerork_b200 as zb
    g, (m, t) = synth(name, mech_dir)
    gd = golden(name)
    pm = zb.Mechanism(m, t)
    ot = oracle_tables(pm)
    w, j, _ = _run(torch, pm, gd["T"], gd["P"], gd["Y"])
    _, _, ws, js = ot.batch_rates_jac_scaled(gd["T"], gd["P"], gd["Y"])
    assert scaled_err(w, gd["wdot"], ws) < TOL
    assert scaled_err(j, gd["jac"], js) < TOL


def test_autotune_keeps_results(torch, mech_dir):
    import zerork_b200 as zb
    from zerork_b200 import mechgen
    g, (m, t) = synth("c1_h2", mech_dir)
    pm = zb.Mechanism(m, t)
    T, P, Y = mechgen.rate_states(g, 999, seed=4)
    dev = torch.device("cuda")
    Td, Pd = torch.from_numpy(T).to(dev), torch.from_numpy(P).to(dev)
    Yd = torch.from_numpy(np.ascontiguousarray(Y.T)).to(dev)
    W = torch.empty((pm.nsp, 999), dtype=torch.float64, device=dev)
    J = torch.empty((pm.nnz, 999), dtype=torch.float64, device=dev)
    cfg, ms = pm.autotune(Td, Pd, Yd, W, J)
    assert ms > 0 and cfg["ts"] in (8, 16, 32)
    w, j, _ = _run(torch, pm, T, P, Y)
    _check(pm, oracle_tables(pm), T, P, Y, w, j)


def test_edge_sizes_and_clamp(torch, mech_dir):
    """n = 1 and ragged tails; zero / negative / tiny mass fractions exercise the
    min_mass_fraction clamp (reactor_nvector_serial.cpp:629-640)."""
    import zerork_b200 as zb
    from zerork_b200 import mechgen
    g, (m, t) = synth("c2_53", mech_dir)
    pm = zb.Mechanism(m, t)
    ot = oracle_tables(pm)
    T, P, Y = mechgen.rate_states(g, 37, seed=21)
    Y[::3, 5] = 0.0
    Y[1::4, 7] = 1e-40
    Y[2::5, 9] = -1e-35
    for n in (1, 2, 17, 37):
        w, j, _ = _run(torch, pm, T[:n], P[:n], Y[:n], ld=n + 3)
        _check(pm, ot, T[:n], P[:n], Y[:n], w, j)


@pytest.mark.parametrize("name", ["c1_h2", "c2_53"])
def test_limited_rates_of_trace_species(torch, name, mech_dir):
    """At 300 K many reverse rate constants are at the step limit.  With their
    reactants' mass fractions near 1e-163 (two: the product of concentrations
    underflows, the rate does not) and 1e-110 (three) the temperature column
    stays finite and the oracle's."""
    import zerork_b200 as zb
    from zerork_b200 import mechgen
    g, (m, t) = synth(name, mech_dir)
    pm = zb.Mechanism(m, t)
    tab = pm.tables()
    rp, rs = tab["reac_ptr"], tab["reac_spc"]
    T, P, Y = mechgen.rate_states(g, 2 * pm.nstep, seed=29)
    T[:], P[:] = 300.0, 101325.0
    for st in range(pm.nstep):
        for i, y in ((st, 3e-163), (pm.nstep + st, 1e-110)):
            Y[i, rs[rp[st]:rp[st + 1]]] = y
    w, j, _ = _run(torch, pm, T, P, Y)
    assert np.isfinite(w).all() and np.isfinite(j).all()
    _check(pm, oracle_tables(pm), T, P, Y, w, j)


def test_ydot_matches_oracle_rhs(torch, mech_dir):
    import zerork_b200 as zb
    from zerork_b200 import mechgen
    g, (m, t) = synth("c1_h2", mech_dir)
    pm = zb.Mechanism(m, t)
    ot = oracle_tables(pm)
    T, P, Y = mechgen.rate_states(g, 50, seed=8)
    _, _, yd = _run(torch, pm, T, P, Y, want_ydot=True)
    _, _, ydo = ot.batch_rates_jac(T, P, Y, want_jac=False, want_ydot=True)
    np.testing.assert_allclose(yd, ydo, rtol=1e-11, atol=1e-300 + 1e-11 * np.abs(ydo).max())


def test_host_entry_point(torch, mech_dir):
    """zrk_rates_jac_host: host buffers in, host buffers out."""
    import zerork_b200 as zb
    from zerork_b200 import mechgen
    g, (m, t) = synth("c1_h2", mech_dir)
    pm = zb.Mechanism(m, t)
    ot = oracle_tables(pm)
    T, P, Y = mechgen.rate_states(g, 40, seed=9)
    w, j = pm.rates_jac_host(T, P, np.ascontiguousarray(Y.T))
    _check(pm, ot, T, P, Y, w.T, j.T)


def test_full_size_properties(torch, mech_dir):
    """At the benchmark size class (2^17 states here), size-independent checks:
    finite outputs, element conservation of wdot (sum_k a_ek W_k^-1 ... via
    mass: sum_k wdot_k W_k = 0), and agreement with the oracle on a sample."""
    import zerork_b200 as zb
    from zerork_b200 import mechgen
    g, (m, t) = synth("c2_53", mech_dir)
    pm = zb.Mechanism(m, t)
    n = 1 << 17
    T, P, Y = mechgen.rate_states(g, n, seed=2)
    w, j, _ = _run(torch, pm, T, P, Y)
    assert np.isfinite(w).all() and np.isfinite(j).all()
    mw = pm.table("mw")
    ot = oracle_tables(pm)
    idx = np.random.default_rng(0).choice(n, 64, replace=False)
    wo, jo, ws, js = ot.batch_rates_jac_scaled(T[idx], P[idx], Y[idx])
    assert scaled_err(w[idx], wo, ws) < TOL and scaled_err(j[idx], jo, js) < TOL
    mass = np.abs((w * mw).sum(axis=1)) / np.maximum((ws_all := np.abs(w) * mw).sum(axis=1), 1e-300)
    assert np.all(mass < 1e-6)


# The reference's shipped mechanisms (committed fixture copies, tests/golden/mech):
# real H2 (Troe falloff, duplicate and third-body reactions), DME (24 species),
# the n-heptane skeleton (159 species) and the SRI falloff and Troe
# known-answer mechanisms, and the two PLOG test mechanisms (single and
# multiple pressures, duplicate and negative lines).  The oracle is pinned bit-exact to the reference
# library on the same files (tests/test_oracle_pin.py).
SHIPPED = [
    ("h2_v1b_mech.txt", "h2_v1a_therm.txt"),
    ("dme_24_mech.txt", "dme_24_therm.txt"),
    ("heptanesymp159_mec.txt", "heptanesymp_therm.txt"),
    ("sri_reaction.mech", "const_specific_heat.therm"),
    ("troe_test.mech", "const_specific_heat.therm"),
    ("hydrogen_no_falloff.mech", "const_specific_heat.therm"),
    ("plog_test.mech", "plog_test.therm"),
    ("plog_test_ideal.mech", "const_specific_heat.therm"),
]


def _shipped_states(nsp, n, seed):
    rng = np.random.default_rng(seed)
    T = rng.uniform(300.0, 3000.0, n)
    P = 101325.0 * 10 ** rng.uniform(0.0, 2.0, n)
    Y = rng.dirichlet(np.full(nsp, 0.5), size=n)
    return T, P, Y


@pytest.mark.parametrize("mech,therm", SHIPPED)
def test_rates_jac_shipped_mechanisms(torch, mech, therm):
    import zerork_b200 as zb
    from plugin_cases import mech_path
    pm = zb.Mechanism(mech_path(mech), mech_path(therm))
    ot = oracle_tables(pm)
    T, P, Y = _shipped_states(pm.nsp, 203, seed=len(mech))
    w, j, _ = _run(torch, pm, T, P, Y, ld=208)
    _check(pm, ot, T, P, Y, w, j)


def test_sri_parameter_count_variants(torch):
    """SRI with 3 and with 5 parameters (sri_reaction.mech holds one of
    each): the reference applies d and T^e only when they are given
    (rate_const.cpp:998-1003); the loader stores d = 1, e = 0 for the
    3-parameter form, so the kernel's unconditional d * T^e is exact
    (pow(T, 0) = 1), and both reactions match the oracle."""
    import zerork_b200 as zb
    from plugin_cases import mech_path
    pm = zb.Mechanism(mech_path("sri_reaction.mech"), mech_path("const_specific_heat.therm"))
    fo_par = pm.table("fo_par").reshape(-1, 8)
    assert fo_par.shape[0] == 2
    assert fo_par[0, 6] == 1.0 and fo_par[0, 7] == 0.0
    assert fo_par[1, 6] == 0.9 and fo_par[1, 7] == 2.0
    ot = oracle_tables(pm)
    T, P, Y = _shipped_states(pm.nsp, 64, seed=7)
    w, j, _ = _run(torch, pm, T, P, Y)
    _check(pm, ot, T, P, Y, w, j)


@pytest.mark.parametrize("star", ["1e400", "1e308", "1e30", "1e15", "1e-30"])
def test_troe_filler_temperatures(torch, star, tmp_path):
    """Troe temperatures that mechanism files use to switch a term on or off for
    good, the infinite one (a number beyond the range) among them: each term is
    the constant 1 or absent, as in the oracle."""
    import re

    import zerork_b200 as zb
    from plugin_cases import mech_path
    with open(mech_path("troe_test.mech")) as f:
        text = f.read()
    for i in (1, 2):  # T***, T*
        def put(k):
            w = k.group(1).split()
            return "troe / " + " ".join(w[:i] + [star] + w[i + 1:]) + " /"
        (tmp_path / "m.mech").write_text(re.sub(r"(?i)troe\s*/([^/]*)/", put, text))
        pm = zb.Mechanism(str(tmp_path / "m.mech"), mech_path("const_specific_heat.therm"))
        assert np.all(pm.table("fo_par").reshape(-1, 8)[:, 3 + i] == float(star))
        T, P, Y = _shipped_states(pm.nsp, 40, seed=5)
        w, j, _ = _run(torch, pm, T, P, Y)
        _check(pm, oracle_tables(pm), T, P, Y, w, j)


def _conc(pm, T, P, Y):
    mw = pm.table("mw")
    rho = P / (8.314462618e3 * T * np.sum(Y / mw, axis=1))
    return rho[:, None] * Y / mw


def _tc_run(torch, pm, T, Cc, lim=None):
    dev = torch.device("cuda")
    Td = torch.from_numpy(np.ascontiguousarray(T)).to(dev)
    Cd = torch.from_numpy(np.ascontiguousarray(Cc.T)).to(dev)
    Ld = None if lim is None else torch.from_numpy(np.ascontiguousarray(lim)).to(dev)
    out = pm.rates_tc(Td, Cd, Ld)
    torch.cuda.synchronize()
    return [o.T.cpu().numpy() for o in out]


@pytest.mark.parametrize("name", ["h2", "c1_h2", "c2_53"])
def test_rates_tc_vs_reference_golden(torch, name, mech_dir):
    """Rates from (T, C), the mechanism_cuda multi-reactor entry: net,
    create, destroy and rates of progress against the reference library's own
    getReactionRatesLimiter outputs (limit 1e22 on every step) in the
    committed fixtures."""
    import zerork_b200 as zb
    from plugin_cases import mech_path
    if name == "h2":
        pm = zb.Mechanism(mech_path("h2_v1b_mech.txt"), mech_path("h2_v1a_therm.txt"))
    else:
        g, (m, t) = synth(name, mech_dir)
        pm = zb.Mechanism(m, t)
    gd = golden(name)
    Cc = np.array([(gd["P"][i] / (8.314462618e3 * gd["T"][i] * np.sum(gd["Y"][i] / pm.table("mw"))))
                   * gd["Y"][i] / pm.table("mw") for i in range(len(gd["T"]))])
    net, cre, des, rop = _tc_run(torch, pm, gd["T"], Cc, np.full(pm.nstep, 1e22))
    sc = np.abs(gd["cre"]) + np.abs(gd["des"])
    for a, b in ((net, gd["net"]), (cre, gd["cre"]), (des, gd["des"])):
        assert scaled_err(a, b, sc) < TOL
    assert scaled_err(rop, gd["rop"], np.abs(gd["rop"])) < TOL


def test_rates_tc_of_a_large_mechanism(torch, mech_dir):
    """650 species, too many for tiles of 8 states: calls run a state per CTA
    whatever their size (up to one state per SM, and beyond)."""
    import zerork_b200 as zb
    from zerork_b200 import mechgen
    g, (m, t) = synth("c4_650", mech_dir)
    pm = zb.Mechanism(m, t)
    ot = oracle_tables(pm)
    T, P, Y = mechgen.rate_states(g, 1500, seed=23)
    Cc = _conc(pm, T, P, Y)
    lim = np.full(pm.nstep, 1e22)
    for n in (148, 149, 1500):
        net, cre, des, rop = _tc_run(torch, pm, T[:n], Cc[:n], lim)
        for i in (0, n // 2, n - 1):
            on, oc, od, orop = ot.rates(T[i], Cc[i], lim)
            assert scaled_err(net[i], on, np.abs(oc) + np.abs(od)) < TOL
            assert scaled_err(rop[i], orop, np.abs(orop)) < TOL


@pytest.mark.parametrize("mech,therm", SHIPPED)
def test_rates_tc_per_step_limiter(torch, mech, therm):
    """Per-step limits (some steps unlimited, L = 0) and no limiter at all,
    against the oracle's calcRatesFromTC(_StepLimiter) restatement; the host
    entry point gives the same numbers as the device one."""
    import zerork_b200 as zb
    from plugin_cases import mech_path
    pm = zb.Mechanism(mech_path(mech), mech_path(therm))
    ot = oracle_tables(pm)
    T, P, Y = _shipped_states(pm.nsp, 64, seed=3)
    Cc = _conc(pm, T, P, Y)
    rng = np.random.default_rng(1)
    lim = np.where(rng.uniform(size=pm.nstep) < 0.5, 10 ** rng.uniform(-2, 12, pm.nstep), 0.0)
    for L in (lim, None):
        net, cre, des, rop = _tc_run(torch, pm, T, Cc, L)
        for i in range(len(T)):
            on, oc, od, orop = ot.rates(T[i], Cc[i], L)
            s = np.abs(oc) + np.abs(od)
            assert scaled_err(net[i], on, s) < TOL and scaled_err(cre[i], oc, s) < TOL
            assert scaled_err(rop[i], orop, np.abs(orop)) < TOL
    hn, hc, hd, hr = pm.rates_tc_host(T, np.ascontiguousarray(Cc.T), lim)
    dn, dc, dd, dr = _tc_run(torch, pm, T, Cc, lim)
    assert np.array_equal(hn.T, dn) and np.array_equal(hr.T, dr)


@pytest.mark.parametrize("jac", [True, False])
@pytest.mark.parametrize("name,shapes", [
    ("c1_h2", ((1, 1), (31, 33), (4737, 4740))),
    ("c2_53", ((1, 1), (7, 9), (9, 10), (1184, 1184), (1185, 1187), (2369, 2370), (4735, 4735), (4736, 4738))),
    ("c3_160", ((3, 3), (1185, 1186))),
    ("c4_650", ((1, 1), (9, 9), (500, 502)))])  # workspace in global memory
def test_default_mapping_edges(torch, name, shapes, jac, mech_dir):
    """The mapping that a call takes from its size at the edges of every rule
    (tile remainders, waves of 148 tiles, two CTAs per SM), with odd and even
    leading dimensions (16-byte accesses or not) and with clamped states (zero
    mass fractions) among the others: states at the ends, at tile edges and
    clamped ones against the oracle at TOL of its rounding scale, and all of
    them, loosely, against a fixed mapping (1e-9 of the state's largest entry:
    misplaced results, not rounding)."""
    import zerork_b200 as zb
    from zerork_b200 import mechgen
    g, (m, t) = synth(name, mech_dir)
    auto, fixed = zb.Mechanism(m, t), zb.Mechanism(m, t)
    fixed.set_launch(8, 1, 8, name == "c4_650", grid=40 if name == "c4_650" else 0)
    ot = oracle_tables(auto)
    T, P, Y = mechgen.rate_states(g, max(n for n, _ in shapes), seed=17)
    Y[5::7, 3:8 if name == "c1_h2" else 20] = 0.0
    mw = auto.table("mw")
    for n, ld in shapes:
        dev = [torch.from_numpy(a[:n].copy()).cuda() for a in (T, P)]
        Yd = torch.zeros((auto.nsp, ld), dtype=torch.float64, device="cuda")
        Yd[:, :n] = torch.from_numpy(np.ascontiguousarray(Y[:n].T))
        out = []
        for pm in (auto, fixed):
            W = torch.zeros((pm.nsp, ld), dtype=torch.float64, device="cuda")
            J = torch.zeros((pm.nnz, ld), dtype=torch.float64, device="cuda") if jac else None
            D = torch.zeros((pm.nsp + 1, ld), dtype=torch.float64, device="cuda")
            pm.rates_jac(dev[0], dev[1], Yd, W, J, D, n=n)
            out.append([x.cpu().numpy() for x in (W, D, J) if x is not None])
        for a, b in zip(*out):
            assert np.all(a[:, n:] == 0.0)
            assert np.all(np.abs(a - b) <= 1e-9 * np.abs(b).max(axis=0, keepdims=True)), n
        idx = sorted({i for i in (0, 5, 7, 8, 12, 15, 16, 31, 32, n // 2, n - 2, n - 1) if 0 <= i < n})
        if name == "c4_650":
            idx = idx[:3] + idx[-2:]
        wo, jo, ws, js = ot.batch_rates_jac_scaled(T[idx], P[idx], Y[idx])
        assert scaled_err(out[0][0][:, idx].T, wo, ws) < TOL, n
        v = 8314.462618 * T[idx] * (Y[idx] / mw).sum(1) / P[idx]
        assert scaled_err(out[0][1][:-1, idx].T, wo * mw * v[:, None], ws * mw * v[:, None]) < TOL, n
        if jac:
            assert scaled_err(out[0][2][:, idx].T, jo, js) < TOL, n


def test_small_rate_calls(torch, mech_dir):
    """Rates from (T, C) at the edges of the small paths (a state per CTA up to
    one per SM, pinned staging up to 256 KB: 40 states of this mechanism)
    against the general path's tiles; the same operations per state, summed in
    the same order."""
    import zerork_b200 as zb
    from zerork_b200 import mechgen
    g, (m, t) = synth("c2_53", mech_dir)
    pm = zb.Mechanism(m, t)
    T, P, Y = mechgen.rate_states(g, 300, seed=19)
    iw = 1.0 / pm.table("mw")
    C = np.ascontiguousarray((Y * iw * (P / (8314.462618 * T) / (Y * iw).sum(1))[:, None]).T)
    lim = np.full(pm.nstep, 1e22)
    ref = [x.cpu().numpy() for x in pm.rates_tc(torch.from_numpy(T).cuda(), torch.from_numpy(C).cuda(),
                                                torch.from_numpy(lim).cuda())]
    for n in (1, 2, 39, 40, 41, 148, 149):
        got = pm.rates_tc_host(T[:n], np.ascontiguousarray(C[:, :n]), lim)
        dev = pm.rates_tc(torch.from_numpy(T[:n].copy()).cuda(), torch.from_numpy(np.ascontiguousarray(C[:, :n])).cuda(),
                          torch.from_numpy(lim).cuda())
        for a, d, r in zip(got, dev, ref):
            scale = np.abs(ref[1][:, :n]).max(axis=0) + np.abs(ref[2][:, :n]).max(axis=0)
            assert np.all(np.abs(a - r[:, :n]) <= 1e-12 * np.maximum(scale, np.abs(r[:, :n])))
            assert np.array_equal(a, d.cpu().numpy())
