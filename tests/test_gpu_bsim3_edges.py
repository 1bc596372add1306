"""The BSIM3 kernel's bit comparisons, one-alternative limiting and
shared-reciprocal quotients against the oracle where they can go wrong:
voltages on the models' thresholds, signed zeros, huge ones and, in the exact
build, infinite and NaN ones; cards of every capMod and mobMod, with and
without series resistance; several devices in parallel; warps that are not
full.  Finite entries meet the parity tolerance of helpers.py; in the exact
build an entry is infinite or NaN exactly where the oracle's is."""
import numpy as np
import pytest

from helpers import ATOL_FRAC, RTOL
from xyce_gb300 import abi, engine, netlists

pytestmark = pytest.mark.gpu

CARDS = {
    "plain": dict(),
    "cap0": dict(CAPMOD=0, MOBMOD=2, XPART=1.0),
    "cap1": dict(CAPMOD=1, MOBMOD=3, XPART=0.5, RSH=5.0),
    "cap2": dict(CAPMOD=2, MOBMOD=1, XPART=0.0, NGATE=1e20),
    "cap3": dict(CAPMOD=3, MOBMOD=2, XPART=1.0, ALPHA0=1e-6, BETA0=25.0),
}
SPECIAL = [0.0, -0.0, 0.7, -0.7, 3.5, 4.0, -0.5, 1.2, 2.0, 1e-310, 8.0]
WILD = [1e300, np.inf, -np.inf, np.nan]


@pytest.mark.parametrize("values", ["ordinary", "special", "wild"])
@pytest.mark.parametrize("card,n,m,fma", [("plain", 1, None, 0), ("plain", 33, [1, 2], 1), ("cap0", 130, None, 0),
                                          ("cap1", 257, [1, 3], 0), ("cap2", 129, None, 1), ("cap2", 129, None, 0),
                                          ("cap3", 300, None, 0), ("cap3", 300, [1, 2], 1)])
def test_bsim3_choices(card, n, m, fma, values, gpu_ctx, oracle_lib):
    from oracle.oracle import OracleCircuit
    if values == "wild" and fma:
        pytest.skip("the FMA build's reciprocals take other paths there")
    nl = netlists.random_mos_netlist(n, max(4, n // 3), dev_type=abi.DEV_BSIM3, seed=12,
                                     models=(abi.Model(abi.DEV_BSIM3, 1, **CARDS[card]),
                                             abi.Model(abi.DEV_BSIM3, -1, **CARDS[card])))
    if m is not None:
        nl.bsim3["m"] = np.random.default_rng(13).choice(m, n).astype(float)
    opt = abi.device_options(fma=fma)
    gpu_ctx.set_options(opt)
    c = engine.Circuit(gpu_ctx, nl)
    gpu_ctx.set_options(abi.device_options())
    params = {t: c.params(t) for t in range(abi.NUM_DEV_TYPES) if nl.count(t)}
    regimes = [abi.load_flags(transient=1, newton_iter=1, pdt=1e11), abi.load_flags(transient=1, newton_iter=0, pdt=1e11),
               abi.load_flags(dcop=1, tranop=1, transient=0, newton_iter=2)]
    for k, flags in enumerate(regimes):
        oc = OracleCircuit(nl, params, opt)
        c.close()
        gpu_ctx.set_options(opt)
        c = engine.Circuit(gpu_ctx, nl)
        gpu_ctx.set_options(abi.device_options())
        sol, sta, sto = netlists.random_state(c.n_unknowns, c.n_state, c.n_store, seed=40 + k, vmax=2.5)
        if values != "ordinary":
            rng = np.random.default_rng(50 + k)
            at = rng.integers(0, c.n_unknowns, max(1, c.n_unknowns // 3))
            sol[0][at] = rng.choice(SPECIAL if values == "special" else SPECIAL + WILD, at.size)
            at = rng.integers(0, c.n_store, max(1, c.n_store // 5))
            for s in sto[:2]:
                s[at] = rng.choice(SPECIAL, at.size)
        c.set_state(sol, sta, sto)
        c.load(flags)
        got = c.outputs()
        want = oc.load(flags, sol, sta, sto)
        for key in ("F", "Q", "dFdxdVp", "dQdxdVp", "dFdx", "dQdx", "sta_next", "sto_next"):
            a, b = np.asarray(got[key]), np.asarray(want[key])
            assert np.array_equal(np.isnan(a), np.isnan(b)), (key, k)
            inf = np.isinf(b)
            assert np.array_equal(np.isinf(a), inf) and np.array_equal(a[inf], b[inf]), (key, k)
            fin = np.isfinite(b)
            if fin.any():
                bound = RTOL * np.abs(b[fin]) + ATOL_FRAC * np.abs(b[fin]).max()
                assert np.all(np.abs(a[fin] - b[fin]) <= bound), (key, k)
    c.close()
