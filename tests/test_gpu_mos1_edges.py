"""The level-1 kernel's select-based evaluation against the oracle where its
choices can go wrong: voltages on the models' thresholds, signed zeros, huge,
infinite and NaN ones, cards with and without body effect, channel-length
modulation, oxide and junction charge and series resistance, several devices
in parallel, and warps that are not full.  Finite entries meet the parity
tolerance of helpers.py; an entry is infinite or NaN exactly where the
oracle's is."""
import numpy as np
import pytest

from helpers import ATOL_FRAC, RTOL
from xyce_gb300 import abi, engine, netlists

pytestmark = pytest.mark.gpu

CARDS = {
    "plain": dict(VTO=0.7, KP=110e-6),
    "full": dict(VTO=0.6, KP=90e-6, GAMMA=0.5, PHI=0.65, LAMBDA=0.03, TOX=2e-8, CGSO=2e-10, CGDO=3e-10, CGBO=1e-10,
                 CBD=2e-14, CBS=3e-14, RD=10.0, RS=20.0),
    "no_body": dict(VTO=0.7, KP=110e-6, LAMBDA=0.05, TOX=4e-8),
}
SPECIAL = [0.0, -0.0, 0.7, -0.7, 3.5, 4.0, -0.5, 1.2, 2.0, 1e-310, 1e300, np.inf, -np.inf, np.nan]


def _netlist(card, n, nodes, seed, m):
    neg = dict(card, VTO=-card["VTO"])
    nl = netlists.random_mos_netlist(n, nodes, seed=seed, models=(abi.Model(abi.DEV_MOS1, 1, **card),
                                                                  abi.Model(abi.DEV_MOS1, -1, **neg)))
    if m is not None:
        nl.mos1["m"] = np.random.default_rng(seed).choice(m, n).astype(float)
    return nl


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("fma", [0, 1])
@pytest.mark.parametrize("card,n,m", [("plain", 1, None), ("plain", 33, [1, 2]), ("full", 130, None),
                                      ("full", 700, [1, 3]), ("no_body", 257, None)])
def test_mos1_choices(card, n, m, fma, special, gpu_ctx, oracle_lib):
    from oracle.oracle import OracleCircuit
    nl = _netlist(CARDS[card], n, max(4, n // 3), 11, m)
    opt = abi.device_options(fma=fma)
    gpu_ctx.set_options(opt)
    c = engine.Circuit(gpu_ctx, nl)
    gpu_ctx.set_options(abi.device_options())
    params = {t: c.params(t) for t in range(abi.NUM_DEV_TYPES) if nl.count(t)}
    oc = OracleCircuit(nl, params, opt)
    regimes = [abi.load_flags(transient=1, newton_iter=1, pdt=1e11), abi.load_flags(transient=1, newton_iter=0, pdt=1e11),
               abi.load_flags(dcop=1, tranop=1, transient=0, newton_iter=0, init_jct=1),
               abi.load_flags(dcop=1, tranop=1, transient=0, newton_iter=2)]
    for k, flags in enumerate(regimes):
        sol, sta, sto = netlists.random_state(c.n_unknowns, c.n_state, c.n_store, seed=20 + k, vmax=6.0)
        if special:
            rng = np.random.default_rng(30 + k)
            at = rng.integers(0, c.n_unknowns, max(1, c.n_unknowns // 3))
            sol[0][at] = rng.choice(SPECIAL, at.size)
            at = rng.integers(0, c.n_store, max(1, c.n_store // 5))
            for s in sto[:2]:
                s[at] = rng.choice(SPECIAL[:11], at.size)
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
