"""The work that users of this framework have it do, as cases that can be timed.

Four kinds of call through the public entry points:
  load    one Newton load of a circuit (Circuit.load): device evaluation and
          stamping of F, Q, the limiter corrections, dF/dx and dQ/dx
  lu      the sparse refactorisation and solve of one Newton step (LU.refactor_solve)
  tran    a whole transient analysis (engine.transient)
  batch   independent transients stepped together (engine.Batch, run_batch)

Sizes come from the benchmark's workloads and the tests, or lie between them.
"""
import math

import numpy as np
import torch

from xyce_gb300 import abi, engine, netlists

VT = 300.15 * (1.3806226e-23 / 1.6021918e-19)   # kT/q at the default temperature
GMIN, IS = 1e-12, 1e-14
LOAD_BYTES = {"mos1": (37 + 27) * 8 + 6 * 4 + 4 * 8, "bsim3": (127 + 55) * 8 + 6 * 4 + 4 * 8}
LOAD_FLOPS = {"mos1": 196 + 48, "bsim3": 1406 + 50}


def listed():
    return [
        # the headline single load: a million BSIM3 devices, contracted arithmetic
        dict(name="load_bsim3_1M", kind="load", model="bsim3", n=1_000_000, nodes=250_000, fma=1),
        # a mid-size ragged BSIM3 circuit with the default options (each product
        # and sum rounded on its own, bit-identical to a serial load)
        dict(name="load_bsim3_30k_default", kind="load", model="bsim3", n=30_001, nodes=7_507, fma=0),
        # a million level-1 devices, contracted arithmetic
        dict(name="load_mos1_1M", kind="load", model="mos1", n=1_000_000, nodes=250_000, fma=1),
        # an ordinary level-1 circuit with the default options
        dict(name="load_mos1_20k_default", kind="load", model="mos1", n=20_011, nodes=5_003, fma=0),
        # the smallest calls: a cell of a few hundred devices of several types,
        # where launches and latency count
        dict(name="load_chain_101", kind="load", model="chain", n=101, nodes=0, fma=1),
        # Newton step of the 200x200 power grid (120,002 unknowns)
        dict(name="lu_grid_200x200", kind="lu", circuit="grid", n=200, m=200, fp32=0),
        # Newton step of a large random-logic block (nearly serial trailing part)
        dict(name="lu_logic_200k", kind="lu", circuit="logic", n=200_000, m=0, fp32=0),
        # the same kind of matrix, smaller, with FP32 factors and refinement
        dict(name="lu_logic_20k_fp32", kind="lu", circuit="logic", n=20_000, m=0, fp32=1),
        # Newton step of the 1,000-stage inverter chain (one block's work)
        dict(name="lu_chain_1000", kind="lu", circuit="chain", n=1000, m=0, fp32=0),
        # a whole transient of that chain: DC point and a rising input edge
        dict(name="tran_chain_1000", kind="tran", circuit="chain", n=1000, m=0, tstop=1e-9, fp32=0, fma=1),
        # a whole transient of a power grid through its breakpoint-dense start,
        # mixed precision
        dict(name="tran_grid_60x60", kind="tran", circuit="grid", n=60, m=60, tstop=10e-12, fp32=1, fma=1),
        # a served batch of Monte-Carlo rings, set-up to results
        dict(name="batch_rings_64", kind="batch", n=64, smallest=5, largest=501, tstop=1e-9, fp32=1),
    ]


def _spread(rng, lo, hi):
    """An integer spread evenly over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["load", "load", "load", "lu", "lu", "lu", "tran", "batch"])
    if kind == "load":
        model = rng.choice(["bsim3", "mos1", "chain"])
        if model == "chain":
            return dict(kind="load", model="chain", n=_spread(rng, 3, 3000), nodes=0, fma=rng.randrange(2))
        n = _spread(rng, 300, 900_000)
        return dict(kind="load", model=model, n=n, nodes=max(16, n // rng.randint(3, 6)), fma=rng.randrange(2))
    if kind == "lu":
        circuit = rng.choice(["grid", "logic", "chain"])
        fp32 = rng.randrange(2)
        if circuit == "grid":
            n = _spread(rng, 12, 180)
            return dict(kind="lu", circuit="grid", n=n, m=max(8, int(n * rng.uniform(0.5, 1.0))), fp32=fp32)
        if circuit == "logic":
            return dict(kind="lu", circuit="logic", n=_spread(rng, 1000, 150_000), m=0, fp32=fp32)
        return dict(kind="lu", circuit="chain", n=_spread(rng, 20, 2000), m=0, fp32=fp32)
    if kind == "tran":
        if rng.randrange(2):
            return dict(kind="tran", circuit="chain", n=_spread(rng, 20, 900), m=0, fp32=rng.randrange(2),
                        tstop=rng.uniform(0.2e-9, 0.9e-9), fma=rng.randrange(2))
        n = _spread(rng, 10, 56)
        return dict(kind="tran", circuit="grid", n=n, m=max(8, int(n * rng.uniform(0.6, 1.0))),
                    tstop=rng.uniform(3e-12, 9e-12), fp32=rng.randrange(2), fma=rng.randrange(2))
    return dict(kind="batch", n=_spread(rng, 2, 60), smallest=5, largest=2 * rng.randint(10, 240) + 1,
                tstop=rng.uniform(0.3e-9, 0.9e-9), fp32=rng.randrange(2))


# ---- circuits ---------------------------------------------------------------------

def _devices(case):
    """Terminals (d, g, s, b), widths and lengths of a random MOSFET netlist.
    The circuit is one of the user's; the state it is loaded at changes."""
    rng = np.random.default_rng([7, 1])
    n = case["n"]
    term = rng.integers(0, case["nodes"], size=(4, n))
    return term, rng.uniform(0.2e-6, 10e-6, n), rng.uniform(0.1e-6, 1e-6, n)


def _random_netlist(case):
    term, w, l = _devices(case)
    n, half = case["n"], case["n"] // 2
    nl = abi.Netlist(case["nodes"])
    t = abi.DEV_MOS1 if case["model"] == "mos1" else abi.DEV_BSIM3
    cards = (dict(VTO=0.7, KP=110e-6), dict(VTO=-0.7, KP=50e-6)) if case["model"] == "mos1" else ({}, {})
    mn, mp = nl.add_model(abi.Model(t, 1, **cards[0])), nl.add_model(abi.Model(t, -1, **cards[1]))
    dev = dict(d=term[0], g=term[1], s=term[2], b=term[3], w=w, l=l,
               model=np.r_[np.full(half, mn), np.full(n - half, mp)])
    setattr(nl, case["model"], dev)
    return nl


def _voltages(case, seed, n):
    """Node voltages U[0, 1.8], and those of the previous Newton iterate."""
    rng = np.random.default_rng([seed, 2])
    v = rng.uniform(0.0, 1.8, n)
    return v, v + rng.normal(0.0, 0.15, n)


def _stored(term, polarity, v):
    """The junction voltages (vbd, vbs, vgs, vds, von) a load keeps per MOSFET."""
    d, g, s, b = v[term]
    vbs, vgs, vds = polarity * (b - s), polarity * (g - s), polarity * (d - s)
    return np.stack([vbs - vds, vbs, vgs, vds, 0.7 * np.broadcast_to(polarity, vds.shape)], 1)


class _DeviceArray:
    """A circuit's device buffer, for torch to view."""

    def __init__(self, circuit, vec):
        self.circuit = circuit
        self.__cuda_array_interface__ = {"shape": (circuit.vec_size(vec),), "typestr": "<f8", "version": 3,
                                         "data": (circuit.device_ptr(vec), False), "strides": None}


def _view(circuit, vec):
    return torch.as_tensor(_DeviceArray(circuit, vec), device="cuda")


OUTPUTS = {"F": abi.VEC_F, "Q": abi.VEC_Q, "dFdxdVp": abi.VEC_DFDXDVP, "dQdxdVp": abi.VEC_DQDXDVP,
           "dFdx": abi.VEC_DFDX, "dQdx": abi.VEC_DQDX, "sta": abi.VEC_STA_NEXT, "sto": abi.VEC_STO_NEXT}


CONTEXT = []


def _context(fma):
    """The program's one context: a circuit keeps the options it was made with."""
    if not CONTEXT:
        CONTEXT.append(engine.Context(0))
    CONTEXT[0].set_options(abi.device_options(fma=fma))
    return CONTEXT[0]


def _circuit(nl, fma):
    return engine.Circuit(_context(fma), nl)


def _netlist(case, seed):
    """(netlist, starting guess of its node voltages)."""
    if case["circuit"] == "grid":
        n, m = case["n"], case["m"]
        sinks = n * m if n * m > 10_000 else n * m // 3
        return netlists.power_grid(n, m, sinks, seed=seed), netlists.power_grid_nodeset(n, m, sinks)
    if case["circuit"] == "logic":
        nl = netlists.random_logic(case["n"], seed=seed)
        return nl, netlists.random_logic_nodeset(nl)
    return netlists.inverter_chain(case["n"]), netlists.inverter_chain_nodeset(case["n"])


def _x0(nl, guess):
    x0 = np.zeros(nl.n_nodes + nl.count(abi.DEV_VSRC))
    x0[: len(guess)] = guess
    return x0


# ---- prepare ------------------------------------------------------------------------

def prepare(case, seed):
    return {"load": _prepare_load, "lu": _prepare_lu, "tran": _prepare_tran, "batch": _prepare_batch}[case["kind"]](
        case, seed)


def _prepare_load(case, seed):
    if case["model"] == "chain":
        nl = netlists.inverter_chain(case["n"])
        c = _circuit(nl, case["fma"])
        term = np.stack([nl.mos1[k] for k in "dgsb"])
        polarity = np.tile([1.0, -1.0], case["n"])
    else:
        nl = _random_netlist(case)
        c = _circuit(nl, case["fma"])
        term = _devices(case)[0]
        polarity = np.where(np.arange(case["n"]) < case["n"] // 2, 1.0, -1.0)
    v, old = _voltages(case, seed, c.n_unknowns)
    c.upload(abi.VEC_SOL_NEXT, np.r_[v, 0.0])
    c.upload(abi.VEC_SOL_CURR, np.r_[old, 0.0])
    sto = _stored(term, polarity, np.r_[old, 0.0]).ravel()
    c.upload(abi.VEC_STO_NEXT, sto)
    c.upload(abi.VEC_STO_CURR, sto)
    # a Newton iteration of a 10 ps time step
    return dict(kind="load", circuit=c, flags=abi.load_flags(transient=1, newton_iter=1, pdt=1e11, time=1e-11),
                out={k: _view(c, vec) for k, vec in OUTPUTS.items()})


def _jacobian(c, nl, guess, seed, h):
    """Newton matrix dQ/dx / h + dF/dx / 2 near the circuit's starting point."""
    rng = np.random.default_rng([seed, 3])
    x = _x0(nl, guess)
    x[: nl.n_nodes] += rng.normal(0.0, 0.05, nl.n_nodes)
    c.upload(abi.VEC_SOL_NEXT, np.r_[x, 0.0])
    c.load(abi.load_flags(transient=1, newton_iter=0, pdt=1.0 / h, time=h))
    c.ctx.synchronize()
    return _view(c, abi.VEC_DQDX) / h + 0.5 * _view(c, abi.VEC_DFDX)


def _update(case, seed, n):
    """A Newton update, the solution of the linear system."""
    return np.random.default_rng([seed, 4]).normal(0.0, 0.05, n)


def _size(case):
    """Unknowns of the case's circuit."""
    if case["circuit"] == "grid":
        nl = case["n"] * case["m"]
        sinks = nl if nl > 10_000 else nl // 3
        return nl + 1 + sinks + sinks + 1
    return case["n"] + 4


def _prepare_lu(case, seed):
    # the circuit is one of the user's, the state it is linearised at changes
    nl, guess = _netlist(case, 7)
    c = _circuit(nl, 1)
    h = 1e-12
    first = _jacobian(c, nl, guess, 0, h)
    lu = engine.LU(c.ctx, c.rowptr, c.colidx, first.cpu().numpy(), abi.LU_FP32 if case["fp32"] else abi.LU_FP64)
    a = _jacobian(c, nl, guess, seed, h)
    values = a.cpu().numpy().astype(np.longdouble)
    x = _update(case, seed, c.n_unknowns)
    b = np.add.reduceat(values * x[c.colidx], c.rowptr[:-1]).astype(np.float64)
    s = dict(kind="lu", circuit=c, lu=lu, values=a, b=torch.from_numpy(b).cuda(),
             x=torch.zeros(c.n_unknowns, dtype=torch.float64, device="cuda"), refine=2 if case["fp32"] else 0)
    torch.cuda.synchronize()
    return s


def _prepare_tran(case, seed):
    nl, guess = _netlist(case, seed)
    if case["circuit"] == "chain":      # another load of the stages for another seed
        nl.cap["value"] = np.random.default_rng([seed, 5]).uniform(8e-15, 12e-15, case["n"])
        record = np.unique(np.linspace(1, nl.n_nodes - 1, 16).astype(np.int32))
    else:
        record = np.unique(np.linspace(0, case["n"] * case["m"] - 1, 16).astype(np.int32))
    return dict(kind="tran", circuit=_circuit(nl, case["fma"]), x0=_x0(nl, guess), record=record,
                tstop=case["tstop"], precision=abi.LU_FP32 if case["fp32"] else abi.LU_FP64,
                refine=1 if case["fp32"] else 0)


def _prepare_batch(case, seed):
    rng = np.random.default_rng([seed, 6])
    stages = 2 * (np.linspace(case["smallest"], case["largest"], case["n"]).astype(int) // 2) + 1
    nls = [netlists.ring_oscillator(int(k), seed=int(rng.integers(1 << 30))) for k in stages]
    return dict(kind="batch", ctx=_context(1), netlists=nls,
                x0=[_x0(nl, netlists.ring_oscillator_nodeset(int(k))) for nl, k in zip(nls, stages)],
                tstop=[case["tstop"]] * case["n"], record=[[1, int(k) // 2 + 1] for k in stages],
                precision=abi.LU_FP32 if case["fp32"] else abi.LU_FP64)


# ---- run ----------------------------------------------------------------------------

def run(s):
    if s["kind"] == "load":
        s["circuit"].load(s["flags"])
        return s["out"]
    if s["kind"] == "lu":
        s["lu"].refactor_solve(s["values"].data_ptr(), s["b"].data_ptr(), s["x"].data_ptr(), s["refine"])
        return s["x"]
    if s["kind"] == "tran":
        t, v, _ = engine.transient(s["circuit"], s["tstop"], 1e-12, s["record"], x0=s["x0"],
                                   precision=s["precision"], n_refine=s["refine"], max_points=4096)
        return {"t": _rows(t, 4096), "v": _rows(v, 4096)}
    b = engine.Batch(s["ctx"], s["netlists"], s["x0"], s["tstop"], s["record"], precision=s["precision"],
                     max_points=2048)
    engine.run_batch(b)
    got = [b.results(i) for i in range(b.n)]
    b.close()
    return {"t": np.stack([_rows(g[0], 2048) for g in got]), "v": np.stack([_rows(g[1], 2048) for g in got])}


def _rows(a, n):
    """An array of n rows that begins with a: inputs differ in how many time
    points they take."""
    out = np.zeros((n,) + a.shape[1:])
    out[: len(a)] = a
    return out


# ---- work ---------------------------------------------------------------------------

def work(case):
    n = case["n"]
    if case["kind"] == "load":
        model, count = ("mos1", 2 * n) if case["model"] == "chain" else (case["model"], n)
        nodes = n if case["model"] == "chain" else case["nodes"]
        entries = 16 * count if case["model"] != "chain" else 4 * count
        return {"bytes": count * LOAD_BYTES[model] + 8 * (4 * nodes + 2 * entries), "flops": count * LOAD_FLOPS[model]}
    if case["kind"] == "lu":
        rows, entries, adds = _matrix(case)
        return {"bytes": 8 * entries + 16 * rows, "flops": 2 * adds}
    if case["kind"] == "tran":
        rows, entries, adds = _matrix(case)
        loads = {"chain": 2 * n * (LOAD_BYTES["mos1"] + 200), "grid": n * case["m"] * 700}[case["circuit"]]
        steps = max(10, int(case["tstop"] / (5e-12 if case["circuit"] == "chain" else 1e-13)))
        return {"bytes": steps * (8 * entries + 16 * rows + loads), "flops": steps * (2 * adds + 500 * rows)}
    rings = n * (case["smallest"] + case["largest"]) // 2
    steps = max(10, int(case["tstop"] / 5e-12))
    return {"bytes": steps * rings * 2 * (LOAD_BYTES["mos1"] + 200), "flops": steps * rings * 2 * 500}


def _matrix(case):
    """About how many rows and entries the case's Newton matrix has, and how
    many multiply-adds its elimination and solves need."""
    if case["circuit"] == "grid":
        rows = _size(case)
        return rows, 4 * rows, 90 * rows
    if case["circuit"] == "logic":
        return case["n"] // 2, 4 * case["n"], 100 * case["n"]
    return case["n"] + 4, 4 * case["n"], 40 * case["n"]


# ---- exact --------------------------------------------------------------------------

def exact(case, seed):
    if case["kind"] == "lu" and case["circuit"] != "logic":
        return _update(case, seed, _size(case))
    if case["kind"] == "lu":
        # the right-hand side was made from this solution in extended precision
        return _update(case, seed, _logic_size(case["n"]))
    if case["kind"] == "load" and case["model"] == "mos1":
        return _exact_mos1(case, seed)
    return None


def _logic_size(n_mos):
    """Unknowns of the random-logic circuit (seed 7): supply and inputs, one
    node per inverter and two per two-input gate, and a current per source."""
    rng = np.random.default_rng(7)
    made = nodes = 0
    while made < n_mos:
        k = int(rng.integers(0, 3))
        made += 2 if k == 0 else 4
        nodes += 1 if k == 0 else 2
    return 1 + 200 + nodes + 201


def _limvds(new, old):
    hi = np.where(new > old, np.minimum(new, 3.0 * old + 2.0), np.where(new < 3.5, np.maximum(new, 2.0), new))
    lo = np.where(new > old, np.minimum(new, 4.0), np.maximum(new, -0.5))
    return np.where(old >= 3.5, hi, lo)


def _fetlim(new, old, vto):
    high = np.abs(2 * (old - vto)) + 2
    low, edge, step = high / 2 + 2, vto + 3.5, new - old
    strong = np.where(step <= 0, np.where(new >= edge, np.where(-step > low, old - low, new), np.maximum(new, vto + 2)),
                      np.where(step >= high, old + high, new))
    on = np.where(old >= edge, strong, np.where(step <= 0, np.maximum(new, vto - 0.5), np.minimum(new, vto + 4)))
    off = np.where(step <= 0, np.where(-step > high, old - high, new),
                   np.where(new <= vto + 0.5, np.where(step > low, old + low, new), vto + 0.5))
    return np.where(old >= vto, on, off)


def _pnjlim(new, old, crit):
    with np.errstate(all="ignore"):
        arg = 1 + (new - old) / VT
        up = np.where(old > 0, np.where(arg > 0, old + VT * np.log(arg), crit), VT * np.log(new / VT))
    return np.where((new > crit) & (np.abs(new - old) > 2 * VT), up, new)


def _exact_mos1(case, seed):
    """Shichman-Hodges MOSFETs without body effect, channel-length modulation
    or charge, their voltages limited against the previous iterate's."""
    term, w, l = _devices(case)
    n, nodes = case["n"], case["nodes"]
    p = np.where(np.arange(n) < n // 2, 1.0, -1.0)
    beta = np.where(p > 0, 110e-6, 50e-6) * w / l
    v, before = _voltages(case, seed, nodes)
    vbd0, vbs0, vgs0, vds0, von = _stored(term, p, before).T
    d, g, s, b = v[term]
    vbs1, vgs1, vds1 = p * (b - s), p * (g - s), p * (d - s)
    vbd1, vgd1 = vbs1 - vds1, vgs1 - vds1
    on = p * von
    crit = VT * math.log(VT / (math.sqrt(2.0) * IS))
    # limiting, forward (vds0 >= 0) and reverse
    f = _fetlim(vgs1, vgs0, on)
    fd = _limvds(f - vgd1, vds0)
    r = _fetlim(vgd1, vgs0 - vds0, on)
    rd = -_limvds(-(vgs1 - r), -vds0)
    vgs, vds = np.where(vds0 >= 0, f, r + rd), np.where(vds0 >= 0, fd, rd)
    vbs = np.where(vds >= 0, _pnjlim(vbs1, vbs0, crit), _pnjlim(vbd1, vbd0, crit) + vds)
    vbd, vgd = vbs - vds, vgs - vds
    # junctions
    gb, cb = {}, {}
    for k, u in (("s", vbs), ("d", vbd)):
        e = np.exp(np.minimum(100.0, np.maximum(u, 0.0) / VT))
        gb[k] = np.where(u <= 0, IS / VT + GMIN, IS * e / VT + GMIN)
        cb[k] = np.where(u <= 0, (IS / VT + GMIN) * u, IS * (e - 1) + GMIN * u)
    # channel
    forward = vds >= 0
    size = np.abs(vds)
    over = np.where(forward, vgs, vgd) - 0.7
    sat, live = over <= size, over > 0
    i = np.where(live, np.where(sat, 0.5 * beta * over**2, beta * size * (over - 0.5 * size)), 0.0)
    gm = np.where(live, np.where(sat, beta * over, beta * size), 0.0)
    gds = np.where(live & ~sat, beta * (over - size), 0.0)
    gm = np.where(forward, gm, -gm)
    i = np.where(forward, p * i, -p * i)
    ns, rs = np.where(forward, gm, 0.0), np.where(forward, 0.0, -gm)
    D, G, S, B = term

    def total(*parts):
        return np.r_[sum(np.bincount(at, what, nodes) for at, what in parts), 0.0]

    fvec = total((B, p * (cb["s"] + cb["d"])), (D, -(p * cb["d"] - i)), (S, -(p * cb["s"] + i)))
    dg = np.where(forward, vgs - vgs1, vgd - vgd1)
    us, ud = (gb["s"] - GMIN) * (vbs - vbs1), (gb["d"] - GMIN) * (vbd - vbd1)
    chan = gds * (vds - vds1) + gm * dg
    lim = total((B, p * (ud + us)), (D, p * (chan - ud)), (S, p * (-us - chan)))
    # the matrix: every pair of a device's four terminals is in the pattern
    zero = np.zeros(n)
    val = {(3, 3): gb["s"] + gb["d"], (3, 0): -gb["d"], (3, 2): -gb["s"], (0, 1): gm, (0, 3): -gb["d"],
           (0, 0): gds + gb["d"] + rs, (0, 2): -gds - ns, (2, 1): -gm, (2, 3): -gb["s"], (2, 0): -(gds + rs),
           (2, 2): gds + gb["s"] + ns}
    at = np.concatenate([term[a].astype(np.int64) * nodes + term[c] for a in range(4) for c in range(4)])
    _, place = np.unique(at, return_inverse=True)
    dfdx = np.bincount(place.ravel(), np.concatenate([val.get((a, c), zero) for a in range(4) for c in range(4)]))
    sto = np.stack([vbd, vbs, vgs, vds, 0.7 * p], 1).ravel()
    return {"F": fvec, "Q": None, "dFdxdVp": lim, "dQdxdVp": None, "dFdx": dfdx, "dQdx": None, "sta": None, "sto": sto}
