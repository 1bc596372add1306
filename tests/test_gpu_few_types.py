"""Loads of circuits with several device types, evaluated in one launch when
they are small and in a launch per type otherwise: against the oracle on both
sides of that line (2,432 blocks of 32 instances), and where a type's last
block is full, one short or one over."""
import pytest

from helpers import compare
from test_gpu_load import _gpu_run, _oracle
from xyce_gb300 import abi, engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fma", [0, 1])
@pytest.mark.parametrize("n", [8, 31, 32, 33, 257, 4096, 120_000])
def test_mixed_types_match_oracle(n, fma, gpu_ctx, oracle_lib):
    from golden import circuits
    from test_oracle_cpu import _random_mixed
    nl = _random_mixed(32, n, max(4, n // 4))
    opt = abi.device_options(fma=fma)
    params = {t: engine.setup_params(nl, t, opt) for t in range(abi.NUM_DEV_TYPES) if nl.count(t)}
    oc = _oracle(nl, opt, params)
    loads = []
    for k, fl in enumerate(circuits.FLAG_SEQUENCE):
        flags = abi.load_flags(**{**dict(transient=0), **fl})
        loads.append((flags, circuits.load_inputs(oc.n_unknowns, oc.n_state, oc.n_store, seed=600 + k)))
    outs = _gpu_run(gpu_ctx, nl, opt, loads)
    for k, (flags, ins) in enumerate(loads):
        rep, bad = compare(outs[k], oc.load(flags, *ins), exact=False)
        assert not bad, (n, fma, k, bad)
