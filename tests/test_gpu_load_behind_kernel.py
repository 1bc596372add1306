"""A load straight behind a kernel of the caller's that writes its vectors
through the device pointers: the launch starts early (xg_launch.cuh) and must
read everything behind its wait.  Each load gives the bits of the same load
with the vectors uploaded and the stream drained before it."""
import numpy as np
import pytest

from xyce_gb300 import abi, engine

pytestmark = pytest.mark.gpu

IN = (abi.VEC_SOL_NEXT, abi.VEC_SOL_CURR, abi.VEC_STA_CURR, abi.VEC_STO_NEXT, abi.VEC_STO_CURR)
OUT = (abi.VEC_F, abi.VEC_Q, abi.VEC_DFDXDVP, abi.VEC_DQDXDVP, abi.VEC_DFDX, abi.VEC_DQDX,
       abi.VEC_STA_NEXT, abi.VEC_STO_NEXT)


class _Buffer:
    def __init__(self, c, vec):
        self.__cuda_array_interface__ = {"shape": (c.vec_size(vec),), "typestr": "<f8", "version": 3,
                                         "data": (c.device_ptr(vec), False), "strides": None}


def _sequence(c, inputs, flags, stream):
    """The outputs of a load per set of inputs (diodes carry their limited
    voltage from one to the next).  With a stream, a kernel on it writes each
    vector, the last one directly ahead of the load."""
    import torch
    view = {v: torch.as_tensor(_Buffer(c, v), device="cuda") for v in set(IN + OUT)}
    torch.cuda.synchronize()
    res = []
    for x in inputs:
        if stream is None:
            for v in IN:
                c.upload(v, x[v])
            c.ctx.synchronize()
        else:
            dev = {v: torch.from_numpy(x[v]).cuda() for v in IN}
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                for v in IN:
                    torch.mul(dev[v], 1.0, out=view[v])
        c.load(flags)
        c.ctx.synchronize()
        res.append({v: view[v].cpu().numpy() for v in OUT})
    return res


@pytest.mark.parametrize("fma", [0, 1])
@pytest.mark.parametrize("newton_iter", [0, 1])
def test_load_behind_a_writing_kernel(newton_iter, fma, gpu_ctx):
    import torch
    from golden import circuits
    from test_oracle_cpu import _random_mixed
    gpu_ctx.set_options(abi.device_options(fma=fma))
    flags = abi.load_flags(transient=1, newton_iter=newton_iter, pdt=1e11, time=1e-11)
    nl = _random_mixed(32, 257, 64)
    a, b = engine.Circuit(gpu_ctx, nl), engine.Circuit(gpu_ctx, nl)
    inputs = []
    for k in range(20):
        sol, sta, sto = circuits.load_inputs(a.n_unknowns, a.n_state, a.n_store, seed=700 + k)
        inputs.append(dict(zip(IN, (sol[0], sol[1], sta[1], sto[0], sto[1]))))
    want = _sequence(a, inputs, flags, None)
    got = _sequence(b, inputs, flags, torch.cuda.ExternalStream(gpu_ctx.stream()))
    for k, (w, g) in enumerate(zip(want, got)):
        for v in OUT:
            assert np.array_equal(w[v], g[v], equal_nan=True), (k, v)
    a.close()
    b.close()
