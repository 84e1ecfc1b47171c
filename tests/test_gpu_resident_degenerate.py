"""Ticks whose every weight underflows, or whose log-densities are infinite, inside resident runs of the
auxiliary filter and of gradient tapes: what the kernels of a tick give, bit for bit (a refused resident
launch selects those)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RHO, SIG, MU = 0.97, 0.15, -1.0
REFUSED = 4


def _series(T, at, value):
    from gpubpf import dgp
    y = np.asarray(dgp.matched_series(T, RHO, SIG, MU, 5)[1], dtype=np.float32)
    y[at] = value
    return y


# 3e18: every first-stage weight underflows, second-stage log-weights are finite and huge; 1e30: the density
# of the observation is zero, its logarithm -inf in both stages; on the first tick and inside the run
@pytest.mark.parametrize("at", [0, 20])
@pytest.mark.parametrize("value", [3e18, 1e30])
@pytest.mark.parametrize("N,nu_obs", [(4096, 0.0), (50001, 0.0), (50001, 5.0), (1500000, 0.0)])
def test_auxiliary_run(bpf, N, nu_obs, value, at):
    from gpubpf import _lib
    lib = bpf.load()
    y = _series(40, at, value)
    ya = (C.c_float * 40)(*y.tolist())
    out = []
    for fault in (0, REFUSED):
        f = bpf.GpuApf(N, RHO, SIG, MU, 0.0, nu_obs, 19)
        assert lib.gpu_apf_debug_resident(f._s, fault, 0, 2000.0) == _lib.BPF_OK
        rec = (_lib.BpfTickRecord * 40)()
        rc = lib.gpu_apf_step_many(f._s, ya, 40, None, rec)
        out.append((rc, bytes(rec), bytes(f.get_particles()), np.float64(f.get_loglik_total()).tobytes()))
        f.close()
    assert out[0] == out[1]
    assert out[0][0] in (_lib.BPF_OK, _lib.BPF_ERR_DEGENERATE)
    if nu_obs == 0.0 or value == 1e30:
        assert out[0][0] == _lib.BPF_ERR_DEGENERATE


@pytest.mark.parametrize("value", [3e18, 1e30])
@pytest.mark.parametrize("N", [5000, 70001])
def test_tape(bpf, N, value):
    """The child list of the degenerate tick itself is not written by either."""
    import torch
    T, at = 30, 12
    y = torch.tensor(_series(T, at, value), device="cuda")
    out = []
    for fault in (0, REFUSED):
        tape = bpf.GradTape(N, T)
        assert tape._lib.gpu_bpf_grad_debug_resident(tape._h, fault, 0, 2000.0) == 0
        ll = tape.forward((MU, RHO, SIG), y, seed=8).cpu().numpy().tobytes()
        recs = tape.records()
        out.append((ll, [bytes(r) for r in recs], [tape.children(t).tobytes() for t in range(T - 1) if t != at]))
        assert recs[at].dloglik == -np.inf and not recs[at].resampled
        tape.close()
    assert out[0] == out[1]
