"""Resident runs longer than one launch: a launch holds its SMs for at most 1024 ticks, and the launches of
a run give the results of the kernels of a tick, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RHO, SIG, MU = 0.97, 0.15, -1.0


def _series(T, seed):
    import torch
    from gpubpf import dgp
    return torch.tensor(np.asarray(dgp.matched_series(T, RHO, SIG, MU, seed)[1], dtype=np.float32), device="cuda")


@pytest.mark.parametrize("ticks,launches", [(1024, 1), (1025, 2), (2500, 3)])
def test_device_run_releases_the_gpu_between_launches(bpf, ticks, launches):
    import torch
    y = _series(ticks, 5)
    out = []
    for fused in (True, False):
        rec = torch.zeros(ticks * 40, dtype=torch.uint8, device="cuda")
        f = bpf.GpuBpf(70001, RHO, SIG, MU, seed=3, ess_threshold=0.5)
        f.set_fused_small(fused)
        n0 = f._lib.gpu_bpf_launch_count()
        f.step_many_device(y.data_ptr(), ticks, rec.data_ptr())
        if fused:
            assert f._lib.gpu_bpf_launch_count() - n0 == launches
        torch.cuda.synchronize()             # the run is on the filter's own stream
        out.append((rec.cpu().numpy().tobytes(), bytes(f.get_particles())))
        f.close()
    assert out[0] == out[1]


@pytest.mark.parametrize("every", [0, 7])
def test_tape_of_several_launches(bpf, every):
    """A tape whose ticks, checkpoints and kept particles cross a launch: that of the three-kernel ticks."""
    T, N = 1100, 5000
    y = _series(T, 6)
    out = []
    for fault in (0, 4):                     # 4: the resident launch is refused
        tape = bpf.GradTape(N, T, checkpoint_every=every)
        assert tape._lib.gpu_bpf_grad_debug_resident(tape._h, fault, 0, 2000.0) == 0
        n0 = tape._lib.gpu_bpf_launch_count()
        ll = tape.forward((MU, RHO, SIG), y, seed=4).item()
        n = tape._lib.gpu_bpf_launch_count() - n0
        assert n == (4 if fault == 0 else 2 + 3 * T)
        out.append((ll, tape.backward().cpu().numpy().tobytes(), [bytes(r) for r in tape.records()],
                    [tape.children(t).tobytes() for t in (0, 1023, 1024, T - 2)]))
        tape.close()
    assert out[0] == out[1]


@pytest.mark.parametrize("N,launches", [(4096, 2), (70001, 17)])
def test_long_device_run_stays_on_the_chip(bpf, N, launches):
    """More ticks than a graph of single ticks is built for: still the runs' launches, and where the
    resident one is refused, tick by tick with the same results."""
    import torch
    T = 16385
    y = _series(T, 5)
    out = []
    for fused, fault in ((True, 0), (True, 4), (False, 0)):
        rec = torch.zeros(T * 40, dtype=torch.uint8, device="cuda")
        f = bpf.GpuBpf(N, RHO, SIG, MU, seed=3, ess_threshold=0.5)
        f.set_fused_small(fused)
        assert f._lib.gpu_bpf_debug_resident(f._s, fault, 0, 2000.0) == 0
        n0 = f._lib.gpu_bpf_launch_count()
        f.step_many_device(y.data_ptr(), T, rec.data_ptr())
        n = f._lib.gpu_bpf_launch_count() - n0
        if fused and (fault == 0 or N <= 65536):
            assert n == launches
        else:
            assert n >= 2 * T
        torch.cuda.synchronize()
        out.append((rec.cpu().numpy().tobytes(), bytes(f.get_particles())))
        f.close()
    assert out[0] == out[1] == out[2]
