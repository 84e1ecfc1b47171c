"""Kept memory of gradient runs (gpu_bpf_kept_bytes, gpu_bpf_trim_kept): what tapes and batches hold to
avoid recomputing. Its results are those of the recomputing runs, bit for bit; all owners together stay
within their share of the device; it is given back with its owner, on request and when an allocation
would fail."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RHO, SIG, MU = 0.97, 0.15, -1.0
TILE = 4096


def _series(T, seed):
    import torch
    from gpubpf import dgp
    return torch.tensor(np.asarray(dgp.matched_series(T, RHO, SIG, MU, seed)[1], dtype=np.float32), device="cuda")


@pytest.fixture
def base(bpf):
    """Nothing kept by what earlier tests left in the library's caches."""
    bpf.trim_kept()
    assert bpf.kept_bytes() == 0
    yield
    bpf.trim_kept()


@pytest.mark.parametrize("N", [5, 70001, 700001])
def test_tape_gives_back_between_forward_and_backward(bpf, base, N):
    T = 37
    y = _series(T, 6)

    def grads(trim):
        tape = bpf.GradTape(N, T)
        out = []
        for seed in (3, 9):
            out.append(tape.forward((MU, RHO, SIG), y, seed=seed).item())
            if seed == 3:
                held = T * -(-N // TILE) * TILE * 4
                assert bpf.kept_bytes() == held
                if trim:
                    assert bpf.trim_kept() == held
            assert bpf.kept_bytes() == (0 if trim else held)
            out.append(tape.backward().cpu().numpy().tobytes())
        tape.close()
        assert bpf.kept_bytes() == 0
        return out

    assert grads(False) == grads(True)


FILTERS = [
    {"mu": -1.0, "rho": 0.97, "sigma_z": 0.15, "n_particles": 1, "seed": 3},
    {"mu": -0.5, "rho": 0.90, "sigma_z": 0.30, "n_particles": 100, "seed": 4},
    {"mu": -0.9, "rho": 0.93, "sigma_z": 0.20, "n_particles": 1025, "seed": 9, "nu_state": 5.0, "nu_obs": 4.0},
    {"mu": -1.2, "rho": 0.99, "sigma_z": 0.10, "n_particles": 4096, "seed": 5},
    {"mu": -0.8, "rho": 0.95, "sigma_z": 0.25, "n_particles": 5000, "seed": 6, "nu_obs": 5.0},
    {"mu": -1.5, "rho": 0.85, "sigma_z": 0.40, "n_particles": 9000, "seed": 7, "nu_state": 6.0},
    {"mu": -1.0, "rho": 0.97, "sigma_z": 0.20, "n_particles": 16384, "seed": 8},
]


@pytest.mark.parametrize("T", [1, 8, 9, 45])
def test_batch_recomputes_what_it_no_longer_keeps(bpf, base, T):
    """One, whole and partial checkpoint segments (8 ticks): kept and recomputed runs of every size class."""
    import torch
    y = _series(T, 4)
    b = bpf.GpuBpfBatch(FILTERS, ess_threshold=0.0)

    def run():
        ll = torch.zeros(len(FILTERS), dtype=torch.float64, device="cuda")
        g = torch.zeros(len(FILTERS) * 3, dtype=torch.float64, device="cuda")
        b.grad_run(y.data_ptr(), T, ll.data_ptr(), g.data_ptr())
        torch.cuda.synchronize()
        return ll.cpu().numpy().tobytes(), g.cpu().numpy().tobytes()

    kept = run()
    # one slot per filter of each class (1024, 2048, 4096, 8192 and 16384 particles)
    held = T * 4 * (2 * 1024 + 2048 + 4096 + 8192 + 2 * 16384)
    assert bpf.kept_bytes() == held
    assert bpf.trim_kept() == held
    recomputed = run()
    assert bpf.kept_bytes() == 0
    b.close()
    assert kept == recomputed
    assert np.isfinite(np.frombuffer(kept[1])).all()


def test_tapes_together_keep_an_eighth(bpf, base):
    import torch
    N, T = 1 << 20, 1400                     # 5.9 GB kept by each tape that may, as much by its child lists
    y = _series(T, 4)
    tapes, lls = [], []
    for _ in range(5):
        tapes.append(bpf.GradTape(N, T))
        lls.append(tapes[-1].forward((MU, RHO, SIG), y, seed=3).item())
        kept = bpf.kept_bytes()
        assert kept <= (torch.cuda.mem_get_info()[0] + kept) // 8 + (1 << 26)   # (its allocations' rounding)
    assert bpf.kept_bytes() >= T * N * 4
    grads = [t.backward().cpu().numpy().tobytes() for t in tapes]
    assert len(set(lls)) == 1 and len(set(grads)) == 1
    for t in tapes:
        t.close()
    assert bpf.kept_bytes() == 0


def test_allocation_takes_kept_memory(bpf, base):
    """A tape that fits only once another gives back what it keeps is created as it would be without."""
    import torch
    N = 1 << 20
    first = bpf.GradTape(N, 1400)
    y = _series(1400, 4)
    ll = first.forward((MU, RHO, SIG), y, seed=3).item()
    assert bpf.kept_bytes() == 1400 * N * 4
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (2 << 30), dtype=torch.uint8, device="cuda")
    second = bpf.GradTape(N, 700)            # 3.1 GB of 2 GB free
    assert bpf.kept_bytes() == 0
    grad = first.backward().cpu().numpy().tobytes()
    second.close()
    del fill
    torch.cuda.empty_cache()
    assert first.forward((MU, RHO, SIG), y, seed=3).item() == ll
    assert first.backward().cpu().numpy().tobytes() == grad
    first.close()
