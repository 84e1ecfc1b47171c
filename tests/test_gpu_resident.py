"""Resident runs (csrc/bpf_resident.cu): consecutive ticks of a medium filter as one cooperative
launch. The records, ancestors, particles and weights equal the tick-per-launch path's bit for bit
(gpu_bpf_set_fused_small(state, 0) selects that one), so the tolerance is zero."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RHO, SIG, MU = 0.97, 0.15, -1.0
TILE = 4096


def _series(T, seed, outliers=False):
    from gpubpf import dgp
    y = np.asarray(dgp.matched_series(T, RHO, SIG, MU, seed)[1], dtype=np.float32)
    if outliers:                      # a few particles take nearly all of the weight
        y[T // 3] = 40.0
        y[T // 2] = -90.0
    return y


def _device_run(bpf, N, thr, nu_obs, nu_state, y, fused, seeds, anc=False):
    import torch
    T = len(y)
    yd = torch.tensor(y, device="cuda")
    rec = torch.zeros(T * 40, dtype=torch.uint8, device="cuda")
    f = bpf.GpuBpf(N, RHO, SIG, MU, nu_state, nu_obs, 17, ess_threshold=thr)
    f.set_fused_small(fused)
    if anc:
        f.record_ancestors(True)
    out = []
    for seed in seeds:                # the second run replays the captured launch
        f.reset(seed)
        f.step_many_device(yd.data_ptr(), T, rec.data_ptr())
        torch.cuda.synchronize()
        w, te, u23 = f.get_resample_inputs()
        out.append((rec.cpu().numpy().tobytes(), bytes(f.get_particles()), bytes(w), bytes(te), u23,
                    f.get_loglik_total(), f.get_resample_count(), bytes(f.get_ancestors()[1]) if anc else b""))
    f.close()
    return out


# one tile more than the cluster path takes; one, two, three and four tiles a CTA at their edges
@pytest.mark.parametrize("N,thr,nu_obs,nu_state,outliers", [
    (65537, 0.5, 0.0, 0.0, False), (74 * TILE - 1, 0.0, 0.0, 0.0, True), (148 * TILE, 0.5, 5.0, 0.0, False),
    (148 * TILE + 1, 0.0, 0.0, 5.0, False), (1000003, 0.5, 5.0, 5.0, True), (296 * TILE, 0.5, 0.0, 6.0, False),
    (296 * TILE + 5, 0.0, 5.0, 0.0, True), (1500000, 0.5, 0.0, 0.0, False), (592 * TILE, 0.5, 0.0, 0.0, True),
    (592 * TILE - 4097, 0.0, 0.0, 0.0, False)])
def test_resident_run_matches_tick_launches(bpf, N, thr, nu_obs, nu_state, outliers):
    y = _series(60, 9, outliers)
    a = _device_run(bpf, N, thr, nu_obs, nu_state, y, True, (17, 5), anc=True)
    b = _device_run(bpf, N, thr, nu_obs, nu_state, y, False, (17, 5), anc=True)
    assert a == b
    assert a[0] != a[1]


def test_resident_long_run_restages_observations(bpf):
    y = _series(2500, 42)
    assert _device_run(bpf, 100001, 0.5, 0.0, 0.0, y, True, (3,)) == _device_run(bpf, 100001, 0.5, 0.0, 0.0, y, False, (3,))


@pytest.mark.parametrize("N,thr", [(70000, 0.0), (700001, 0.5)])
def test_resident_host_runs_and_single_ticks_interleave(bpf, N, thr):
    """step_many (chunks and a remainder), single steps and a checkpoint between them."""
    y = _series(200, 21).tolist()

    def run(fused):
        f = bpf.GpuBpf(N, RHO, SIG, MU, seed=4, ess_threshold=thr)
        f.set_fused_small(fused)
        recs = f.step_many(y[:70], records=True)
        for v in y[70:73]:
            f.step(v)
            recs.append(f.get_record())
        blob = f.save()
        recs += f.step_many(y[73:], records=True)
        f.load(blob)
        recs += f.step_many(y[73:], records=True)
        parts = bytes(f.get_particles())
        f.close()
        return [bytes(r) for r in recs], parts

    assert run(True) == run(False)


def test_resident_degenerate_tick(bpf):
    """A tick whose every weight underflows: the same records as tick by tick."""
    y = _series(40, 3)
    y[20] = 3e18
    a = _device_run(bpf, 80000, 0.5, 0.0, 0.0, y, True, (17,))
    b = _device_run(bpf, 80000, 0.5, 0.0, 0.0, y, False, (17,))
    assert a == b


@pytest.mark.parametrize("N,nu_obs,nu_state,outliers", [
    (1, 0.0, 0.0, False), (4097, 5.0, 0.0, True), (50000, 0.0, 0.0, False), (148 * TILE + 1, 0.0, 5.0, True),
    (1500000, 5.0, 0.0, False)])
def test_resident_apf_matches_kernel_launches(bpf, N, nu_obs, nu_state, outliers):
    """Auxiliary-filter runs: a filter that records its ancestors keeps the launch per kernel."""
    y = _series(70, 13, outliers).tolist()
    out = []
    for record in (False, True):
        f = bpf.GpuApf(N, RHO, SIG, MU, nu_state, nu_obs, 19)
        f.record_ancestors(record)
        recs = f.step_many(y[:66], records=True)
        recs += f.step_many(y[66:], records=True)
        out.append(([bytes(r) for r in recs], bytes(f.get_particles()), f.get_loglik_total()))
        f.close()
    assert out[0] == out[1]


@pytest.mark.parametrize("N", [3, 65537, 700001, 1300000])
def test_resident_tape_matches_plain_ticks(bpf, N):
    """Child lists, records and checkpoint-driven gradient inputs of a taped run: the ancestors of single
    plain ticks (three kernels), bit for bit, outliers included."""
    import torch
    T = 12
    y = _series(T, 31, True)
    tape = bpf.GradTape(N, T, checkpoint_every=4)
    ll = tape.forward((MU, RHO, SIG), torch.tensor(y, device="cuda"), seed=8).item()
    f = bpf.GpuBpf(N, RHO, SIG, MU, seed=8, ess_threshold=0.0)
    f.set_fused_small(False)
    f.record_ancestors(True)
    recs = tape.records()
    for t in range(T):
        f.step(float(y[t]))
        assert bytes(f.get_record()) == bytes(recs[t])
        np.testing.assert_array_equal(tape.ancestors(t), np.frombuffer(f.get_ancestors()[1], dtype=np.int32))
    assert ll == f.get_record().loglik_total
    g = tape.backward().cpu().numpy()
    ref = tape.replay((MU, RHO, SIG)).cpu().numpy()[1:]
    assert np.max(np.abs(g - ref)) <= 1e-4 * np.max(np.abs(ref))     # the gradient tests' bound
    f.close()
    tape.close()


@pytest.mark.parametrize("N", [5, 70001, 700001])
def test_resident_tape_with_and_without_kept_particles(bpf, N):
    """The default tape keeps every tick's particles, one with an interval recomputes them: equal bits."""
    import torch
    T = 37
    y = torch.tensor(_series(T, 6, True), device="cuda")
    out = []
    for every in (0, 16, 5):
        tape = bpf.GradTape(N, T, checkpoint_every=every)
        for seed in (3, 9):
            out.append((tape.forward((MU, RHO, SIG), y, seed=seed).item(), tape.backward().cpu().numpy().tobytes()))
        tape.close()
    assert out[0:2] == out[2:4] == out[4:6]


def test_resident_runs_on_several_streams_and_threads(bpf):
    """Filters that together need more SMs than there are, running at the same time on their own streams
    from two host threads, beside single ticks of another: each equals its own run alone."""
    import threading
    import torch
    T, sizes = 150, (1000003, 300000, 1500000, 70000)
    y = _series(T, 12)
    yd = torch.tensor(y, device="cuda")
    alone = [_device_run(bpf, n, 0.5, 0.0, 0.0, y, True, (17,))[0][:2] for n in sizes]
    out = {}

    # created beforehand: creating a filter synchronises the device, which no other thread's stream
    # capture survives
    fs = {n: (bpf.GpuBpf(n, RHO, SIG, MU, seed=17, ess_threshold=0.5),
              torch.zeros(T * 40, dtype=torch.uint8, device="cuda")) for n in sizes}
    g = bpf.GpuBpf(200000, RHO, SIG, MU, seed=1)
    g.step(0.1)
    torch.cuda.synchronize()

    def worker(part):
        for _ in range(3):
            for n in part:
                fs[n][0].reset(17)
                fs[n][0].step_many_device(yd.data_ptr(), T, fs[n][1].data_ptr())
        for n in part:
            parts = bytes(fs[n][0].get_particles())   # waits for the filter's stream
            out[n] = parts

    ts = [threading.Thread(target=worker, args=(part,)) for part in (sizes[:2], sizes[2:])]
    for t in ts:
        t.start()
    for v in y[:40]:
        g.step(float(v))
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    out = {n: (fs[n][1].cpu().numpy().tobytes(), p) for n, p in out.items()}
    for f, _ in fs.values():
        f.close()
    g.close()
    assert [out[n] for n in sizes] == alone
