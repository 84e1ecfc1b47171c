"""Resident runs whose CTAs give up waiting: made on purpose by gpu_bpf_debug_resident (a mailbox that gets no
records or no flags, an absent CTA, a limit of 20 ms on the waits), so the kernel returns its status and
no GPU fault is involved. The run must end with BPF_ERR_STATE whichever CTA gave up and however late, and
a reset filter must then run as a new one, bit for bit."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RHO, SIG, MU = 0.97, 0.15, -1.0
TILE = 4096
RECORDS, FLAGS, ABSENT, REFUSED = 1, 2, 3, 4
T = 12


def _series(T, seed):
    from gpubpf import dgp
    return np.asarray(dgp.matched_series(T, RHO, SIG, MU, seed)[1], dtype=np.float32)


def _arm(f, fn, fault=0, mailbox=0, limit_ms=2000.0):
    from gpubpf import _lib
    assert getattr(f._lib, fn)(f._s, fault, mailbox, limit_ms) == _lib.BPF_OK


# The last CTA writes the state and polls mailbox (CTAs - 1) % 16: 18 CTAs of one tile, 123 of two, 148 of four.
# With one tick and no resampling its waits are all answered while CTAs of the mailbox give up.
CASES = [(70000, 1e-6, 1, RECORDS, 0), (70000, 1e-6, 1, RECORDS, 1), (70000, 0.0, T, FLAGS, 5),
         (70000, 0.0, T, RECORDS, 3), (70000, 0.0, T, ABSENT, 0), (1000003, 1e-6, 1, RECORDS, 7),
         (592 * TILE, 1e-6, 1, RECORDS, 15), (592 * TILE, 0.5, T, ABSENT, 0)]


@pytest.mark.parametrize("N,thr,ticks,fault,mailbox", CASES)
def test_run_with_a_wait_given_up_reports_it(bpf, N, thr, ticks, fault, mailbox):
    import torch
    from gpubpf import _lib
    y = _series(T, 9)
    f = bpf.GpuBpf(N, RHO, SIG, MU, seed=3, ess_threshold=thr)
    want = [bytes(r) for r in f.step_many(y.tolist(), records=True)], bytes(f.get_particles())
    yd = torch.tensor(y, device="cuda")
    rec = torch.zeros(T * 40, dtype=torch.uint8, device="cuda")

    f.reset(3)
    _arm(f, "gpu_bpf_debug_resident", fault, mailbox, 20.0)
    f.step_many_device(yd.data_ptr(), ticks, rec.data_ptr())          # reported by the read-backs
    for read in (f.get_record, f.get_particles, f.save, f.get_result):
        with pytest.raises(bpf.BpfError) as e:
            read()
        assert e.value.code == _lib.BPF_ERR_STATE
    assert math.isnan(f.get_loglik_total())
    _arm(f, "gpu_bpf_debug_resident")                                 # a later run does not start on that state
    with pytest.raises(bpf.BpfError) as e:
        f.step_many(y.tolist())
    assert e.value.code == _lib.BPF_ERR_STATE
    f.reset(3)
    assert ([bytes(r) for r in f.step_many(y.tolist(), records=True)], bytes(f.get_particles())) == want
    if ticks > 1:                                                     # and by a host run itself
        _arm(f, "gpu_bpf_debug_resident", fault, mailbox, 20.0)
        f.reset(3)
        with pytest.raises(bpf.BpfError) as e:
            f.step_many(y.tolist())
        assert e.value.code == _lib.BPF_ERR_STATE
    f.close()


@pytest.mark.parametrize("N,tiles", [(70000, 1), (1000003, 2), (592 * TILE, 4)])
def test_last_resampling_with_a_wait_given_up_reports_it(bpf, N, tiles):
    """One tick that resamples, its flags kept from one mailbox after another: the CTAs that poll it give up
    if and only if children of another CTA's particles fall into their slots, which the ancestors of the
    same tick say. The last CTA's own mailbox is left alone, so that its waits are answered."""
    import torch
    from gpubpf import _lib
    y = torch.tensor(_series(T, 9), device="cuda")
    rec = torch.zeros(40, dtype=torch.uint8, device="cuda")
    f = bpf.GpuBpf(N, RHO, SIG, MU, seed=3, ess_threshold=0.0)
    f.record_ancestors(True)
    f.step_many_device(y.data_ptr(), 1, rec.data_ptr())
    owner = np.arange(N) // (tiles * TILE)
    waits = np.unique(owner[np.frombuffer(f.get_ancestors()[1], dtype=np.int32) // (tiles * TILE) != owner])
    assert len(waits) > 0
    seen = set()
    for mailbox in sorted(set(range(16)) - {int(owner[-1]) % 16}):
        _arm(f, "gpu_bpf_debug_resident", FLAGS, mailbox, 20.0)
        f.reset(3)
        f.step_many_device(y.data_ptr(), 1, rec.data_ptr())
        gives_up = bool(np.any(waits % 16 == mailbox))
        seen.add(gives_up)
        if gives_up:
            with pytest.raises(bpf.BpfError) as e:
                f.get_particles()
            assert e.value.code == _lib.BPF_ERR_STATE
        else:
            f.get_particles()
    assert True in seen
    f.close()


@pytest.mark.parametrize("N", [50000, 1500000])
@pytest.mark.parametrize("fault,mailbox", [(RECORDS, 0), (FLAGS, 1), (ABSENT, 0)])
def test_auxiliary_run_with_a_wait_given_up_reports_it(bpf, N, fault, mailbox):
    from gpubpf import _lib
    y = _series(T, 9).tolist()
    f = bpf.GpuApf(N, RHO, SIG, MU, seed=3)
    _arm(f, "gpu_apf_debug_resident", fault, mailbox, 20.0)
    with pytest.raises(bpf.BpfError) as e:
        f.step_many(y)
    assert e.value.code == _lib.BPF_ERR_STATE
    f.close()


def test_rejects_bad_arguments(bpf):
    from gpubpf import _lib
    f = bpf.GpuBpf(70000, RHO, SIG, MU, seed=3)
    for args in ((5, 0, 10.0), (-1, 0, 10.0), (1, -1, 10.0), (1, 16, 10.0), (1, 0, 0.0), (1, 0, 2001.0), (1, 0, math.nan)):
        assert f._lib.gpu_bpf_debug_resident(f._s, *args) == _lib.BPF_ERR_ARG
    f.close()


@pytest.mark.parametrize("every", [0, 4])
@pytest.mark.parametrize("N,ticks,fault,mailbox", [(70001, T, RECORDS, 0), (70001, T, FLAGS, 0), (700001, T, FLAGS, 2),
                                                   (70001, T, ABSENT, 0)])
def test_tape_with_a_wait_given_up_has_no_gradient(bpf, N, ticks, fault, mailbox, every):
    """With and without the particles of every tick kept: NaN from forward and backward, an error from the
    calls that read the tape, and a sound tape from the next forward run."""
    import torch
    from gpubpf import _lib
    y = torch.tensor(_series(ticks, 9), device="cuda")
    theta = (MU, RHO, SIG)

    def clean(tape):
        return tape.forward(theta, y, seed=8).item(), tape.backward().cpu().numpy().tobytes(), bytes(tape.children(0))

    other = bpf.GradTape(N, T, checkpoint_every=every)
    want = clean(other)
    other.close()
    tape = bpf.GradTape(N, T, checkpoint_every=every)
    assert tape._lib.gpu_bpf_grad_debug_resident(tape._h, fault, mailbox, 20.0) == _lib.BPF_OK
    assert math.isnan(tape.forward(theta, y, seed=8).item())      # a tape that no run has filled before
    assert np.isnan(tape.backward().cpu().numpy()).all()
    for read in (tape.records, lambda: tape.children(0), lambda: tape.replay(theta)):
        with pytest.raises(bpf.BpfError) as e:
            read()
        assert e.value.code == _lib.BPF_ERR_STATE
    assert tape._lib.gpu_bpf_grad_debug_resident(tape._h, 0, 0, 2000.0) == _lib.BPF_OK
    assert clean(tape) == want
    tape.close()


@pytest.mark.parametrize("N,ticks", [(70000, 70), (1000003, 12)])
def test_refused_run_goes_tick_by_tick(bpf, N, ticks):
    """A cooperative launch that the device refuses: the same results from the kernels of a tick, from host
    and device observations, with no error and no other attempt."""
    import torch
    y = _series(ticks, 5)
    yd = torch.tensor(y, device="cuda")

    def run(fault, fused):
        rec = torch.zeros(ticks * 40, dtype=torch.uint8, device="cuda")
        f = bpf.GpuBpf(N, RHO, SIG, MU, seed=3, ess_threshold=0.5)
        f.set_fused_small(fused)
        _arm(f, "gpu_bpf_debug_resident", fault)
        n0 = f._lib.gpu_bpf_launch_count()
        out = [bytes(r) for r in f.step_many(y.tolist(), records=True)] + [bytes(f.get_particles())]
        n1 = f._lib.gpu_bpf_launch_count()
        for _ in range(2):
            f.reset(7)
            f.step_many_device(yd.data_ptr(), ticks, rec.data_ptr())
            out += [bytes(f.get_record()), bytes(f.get_particles()), rec.cpu().numpy().tobytes()]
        n2 = f._lib.gpu_bpf_launch_count()
        f.close()
        return out, n1 - n0, n2 - n1

    resident, refused, plain = run(0, True), run(REFUSED, True), run(0, False)
    assert resident[0] == refused[0] == plain[0]
    assert resident[1] == 1 and refused[1:] == plain[1:] and refused[1] >= 2 * ticks


def test_refused_device_run_first(bpf):
    """The refusal met while the device run is captured."""
    import torch
    y = torch.tensor(_series(T, 5), device="cuda")
    out = []
    for fault in (0, REFUSED):
        rec = torch.zeros(T * 40, dtype=torch.uint8, device="cuda")
        f = bpf.GpuBpf(300000, RHO, SIG, MU, seed=3, ess_threshold=0.0)
        _arm(f, "gpu_bpf_debug_resident", fault)
        f.step_many_device(y.data_ptr(), T, rec.data_ptr())
        out.append((bytes(f.get_record()), bytes(f.get_particles()), rec.cpu().numpy().tobytes()))
        f.close()
    assert out[0] == out[1]


@pytest.mark.parametrize("N", [5000, 300000])
def test_refused_auxiliary_run_goes_kernel_by_kernel(bpf, N):
    """70 + 66 ticks: single ticks, then the 64-tick graph and a remainder."""
    y = _series(136, 5).tolist()
    out = []
    for fault in (0, REFUSED):
        f = bpf.GpuApf(N, RHO, SIG, MU, seed=3)
        _arm(f, "gpu_apf_debug_resident", fault)
        recs = f.step_many(y[:70], records=True)
        recs += f.step_many(y[70:], records=True)
        out.append(([bytes(r) for r in recs], bytes(f.get_particles()), f.get_loglik_total()))
        f.close()
    assert out[0] == out[1]


@pytest.mark.parametrize("every", [0, 4])
@pytest.mark.parametrize("N,nu_state,nu_obs", [(3, 0.0, 0.0), (70001, 0.0, 5.0), (700001, 5.0, 0.0)])
def test_refused_tape_is_taped_by_the_kernels(bpf, N, nu_state, nu_obs, every):
    """The three kernels a tick write the tape that the resident run writes: log-likelihood, records, child
    lists and gradient, bit for bit, whichever of the two a tape has used before."""
    import torch
    y = torch.tensor(_series(37, 6), device="cuda")

    def read(tape, seed):
        ll = tape.forward((MU, RHO, SIG), y, seed=seed, nu_obs=nu_obs, nu_state=nu_state).item()
        return (ll, tape.backward().cpu().numpy().tobytes(), [bytes(r) for r in tape.records()],
                [tape.children(t).tobytes() for t in (0, 17, 35)])

    out = []
    for faults in ((0, 0), (REFUSED, REFUSED), (0, REFUSED), (REFUSED, 0)):
        tape = bpf.GradTape(N, 37, checkpoint_every=every)
        got = []
        for fault, seed in zip(faults, (3, 9)):
            assert tape._lib.gpu_bpf_grad_debug_resident(tape._h, fault, 0, 2000.0) == 0
            got.append(read(tape, seed))
        tape.close()
        out.append(got)
    assert out[0] == out[1] == out[2] == out[3]


@pytest.mark.parametrize("N", [5000, 300000])
def test_recording_auxiliary_run_replays_its_graph(bpf, N):
    """A filter that records its ancestors keeps the kernels: a single tick, the 64-tick graph, the graph again
    and a remainder. Records and particles equal the resident run's, the last tick's ancestors those
    of the same run ended by a single tick."""
    y = _series(131, 5).tolist()
    f = bpf.GpuApf(N, RHO, SIG, MU, seed=3)
    want = [bytes(r) for r in f.step_many(y, records=True)], bytes(f.get_particles()), f.get_loglik_total()
    f.close()
    anc = []
    for last in (66, 1):
        f = bpf.GpuApf(N, RHO, SIG, MU, seed=3)
        f.record_ancestors(True)
        recs = f.step_many(y[:1], records=True) + f.step_many(y[1:65], records=True)
        recs += f.step_many(y[65:131 - last], records=True) if last == 1 else []
        recs += f.step_many(y[131 - last:], records=True)
        assert ([bytes(r) for r in recs], bytes(f.get_particles()), f.get_loglik_total()) == want
        anc.append([bytes(a) for a in f.get_ancestors()])
        f.close()
    assert anc[0] == anc[1]
