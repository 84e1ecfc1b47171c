"""The autotuner's cache file: entries of builds with other kernels are not taken."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_cache_of_an_earlier_build_is_measured_again(bpf, tmp_path):
    import torch
    from gpubpf import dgp
    y = np.asarray(dgp.matched_series(20, 0.97, 0.2, -1.0, 4)[1], dtype=np.float32).tolist()
    p = torch.cuda.get_device_properties(0)
    old = f"{p.name.replace(' ', '_')}_sm{p.multi_processor_count}"
    cache = tmp_path / "tune.txt"
    cache.write_text(f"{old} 2 64\n")        # 64 threads for 4096 particles: the generic kernel, far from the fastest
    filters = [{"mu": -1.0, "rho": 0.97, "sigma_z": 0.2, "n_particles": 4096, "seed": s} for s in range(200)]
    b = bpf.GpuBpfBatch(filters, ess_threshold=0.0)
    b.autotune(y, cache_path=str(cache))
    lines = cache.read_text().splitlines()
    assert len(lines) == 2 and lines[0] == f"{old} 2 64"
    key, cls, threads = lines[1].split()
    assert key.startswith(old + "_k") and cls == "2"
    assert b._lib.gpu_bpf_batch_get_threads(b._h, 2) == int(threads)
    again = bpf.GpuBpfBatch(filters, ess_threshold=0.0)
    again.autotune(y, cache_path=str(cache))             # this build's entry is taken
    assert cache.read_text().splitlines() == lines
    assert again._lib.gpu_bpf_batch_get_threads(again._h, 2) == int(threads)
    b.close()
    again.close()
