"""Device memory of a filter: the exchange buffer of resident runs (over 600 KB at 592 tiles) is part of
filters that such runs take, and of no other."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

TILE = 4096


def test_exchange_buffer_only_where_resident_runs_are(bpf):
    import torch
    lib = bpf.load()
    limit = 4 * torch.cuda.get_device_properties(0).multi_processor_count     # tiles of a resident run

    def size(tiles):
        before = lib.gpu_bpf_debug_live_bytes()
        f = bpf.GpuBpf(tiles * TILE, 0.97, 0.15, -1.0)
        n = lib.gpu_bpf_debug_live_bytes() - before
        f.close()
        assert lib.gpu_bpf_debug_live_bytes() == before
        return n

    last, above, far = size(limit), size(limit + 1), size(limit + 2)
    per_tile = far - above
    assert 3 * TILE * 4 <= per_tile < 4 * TILE * 4               # particles (two buffers) and weights
    assert last > above - per_tile + 16 * 64 * limit             # 16 mailboxes of 64 bytes a tile, and more
