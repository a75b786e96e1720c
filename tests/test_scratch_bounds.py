"""Scratch (host code only): the library's bound for a batch covers what its kernels take for any projection and any number of
buckets; the package's buffers are one per stream."""

import pytest
import torch

from nanovllm_voxcpm_b200 import _native as N
from nanovllm_voxcpm_b200 import lora as LORA

ROWS = [1, 31, 32, 33, 100, 512, 600, 608, 640, 700, 768, 1000, 1600, 2367, 2368, 2400, 4000, 8192, 20000, 28000]
BUCKETS = [1, 2, 20, 37, 60, 64, 75, 100, 148, 149, 177, 300, 900, 2000]


@pytest.mark.parametrize("r", [16, 32, 64])
@pytest.mark.parametrize("n_slices", [1, 2, 3, 4])
def test_query_covers_the_grouped_kernels(n_slices, r):
    lib = N.lib()
    for T in ROWS:
        given = lib.lora_b200_workspace_bytes(T, n_slices, r)
        assert given <= 8 * n_slices * T * r * 4 + 128 * r * 2 + 1024
        for S in BUCKETS:
            for in_dim in (64, 200, 1024, 4096, 6144, 14336, 100000):
                need = lib.lora_b200_grouped_workspace_bytes(T, in_dim, n_slices, r, S)
                assert n_slices * T * r * 4 + 256 <= need <= given, (T, S, in_dim)


def test_no_scratch_for_ranks_that_the_grouped_kernels_do_not_run():
    assert N.lib().lora_b200_grouped_workspace_bytes(64, 1024, 1, 48, 8) == 0


def test_every_stream_has_a_buffer_of_its_own(monkeypatch):
    current = [1]
    monkeypatch.setattr(N, "current_stream", lambda device: current[0])
    monkeypatch.setattr(LORA, "_SCRATCH", {})
    monkeypatch.setattr(LORA, "_SCRATCH_FLOOR", {})
    monkeypatch.setattr(LORA, "_RETIRED_SCRATCH", [])
    cpu = torch.device("cpu")
    first = LORA.scratch_for(cpu, 100)
    assert LORA.scratch_for(cpu, 1000) is first
    current[0] = 2
    second = LORA.scratch_for(cpu, 100)
    assert second.data_ptr() != first.data_ptr()
    grown = LORA.reserve_scratch(cpu, 3 << 20)
    assert grown.numel() == 3 << 20 and LORA._RETIRED_SCRATCH == [second]
    current[0] = 3
    assert LORA.scratch_for(cpu, 1).numel() == 3 << 20  # what was reserved holds for every stream
    current[0] = 1
    assert LORA.scratch_for(cpu, 100) is first
