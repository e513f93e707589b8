"""The rules that send prompt portions to the tcgen05 attention kernels, on work lists made on the CPU."""

from __future__ import annotations

import types

import numpy as np
import pytest
import torch

from mini_llm_runtime_b200.ops import AttentionBatch
from mini_llm_runtime_b200.ops import cuda_ops


def batch(lengths, before):
    lengths, before = np.array(lengths, np.int32), np.array(before, np.int32)
    arrays, counts = cuda_ops.plan_attention(lengths, before)
    return AttentionBatch(None, None, None, None, None, len(lengths), int(lengths.max()), int((lengths + before).max()), arrays, counts)


@pytest.mark.parametrize("lengths,before,window,keys", [
    ([2, 1], [40, 2000], 0, 42), ([1, 2, 7], [2000, 40, 100], 0, 107), ([9], [300], 0, 309), ([1, 1], [5, 2000], 0, 0),
    ([2, 1], [900, 2000], 100, 102), ([300], [900], 100, 228), ([300], [0], 1000, 300)])
def test_the_keys_that_prompt_rows_see(lengths, before, window, keys):
    assert cuda_ops.prompt_keys(batch(lengths, before), window) == keys


@pytest.mark.parametrize("decoded", [[], [3], [2000, 5]])
def test_decoded_rows_contexts_do_not_move_the_borders(decoded):
    """Few rows that see few keys stay on the older kernels however long the contexts beside them are; many rows or keys do not."""
    ones, few = [1] * len(decoded), 192 if decoded else 96
    for lengths, before, latent, diff in (([2], [40], False, False), ([4], [40], False, False), ([4], [few], True, True),
                                          ([4], [few - 4], few > 96, False), ([4], [92], False, False), ([4], [93], True, not decoded),
                                          ([2], [few], True, False), ([7], [0], False, False), ([8], [0], False, True), ([65], [0], True, True)):
        b, rows = batch(lengths + ones, before + decoded), sum(lengths) + len(ones)
        assert cuda_ops.latent_prompt_on_tcgen05(b, rows, 0) == latent, (lengths, before)
        assert cuda_ops.diff_prompt_on_tcgen05(b, rows, 0, 0) == diff, (lengths, before)
        # a window shorter than the border hides the keys behind it
        assert cuda_ops.latent_prompt_on_tcgen05(b, rows, 50) == (rows - len(ones) > 64), (lengths, before)


@pytest.mark.parametrize("lengths,before,dim,few", [
    ([64], [0], 128, True), ([1], [63], 64, True), ([1], [64], 64, False), ([1] * 8, [64] * 8, 128, False), ([128], [0], 128, False), ([129], [0], 128, True),
    ([1] * 74, [255] * 74, 128, True), ([1] * 75, [255] * 75, 128, False), ([1] * 75, [127] * 75, 128, False), ([16, 1], [500, 2000], 128, True), ([512], [0], 128, True),
    ([513], [0], 128, False), ([129], [0], 64, False)])
def test_sigmoid_attention_of_few_keys_stays_on_mma_sync(lengths, before, dim, few):
    """Contexts of half a key tile; with heads of 128, several tiles of an entry while all entries' tiles are a round of the SMs."""
    b = batch(lengths, before)
    assert cuda_ops.CudaOps._sigmoid_few(b.max_kv_len, b.counts["tiles"], dim, 148) == few


def test_a_product_is_told_the_room_that_its_workspace_has(monkeypatch):
    """The kernel refuses plans that do not fit; what counts is the memory there is, not what a workspace made later would get."""
    asked = []
    library = types.SimpleNamespace(mlr_gemm_tcgen05=lambda *args: asked.append((args[12], args[14])) or cuda_ops._NO_ROOM)
    monkeypatch.setattr(cuda_ops, "_declared_library", lambda name: library)
    monkeypatch.setattr(cuda_ops, "_raw_stream", lambda: 0)
    operations = cuda_ops.CudaOps()
    space = {"gemm_scratch": torch.empty(512, dtype=torch.uint8), "gemm_counters": torch.zeros(7, dtype=torch.int32),
             "error_word": torch.zeros(1, dtype=torch.int32)}
    monkeypatch.setattr(operations, "_workspace", lambda device: space)
    operations.GEMM_SCRATCH_BYTES = operations.GEMM_COUNTERS = 1 << 20
    x, w = torch.zeros(64, 128, dtype=torch.bfloat16), torch.zeros(256, 128, dtype=torch.bfloat16)
    assert operations._linear_tcgen05(x, w, None, torch.bfloat16) is None
    assert asked == [(512, 7)]
