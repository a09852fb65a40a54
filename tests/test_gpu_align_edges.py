"""Sort-and-pad where its launch shape changes: one block or several (1024 assignments), longer chunks
(2^17), more than 48 KiB of shared memory (592 experts); and runs of one expert or none in a warp."""

import numpy as np
import pytest
import torch

from moe_bench_b200 import capi
from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("assignments,experts", [(1, 1), (512, 256), (513, 256), (1024, 7), (1025, 256), (4096, 256),
                                                 (4097, 256), (512, 257), (513, 257), (131072, 300), (131073, 300),
                                                 (524289, 32), (131072, 32), (131073, 32), (1000, 592), (1000, 593),
                                                 (65537, 1024), (1024, 256), (1025, 1), (2049, 2)])
@pytest.mark.parametrize("mapped", [False, True])
def test_align_at_the_edges(assignments, experts, mapped):
    rng = np.random.default_rng(assignments + experts)
    ids = rng.integers(0, experts, (assignments, 1)).astype(np.int32)
    ids[rng.random(assignments) < 0.3] = min(3, experts - 1)  # one popular expert
    emap, local = None, experts
    if mapped:  # every other expert lives elsewhere
        local = (experts + 1) // 2
        emap = np.where(np.arange(experts) % 2 == 0, np.arange(experts) // 2, -1).astype(np.int32)
    counts, prefix, sorted_ids, inverse = capi.align(
        torch.from_numpy(ids).to(DEV), None if emap is None else torch.from_numpy(emap).to(DEV), local, 16)
    o_counts, o_off, o_sorted, o_inv = O.align(ids, emap, local, 16)
    assert np.array_equal(counts.cpu().numpy(), o_counts)
    assert np.array_equal(prefix.cpu().numpy() * 16, o_off)
    assert np.array_equal(sorted_ids.cpu().numpy()[: int(o_off[-1])], o_sorted)
    assert np.array_equal(inverse.cpu().numpy(), o_inv)
