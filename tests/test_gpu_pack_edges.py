"""The device packer on payloads that begin at any byte of an allocation and end
within a word, with column lengths around its 64-individual chunks, few and many
slices: counts and ragged lists equal to the host's decoding, which is exact."""
import numpy as np
import pytest
import torch

from bayesrrcmd_gb300 import gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [5, 63, 64, 65, 129, 1027, 16_003])   # the last: lists past a warp's buffer
@pytest.mark.parametrize("offset,grid", [(0, 0), (1, 2), (2, 1), (3, 0)])
def test_packed_counts_and_lists(gpu_lib, N, offset, grid):
    M, nb = 37, (N + 3) // 4
    rng = np.random.default_rng(N + offset)
    code = rng.choice(4, size=(M, 4 * nb), p=[0.1, 0.05, 0.25, 0.6]).astype(np.uint8)   # the payload's padding bits too
    code[:, 0], code[:, 1] = 2, 3
    bed = (code.reshape(M, nb, 4) << np.array([0, 2, 4, 6], np.uint8)).sum(2).astype(np.uint8)
    room = torch.zeros(offset + bed.size, dtype=torch.uint8, device="cuda")
    room[offset:] = torch.from_numpy(bed.ravel()).cuda()
    torch.cuda.synchronize()
    code = code[:, :N]
    with gpu.Chain(gpu.ChainConfig(N=N, M=M, kind=gpu.KIND_RAGGED, S=[[0.01, 0.001]], grid=grid)) as ch:
        ch.pack_bed_device(room.data_ptr() + offset, bed.size)
        _, counts = ch.marker_table()
        lists = ch.ragged_lists(counts)
    for col, c in enumerate((3, 2, 0, 1)):   # g = 0, 1, 2, missing
        np.testing.assert_array_equal(counts[:, col], (code == c).sum(1))
    for (off, idx), c in zip(lists, (2, 0, 1)):
        for j in range(M):
            np.testing.assert_array_equal(idx[off[j]:off[j + 1]], np.flatnonzero(code[j] == c))
