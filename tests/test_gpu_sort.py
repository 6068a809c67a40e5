"""The stable radix sort at the ends of its tiles (2,048 keys; 4,096 from 2^19
keys on), of its warps' runs and of its digits, with and without values, against
numpy's stable order of the low bits, rounded up to whole 8-bit digits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 8, 9, 17, 32])
@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 2047, 2048, 2049, 36863, 524287, 524288, 524289, 1000003])
def test_sort_at_tile_edges(n, bits):
    import sphg as S
    import torch
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    if n % 2:  # few distinct keys: long runs of equal digits, stability decides
        keys &= np.uint32(0x80030101)
    vals = rng.integers(0, 1 << 31, n, dtype=np.int32)
    order = np.argsort(keys & np.uint32((1 << (bits + 7) // 8 * 8) - 1), kind="stable")
    k = torch.from_numpy(keys.view(np.int32)).cuda()
    v = torch.from_numpy(vals).cuda()
    ko, vo = torch.empty_like(k), torch.empty_like(v)
    stream = torch.cuda.current_stream()
    for given in (None, v):
        S.sort_pairs(k.data_ptr(), given.data_ptr() if given is not None else None, ko.data_ptr(), vo.data_ptr(), n,
                     bits, stream=stream)
        assert np.array_equal(ko.cpu().numpy().view(np.uint32), keys[order])
        assert np.array_equal(vo.cpu().numpy(), order.astype(np.int32) if given is None else vals[order])
