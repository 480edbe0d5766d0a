"""GPU: the sample offsets against torch.topk on the same random numbers, at the block sizes of the presets and between them, and with
equal numbers (where the framework leaves the order open: ascending position here)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("block,keep", [(128, 32), (64, 16), (32, 8), (48, 12), (128, 128), (1, 1), (127, 1)])
@pytest.mark.parametrize("B,H", [(1, 1), (2, 13), (1, 40)])
def test_offsets_equal_topk(block, keep, B, H):
    from psa_b200 import ops
    torch.manual_seed(block * H)
    got = ops.draw_sample_indices(B, H, block, keep, torch.device(DEV))
    torch.manual_seed(block * H)
    r = torch.rand(B, H, 1, block, device=DEV)
    assert all(len(set(row.tolist())) == block for row in r.view(-1, block))      # no equal numbers at these seeds
    want = torch.topk(r, keep, dim=3).indices.view(B, H, keep)
    assert got.dtype == torch.int64 and torch.equal(got, want)


def test_equal_numbers_by_ascending_position():
    from psa_b200 import _lib
    r = torch.tensor([[0.5, 0.25, 0.5, 0.0, 0.5, 0.25, 0.0, 0.75]], device=DEV)
    idx = torch.full((1, 6), -1, dtype=torch.int64, device=DEV)
    assert _lib.lib.psa_draw_samples(r.data_ptr(), idx.data_ptr(), 1, 8, 6, None) == 0
    torch.cuda.synchronize()
    assert idx.tolist() == [[7, 0, 2, 4, 1, 5]]
    assert _lib.lib.psa_draw_samples(r.data_ptr(), idx.data_ptr(), 1, 129, 6, None) == _lib.PSA_ERR_UNSUPPORTED
