"""Stable ranks of token copies within their experts: lists that end inside a thread, a warp and a round."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [1, 5, 4095, 4096, 4097, 13000])
@pytest.mark.parametrize("E", [1, 7, 512])
def test_expert_ranks(n, E):
    from mindformers_b200.ops import _lib
    torch.manual_seed(n)
    ids = torch.randint(0, E + 1, (n,), device=DEV)              # E itself: a copy without an expert
    rank, counts = torch.full((n,), -1, dtype=torch.int32, device=DEV), torch.zeros(E, dtype=torch.int32, device=DEV)
    _lib.check(_lib.get_lib().mfb_moe_rank(ids.data_ptr(), n, E, rank.data_ptr(), counts.data_ptr(), _lib.stream_ptr()), "rank")
    hot = torch.nn.functional.one_hot(ids, E + 1)[:, :E]
    assert torch.equal(counts.long(), hot.sum(0))
    want = ((hot.cumsum(0) - 1) * hot).sum(1)
    assert torch.equal(rank.long(), torch.where(ids < E, want, -1))
