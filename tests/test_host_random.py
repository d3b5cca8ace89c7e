"""rte_host_randint: the integers torch's seeded CPU generator draws (the shortlist head's random negatives)."""
import pytest
import torch

from speedup_thingy_b200 import _abi as A


@pytest.mark.parametrize("seed,n,vocab", [(0, 1, 2048), (1337, 624, 96), (7, 1249, 5000), (2 ** 33 + 5, 3000, 2 ** 28 - 1), (3, 10_000, 1)])
def test_draws_are_torchs(seed, n, vocab):
    out = torch.full((n + 1,), -7, dtype=torch.int32)
    A.check(A.load().rte_host_randint(seed, n, vocab, out.data_ptr()), "rte_host_randint")
    want = torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(seed))
    assert torch.equal(out[:n].long(), want) and int(out[n]) == -7


def test_ranges_torch_draws_differently_are_refused():
    out = torch.zeros(4, dtype=torch.int32)
    assert A.load().rte_host_randint(0, 4, 2 ** 28, out.data_ptr()) < 0
