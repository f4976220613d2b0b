"""GF4 packer on the GPU against the host packer, bit for bit, where its kernels change shape: CTA sizes (K up to 1024,
2048, longer), arrays that leave shared memory (K from about 5000), rows of few distinct values, more rows than a chunk."""
import pytest
import torch

import if_i_could_turn_back_time_b200 as jq
from test_gpu_parity import DEV, _weights

pytestmark = pytest.mark.gpu


def _same(W, spec):
    host, dev = jq.pack_weight(W, spec), jq.pack_weight(W.to(DEV), spec)
    assert torch.equal(dev.codebook.cpu().view(torch.int16), host.codebook.view(torch.int16))
    assert torch.equal(dev.qweight.cpu(), host.qweight)
    if spec.group_size:
        assert torch.equal(dev.scales.cpu().view(torch.int16), host.scales.view(torch.int16))


@pytest.mark.parametrize("N,K,g,had", [(3, 1, 0, 0), (3, 16, 0, 0), (4, 17, 0, 0), (5, 1024, 64, 0), (5, 1025, 0, 0), (4, 2048, 128, 128),
                                       (4, 2304, 256, 0), (3, 4864, 128, 0), (3, 6001, 0, 0), (2, 20000, 0, 0), (2, 32768, 128, 0),
                                       (1300, 96, 32, 0)])
def test_packer_shapes(N, K, g, had):
    _same(_weights(N, K, N + K), jq.QuantSpec("gf4", g, had))


@pytest.mark.parametrize("K", [300, 1500, 5000, 9001, 27000])
def test_packer_ties_and_near_ties(K):
    """Values on a grid (many equal costs), values that differ in the last bit, wide magnitudes, all equal.  Long rows of few
    values keep their arrays in shared memory, with the reciprocals beside them (9001) or not (27000)."""
    g = torch.Generator("cpu").manual_seed(K)
    grid = torch.round(torch.randn(3, K, generator=g) * 8) / 8
    near = 1.0 + torch.randint(0, 40, (3, K), generator=g).float() * 2.0 ** -23
    wide = torch.randn(3, K, generator=g) * torch.logspace(-12, 4, K)[None]
    few = torch.randint(0, 12, (2, K), generator=g).float()
    _same(torch.cat([grid, near, wide, few, torch.full((1, K), 0.25)]), jq.QuantSpec("gf4", 0, 0))


def test_packer_rows_of_few_and_of_many_values_in_turn():
    """More rows than CTAs: a CTA's row of few distinct values follows one of many and the other way round."""
    g = torch.Generator("cpu").manual_seed(3)
    W = torch.randn(312, 4600, generator=g)
    few = torch.rand(312, generator=g) < 0.5
    W[few] = torch.round(W[few] * 8) / 8
    _same(W, jq.QuantSpec("gf4", 0, 0))
