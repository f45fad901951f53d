"""One-kernel EDEN and the tiled whole-vector Hadamard transform at the edges of their splits."""
import pytest
import torch

from dynamiq_sigcomm_artifact_b200.parallel import eden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", range(1, 9))
@pytest.mark.parametrize("n,offset", [(1, 0), (1024, 0), (9 * 1024 + 517, 1)])
def test_eden_kernels_match_the_operator_chain(bits, n, offset):
    g = torch.Generator().manual_seed(100 * bits + n)
    x = torch.randn(n + offset, generator=g)
    if n > 1:
        x[offset + 3] = float("inf")  # counts as zero
    cpu, gpu = eden.Eden(bits, seed=7), eden.Eden(bits, seed=7)
    wc, sc, _ = cpu.compress(x[offset:], step=2)
    wg, sg, _ = gpu.compress(x.cuda()[offset:], step=2)
    assert wg.shape == wc.shape and sg.shape == sc.shape
    bc = eden.unpack_bins(wc, bits, sc.numel() * 1024).int()
    bg = eden.unpack_bins(wg.cpu(), bits, sc.numel() * 1024).int()
    assert int((bc - bg).abs().max()) <= 1 and float((bc != bg).float().mean()) < 2e-3
    assert torch.allclose(sg.cpu(), sc, rtol=2e-3)
    back, ref = gpu.decompress((wc.cuda(), sc.cuda(), n), step=2).cpu(), cpu.decompress((wc, sc, n), step=2)
    assert back.shape == ref.shape and torch.allclose(back, ref, atol=1e-5 * max(1.0, float(ref.abs().max())))


@pytest.mark.parametrize("log2d", [0, 1, 5, 11, 14, 22, 23, 24])
def test_whole_vector_transform_over_tiles(log2d):
    from dynamiq_sigcomm_artifact_b200.ops.fwht import fwht_pow2

    d = 1 << log2d
    x = torch.randn(d, generator=torch.Generator().manual_seed(log2d))
    got = fwht_pow2(x.cuda()).cpu()
    want = fwht_pow2(x)
    assert float((got - want).abs().max()) < 1e-5 * float(want.abs().max()) + 1e-6
