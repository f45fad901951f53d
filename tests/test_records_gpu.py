"""Plan, controller and mean kernels of the superchunk records at the edges of their splits."""
import pytest
import torch

from dynamiq_sigcomm_artifact_b200 import bitalloc

pytestmark = pytest.mark.gpu


def _dq():
    from dynamiq_sigcomm_artifact_b200 import ops

    return ops.require()


@pytest.mark.parametrize("nsc", [1, 4 * 1023, 4 * 1025 + 2, 4 * (1 << 16), 4 * (1 << 16) + 1])
def test_plan_by_one_cta_and_by_scan(nsc):
    g = torch.Generator().manual_seed(nsc)
    w = torch.tensor([2, 4, 8], dtype=torch.uint8)[torch.randint(0, 3, (nsc,), generator=g)]
    plan, nb = _dq().superchunk_plan(w.cuda()).cpu(), (nsc + 3) // 4
    wp = torch.cat([w, torch.full((4 * nb - nsc,), 2, dtype=torch.uint8)]).view(nb, 4).long()
    assert torch.equal(plan[1: nb + 1].long(), torch.cumsum((16 * (2 * wp + 1) + 2).sum(1) // 8, 0)) and int(plan[0]) == 0
    assert torch.equal(plan[nb + 1:].long(), (wp << torch.tensor([0, 8, 16, 24])).sum(1))


@pytest.mark.parametrize("n", [1, 8191, 8193, 300_000])
def test_controller_counts_unsorted_scores(n):
    """Three steps of the device controller against the host controller on the same energies."""
    g = torch.Generator().manual_seed(n)
    host, dev = bitalloc.DynamicBitrateController(5), bitalloc.DeviceBitrateController(5, "cuda")
    for step in range(3):
        energy = torch.exp(4.0 * torch.randn(n, generator=g)) * 10.0 ** step
        stats = torch.stack([torch.zeros(n), energy], 1).cuda()
        dev.widths(stats)
        dev.end_of_step()
        host.observe(energy)
        host.end_of_step()
        u, initialised, avg, _ = dev.state.tolist()
        assert initialised == 1.0 and abs(u - host.u) < 1e-5 and abs(avg - host.last_avg) < 2e-3 + 1.0 / n


@pytest.mark.parametrize("n,offset", [(1, 0), (255, 0), (1024 * 37 + 3, 0), (5000, 1), (4096, 4)])
def test_add_mean(n, offset):
    nsc = (n + 255) // 256
    resid, mean = torch.randn(nsc * 256, device="cuda"), torch.randn(nsc, device="cuda")
    for dtype in (torch.float32, torch.bfloat16):
        out = torch.zeros(n + offset, device="cuda", dtype=dtype)
        _dq().superchunk_add_mean(resid, mean, out[offset:])
        want = (resid.view(nsc, 256) + mean[:, None]).reshape(-1)[:n].to(dtype)
        assert torch.equal(out[offset:], want) and float(out[:offset].float().abs().sum()) == 0
