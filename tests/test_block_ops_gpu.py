"""Fused sub-layer kernels at the edges of their tiles, against plain PyTorch in fp32."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _dq():
    from dynamiq_sigcomm_artifact_b200 import ops

    return ops.require()


def _close(a, b, tol):
    assert float((a.float() - b).norm()) <= tol * float(b.norm()) + 1e-6


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,H", [(1, 8), (7, 248), (300, 256), (33, 264), (1500, 768), (5, 2040), (700, 2048)])
@pytest.mark.parametrize("rms,extra", [(False, "ds"), (True, "dy2"), (True, None)])
def test_add_norm(rows, H, dtype, rms, extra):
    dq, tol = _dq(), 8e-3 if dtype == torch.bfloat16 else 1e-5
    torch.manual_seed(rows + H)
    x, d, dy, e = (torch.randn(rows, H, device="cuda").to(dtype) for _ in range(4))
    bias, w = torch.randn(H, device="cuda"), torch.randn(H, device="cuda")
    b = None if rms else torch.randn(H, device="cuda")
    s, y, mean, rstd = dq.add_norm_fwd(x, d, bias, w, b, 1e-5, rms)
    _close(s, x.float() + d.float() + bias, tol)
    sf = s.float().requires_grad_()
    wf, bf = w.clone().requires_grad_(), None if rms else b.clone().requires_grad_()
    ref = sf * torch.rsqrt(sf.pow(2).mean(-1, keepdim=True) + 1e-5) * wf if rms else F.layer_norm(sf, (H,), wf, bf, 1e-5)
    _close(y, ref.detach(), tol)
    dx, dw, db, dbias = dq.add_norm_bwd(dy, e if extra == "dy2" else None, e if extra == "ds" else None, s, w, mean, rstd, rms,
                                        True)
    ref.backward(dy.float() + e.float() if extra == "dy2" else dy.float())
    want = sf.grad + e.float() if extra == "ds" else sf.grad
    _close(dx, want, tol)
    _close(dw, wf.grad, tol)
    _close(dbias, want.sum(0), 3 * tol)
    if not rms:
        _close(db, bf.grad, tol)
    _close(dq.residual_add(x, d, bias), x.float() + d.float() + bias, tol)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tanh", [True, False])
@pytest.mark.parametrize("rows,cols", [(1, 8), (17, 264), (1000, 512), (5, 3072)])
def test_gelu_with_bias(rows, cols, tanh, dtype):
    dq, tol = _dq(), 6e-3 if dtype == torch.bfloat16 else 1e-5
    torch.manual_seed(cols)
    pre, d = (4 * torch.randn(rows, cols, device="cuda")).to(dtype), torch.randn(rows, cols, device="cuda").to(dtype)
    bias = torch.randn(cols, device="cuda")
    pf = (pre.float() + bias).requires_grad_()
    ref = F.gelu(pf, approximate="tanh" if tanh else "none")
    _close(dq.gelu_fwd(pre, bias, tanh), ref.detach(), tol)
    ref.backward(d.float())
    dpre, db = dq.gelu_bwd(d, pre, bias, tanh, None)
    _close(dpre, pf.grad, tol)
    _close(db, pf.grad.sum(0), 2 * tol)


@pytest.mark.parametrize("B,S,nh,nkv,D", [(1, 1, 1, 1, 16), (2, 33, 3, 1, 64), (3, 100, 4, 4, 32), (1, 700, 12, 12, 64)])
def test_attention_surroundings(B, S, nh, nkv, D):
    from dynamiq_sigcomm_artifact_b200.ops.layers import rope_tables

    dq = _dq()
    torch.manual_seed(S)
    cos, sin = rope_tables(S, D, 1e4, "cuda")
    qkv = torch.randn(B, S, (nh + 2 * nkv) * D, device="cuda", dtype=torch.bfloat16)

    def rotate(t, sign):  # [B, S, heads, D]
        a, b, c, s = t[..., : D // 2], t[..., D // 2:], cos.view(1, S, 1, -1), sign * sin.view(1, S, 1, -1)
        return torch.cat([a * c - b * s, b * c + a * s], -1)

    heads = qkv.float().view(B, S, nh + 2 * nkv, D)
    want = torch.cat([rotate(heads[:, :, : nh + nkv], 1), heads[:, :, nh + nkv:]], 2)
    got = qkv.clone()
    dq.rope_qkv_(got, cos, sin, nh, nkv, D)
    _close(got.view_as(want), want, 5e-3)
    gq, gk, gv = (torch.randn(B, n, S, D, device="cuda", dtype=torch.bfloat16) for n in (nh, nkv, nkv))
    gk = gk.transpose(1, 2).contiguous().transpose(1, 2)  # another layout than its neighbours
    flat = torch.cat([t.float().transpose(1, 2) for t in (gq, gk, gv)], 2)
    want = torch.cat([rotate(flat[:, :, : nh + nkv], -1), flat[:, :, nh + nkv:]], 2)
    _close(dq.qkv_grad_pack(gq, gk, gv, cos, sin, False, None)[0].view_as(want), want, 5e-3)
    packed, db = dq.qkv_grad_pack(gq, gk, gv, None, None, True, None)
    assert torch.equal(packed.float().view_as(flat), flat)
    sums = flat.sum((0, 1))
    sums[nh: nh + nkv] = 0  # the softmax does not see the key bias
    _close(db, sums.reshape(-1), 1e-4)


@pytest.mark.parametrize("B,S,H,P", [(1, 1, 8, 1), (3, 50, 136, 64), (9, 128, 768, 128)])
def test_embedding(B, S, H, P):
    dq, V = _dq(), 97
    torch.manual_seed(H)
    ids = torch.randint(0, V, (B, S), device="cuda")
    tok, pos, typ = torch.randn(V, H, device="cuda").bfloat16(), torch.randn(P, H, device="cuda"), torch.randn(2, H, device="cuda")
    _close(dq.embed_fwd(ids, tok, pos, typ), tok.float()[ids] + pos[:S] + typ[0], 5e-3)
    assert torch.equal(dq.embed_fwd(ids, tok, None, None), tok[ids])
    dx = torch.randn(B, S, H, device="cuda").bfloat16()
    base = torch.randn(V, H, device="cuda")
    for with_pos in (True, False):
        got, gpos = base.clone(), torch.full((P, H), 7.0, device="cuda")
        dq.embed_bwd(dx, ids, got, gpos if with_pos else None)
        _close(got, base.index_add(0, ids.reshape(-1), dx.float().view(-1, H)), 1e-5)
    dq.embed_bwd(dx, ids, None, gpos)
    _close(gpos[:S], dx.float().sum(0), 1e-5)
    assert float(gpos[S:].abs().sum()) == 0


@pytest.mark.parametrize("N,vocab,width,colsum", [(1, 1, 8, True), (37, 1000, 1024, False), (300, 4099, 4104, True),
                                                  (5, 50257, 50304, False), (9, 60000, 60032, True), (4, 128256, 128256, False)])
def test_fused_cross_entropy_and_gradient(N, vocab, width, colsum):
    dq = _dq()
    torch.manual_seed(N)
    logits = (3 * torch.randn(N, width, device="cuda")).bfloat16()
    labels = torch.randint(0, vocab, (N,), device="cuda")
    if N > 3:
        labels[1::3] = -100
        logits[0, 0] = 60.0
    ref = logits.float()[:, :vocab].requires_grad_()
    want = F.cross_entropy(ref, labels, ignore_index=-100)
    want.backward()
    work = logits.clone()
    loss, sums = dq.ce_fused(work, labels, vocab, -100, False, colsum)
    assert abs(loss.item() - want.item()) < 1e-4 * max(1.0, abs(want.item()))
    _close(work[:, :vocab], ref.grad, 5e-3)
    assert float(work[:, vocab:].float().abs().sum()) == 0
    if colsum:
        _close(sums[:vocab], ref.grad.sum(0), 5e-3)
    dq.ce_rescale_(work, torch.full((1,), 0.5, device="cuda"))
    _close(work[:, :vocab], 0.5 * ref.grad, 5e-3)


def test_shifted_labels():
    dq = _dq()
    logits, labels = torch.randn(3 * 7, 64, device="cuda").bfloat16(), torch.randint(0, 64, (3, 7), device="cuda")
    want = F.cross_entropy(logits.float().view(3, 7, 64)[:, :-1].reshape(-1, 64), labels[:, 1:].reshape(-1))
    loss, _ = dq.ce_fused(logits, labels, 64, -100, True, False)
    assert abs(loss.item() - want.item()) < 1e-4
