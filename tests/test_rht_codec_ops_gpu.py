"""The standalone rotation-codec operators at the edges of their block and warp split, against the CPU oracle."""
import numpy as np
import pytest
import torch

from dynamiq_sigcomm_artifact_b200 import codec_ref as cr
from dynamiq_sigcomm_artifact_b200.parallel import cpu_backend as cb
from dynamiq_sigcomm_artifact_b200.parallel import schedules as sch

from helpers import heavy_tail_grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bits,offset,dtype", [(1, 5, 0, torch.float32), (1023, 3, 0, torch.float32),
                                                 (1025, 8, 1, torch.float32), (24 * 1024, 5, 0, torch.bfloat16),
                                                 (19 * 1024 + 7, 4, 3, torch.bfloat16), (40 * 1024, 6, 1, torch.float32)])
def test_operators_match_the_oracle(n, bits, offset, dtype):
    """One CTA of eight warps: more blocks than warps, ragged tails, inputs that no bulk copy may fetch."""
    from dynamiq_sigcomm_artifact_b200.parallel.fused import RhtCodec

    seed, step, bucket = 31, 4, 6
    x = torch.from_numpy(np.concatenate([np.zeros(offset, np.float32), heavy_tail_grad(n, 3)])).to(dtype)
    xd = x.cuda()[offset:]
    x = x[offset:].float().numpy()
    codec = RhtCodec(bits, n, seed=seed, ctas=1, threads=256)
    words, scales = codec.compress(xd, step=step, bucket_id=bucket)
    ref = cb.RhtCodecCPU(bits, seed, step, bucket, world=1)
    y = ref.rotate(cr.to_blocks(x))
    codes, rscale = cr.quantize(y, bits, np.arange(y.shape[0]), ref._tag_base | sch.TAG_ENCODE, step, seed)
    assert np.array_equal(words.cpu().numpy().view(np.uint32), cr.pack(codes, bits))
    assert np.array_equal(scales.cpu().numpy(), rscale)
    w2, s2 = codec.dec_comp((words, scales), xd, step=step, bucket_id=bucket)
    v = cr.dequantize_add(codes, rscale, bits, y)
    c2, rs2 = cr.quantize(v, bits, np.arange(v.shape[0]), ref._tag_base | (sch.TAG_ENCODE + 1), step, seed)
    assert np.array_equal(w2.cpu().numpy().view(np.uint32), cr.pack(c2, bits)) and np.array_equal(s2.cpu().numpy(), rs2)
    out = codec.decompress((w2, s2), n, step=step, bucket_id=bucket, post_scale=0.5, dtype=dtype)
    want = torch.from_numpy(cr.rotate_inv(cr.dequantize(c2, rs2, bits), ref.signs, 0.5).reshape(-1)[:n].copy()).to(dtype)
    assert torch.equal(out.cpu(), want)
