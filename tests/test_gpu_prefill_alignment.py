"""f32 prompts whose buffers start off a 16-byte boundary (scalar conversion) give what aligned ones (four values at a
time) give, bit for bit: maxima and roundings do not depend on how the values are read."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seq,nh,nkv,hd,off", [(1, 1, 1, 64, 1), (37, 9, 3, 64, 3), (130, 4, 2, 128, 2)])
def test_f32_prefill_does_not_depend_on_the_alignment(seq, nh, nkv, hd, off):
    import torch
    import flarellm_b200 as fb
    g = torch.Generator(device="cuda").manual_seed(seq)
    eng = fb.Engine(0)
    outs = []
    data = [torch.randn(seq * h * hd, device="cuda", generator=g) * s for h, s in ((nh, 0.5), (nkv, 300.0), (nkv, 1.0))]
    data[0][-1] = -9.0                                   # the maximum in the last element
    for o in (0, off):
        bufs = [torch.zeros(t.numel() + o, device="cuda") for t in data]
        for b, t in zip(bufs, data):
            b[o:] = t
        out = torch.zeros(seq * nh * hd, device="cuda")
        torch.cuda.synchronize()
        eng.prefill(*(b[o:].data_ptr() for b in bufs), 1, seq, nh, nkv, hd, in_dtype=fb.DT_F32, out_dtype=fb.DT_F32, out=out.data_ptr())
        eng.sync()
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.isfinite(outs[0]).all()
    eng.close()
