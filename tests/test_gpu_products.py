"""The Q8_0 product at the edges of its tiles (16 rows, 8 input vectors, steps of up to 64 blocks spread over 8 warps)
and the forward pass on the launches that go through it: the attention kernel reading [q | k | v] rows and writing input
blocks, and the widths whose norm has a kernel of its own."""
import numpy as np
import pytest

from util import assert_bits_equal
from test_gpu_forward import _make_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,batch", [
    (1, 32, 1), (15, 64, 7), (16, 576, 8), (17, 576, 9),     # tile and vector-group remainders, few blocks for 8 warps
    (48, 2048, 8), (31, 2080, 8), (16, 2112, 3),             # the widest single step, one block more (33 + 32), 33 + 33
    (70, 8192, 17), (20, 6176, 1),                           # several steps; 193 blocks = 49 + 49 + 49 + 46
    (16 * 148 * 2 + 5, 96, 8), (40, 64, 256),                # more tiles than resident CTAs; every group of vectors
])
def test_product_is_bit_exact_at_tile_edges(orc, rows, cols, batch):
    import torch
    import flarellm_b200 as fb
    rng = np.random.default_rng(rows * 7 + cols + batch)
    blocks = orc.quantize_q8_0(rng.standard_normal((rows, cols), dtype=np.float32))
    x = rng.standard_normal((batch, cols), dtype=np.float32)
    x[-1, -32:] = 0.0                                        # d == 0
    x[0, 3] = 3.0e4                                          # a block dominated by one value
    want = np.stack([orc.matvec_q8_0(blocks, x[b], rows) for b in range(batch)])
    eng = fb.Engine(0)
    w = eng.weight_upload_q8_0(blocks, rows, cols)
    assert_bits_equal(eng.matvec_q8_0(w, x), want, "host buffers")
    # device input off a 16-byte boundary: quantised by the separate kernel
    xd = torch.empty(batch * cols + 1, device="cuda")
    xd[1:] = torch.from_numpy(x.reshape(-1)).cuda()
    od = torch.empty(batch, rows, device="cuda")
    torch.cuda.synchronize()
    eng.matvec_q8_0(w, xd[1:].data_ptr(), out=(od.data_ptr(), batch))
    eng.sync()
    assert_bits_equal(od.cpu().numpy(), want, "device input on a 4-byte boundary")
    w.free(); eng.close()


@pytest.mark.parametrize("batch,nh,nkv,hd,dim,inter,held", [
    (1, 8, 4, 64, 512, 1024, 0),          # everything fused, first token of an empty cache
    (3, 32, 8, 64, 576, 96, 700),         # 18 blocks a row; [q | k | v] rows taken from one buffer; several slot ranges
    (9, 16, 8, 128, 256, 64, 40),         # two groups of vectors, heads of 128
    (1, 8, 8, 64, 2112, 2112, 5000),      # 66 blocks a row: norm and quantiser as kernels; the attention merges by kernel
])
def test_forward_token_fused_step(orc, batch, nh, nkv, hd, dim, inter, held):
    """Q8_0 cache on the tensor-core attention kernel.  Logits within 2 % of their largest: the attention output, inside
    its own tolerance, is rounded to 8-bit codes by the next product."""
    import flarellm_b200 as fb
    rng = np.random.default_rng(dim + batch)
    cfg = dict(hidden_dim=dim, num_heads=nh, num_kv_heads=nkv, head_dim=hd, intermediate_dim=inter, vocab_size=500, rms_norm_eps=1e-5)
    n_layers, max_seq, theta = 2, (held + 8 + 31) // 32 * 32, 10000.0
    layers, output_norm, out_q8, _ = _make_model(orc, rng, cfg, n_layers, True)
    cos, sin = orc.rope_table(hd, max_seq, theta)
    eng = fb.Engine(0)
    kv = eng.kv_alloc(n_layers, batch, max_seq, nkv, hd, fb.KV_Q8_0)
    kv.set_rope_table(cos, sin)
    model = eng.model_create(num_layers=n_layers, **cfg)
    for li, lw in enumerate(layers):
        model.set_layer(li, **lw)
    model.set_output(output_norm, output_q8=out_q8)
    store = lambda r: orc.dequant_q8_0(orc.quantize_q8_0(r))
    caches = [([np.zeros((max_seq, nkv * hd), np.float32) for _ in range(n_layers)],
               [np.zeros((max_seq, nkv * hd), np.float32) for _ in range(n_layers)]) for _ in range(batch)]
    for b in range(batch):
        if held:
            for li in range(n_layers):
                k = rng.standard_normal((held, nkv * hd), dtype=np.float32)
                v = rng.standard_normal((held, nkv * hd), dtype=np.float32)
                kv.append(li, b, k, v)
                caches[b][0][li][:held], caches[b][1][li][:held] = store(k).reshape(held, -1), store(v).reshape(held, -1)
            kv.advance(b, held)
    for t in range(held, held + 2):
        x = rng.standard_normal((batch, dim), dtype=np.float32)
        got = model.forward(kv, x, positions=[t] * batch)
        for b in range(batch):
            want = orc.forward_token_q8(cfg, layers, output_norm, out_q8, None, cos, sin, theta, caches[b][0], caches[b][1], t, x[b], t, store=store)
            err = float(np.abs(got[b] - want).max())
            assert err <= 2e-2 * float(np.abs(want).max()), (t, b, err, float(np.abs(want).max()))
    model.free(); kv.free(); eng.close()
