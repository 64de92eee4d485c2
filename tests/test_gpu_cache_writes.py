"""The kernels that store many rows at once against the same rows stored one by one: byte for byte, every plane."""
import numpy as np
import pytest

from util import assert_bits_equal

pytestmark = pytest.mark.gpu
PLANES = {"f32": (0, 1), "q8": (2, 3, 4, 5), "g32": (2, 3, 4, 5, 8, 9)}


def _planes(fb, kv, cache, seq):
    return [kv.export_plane(1, seq, p) for p in PLANES[cache]]


@pytest.mark.parametrize("cache,nkv,hd,max_seq,first,rows,offset", [
    ("q8", 8, 64, 128, 0, 100, 0), ("q8", 3, 32, 64, 60, 9, 0),       # one pass; across the end of the ring, 24 lanes a row
    ("q8", 1, 32, 33, 5, 33, 1), ("q8", 8, 128, 70, 3, 150, 0),       # sources on a 4-byte boundary; more rows than slots
    ("f32", 3, 64, 96, 90, 40, 0), ("f32", 3, 64, 96, 0, 7, 1),       # quads; scalar for the sources' sake
    ("f32", 1, 6, 11, 4, 30, 0),                                      # scalar for the row's sake, more rows than slots
])
def test_append_equals_rows_one_by_one(cache, nkv, hd, max_seq, first, rows, offset):
    import torch
    import flarellm_b200 as fb
    kvd = nkv * hd
    rng = np.random.default_rng(rows + kvd)
    eng = fb.Engine(0)
    a, b = (eng.kv_alloc(2, 2, max_seq, nkv, hd, fb.KV_F32 if cache == "f32" else fb.KV_Q8_0) for _ in range(2))
    k = rng.standard_normal((first + rows, kvd), dtype=np.float32)
    v = rng.standard_normal((first + rows, kvd), dtype=np.float32)
    k[first, :3] = 0.0
    for t in range(first + rows):
        b.write(1, 1, t, k[t], v[t])
        b.advance(1, 1)
    for t in range(first):
        a.write(1, 1, t, k[t], v[t])
        a.advance(1, 1)
    dev = torch.zeros(2, rows * kvd + offset, device="cuda")
    dev[0, offset:] = torch.from_numpy(k[first:].reshape(-1)).cuda()
    dev[1, offset:] = torch.from_numpy(v[first:].reshape(-1)).cuda()
    dk, dv = dev[0, offset:], dev[1, offset:].clone() if not offset else dev[1, offset:]
    torch.cuda.synchronize()
    a.append(1, 1, dk.data_ptr(), dv.data_ptr(), n_rows=rows)
    a.advance(1, rows)
    for got, want in zip(_planes(fb, a, cache, 1), _planes(fb, b, cache, 1)):
        assert_bits_equal(got, want, f"{cache} planes")
    a.free(); b.free(); eng.close()


@pytest.mark.parametrize("nkv,hd,lengths,max_seq", [
    (8, 64, [0, 1, 127, 128, 159, 160], 256),       # before, at and between the tokens that send a group to the codes
    (1, 32, [256, 300, 511, 512], 256),             # wrapped rings, a trigger among them
    (4, 64, [5, 9], 128),                           # nobody triggers: the narrow launch
])
def test_g32_step_of_a_batch_equals_one_sequence_at_a_time(nkv, hd, lengths, max_seq):
    import flarellm_b200 as fb
    kvd, batch = nkv * hd, len(lengths)
    rng = np.random.default_rng(kvd + batch)
    eng = fb.Engine(0)
    a, b = (eng.kv_alloc(2, batch, max_seq, nkv, hd, fb.KV_KIVI_G32) for _ in range(2))
    for s, n in enumerate(lengths):
        if n:
            k, v = rng.standard_normal((2, n, kvd), dtype=np.float32)
            for kv in (a, b):
                for lo in range(0, n, max_seq):
                    m = min(max_seq, n - lo)
                    kv.append(1, s, k[lo:lo + m], v[lo:lo + m])
                    kv.advance(s, m)
    for step in range(3):
        k, v = rng.standard_normal((2, batch, kvd), dtype=np.float32)
        a.write_step(1, k, v)
        for s in range(batch):
            b.append(1, s, k[s:s + 1], v[s:s + 1])
        for s in range(batch):
            for got, want in zip(_planes(fb, a, "g32", s), _planes(fb, b, "g32", s)):
                assert_bits_equal(got, want, f"step {step}, sequence {s}")
        a.advance(-1, 1); b.advance(-1, 1)
    a.free(); b.free(); eng.close()
