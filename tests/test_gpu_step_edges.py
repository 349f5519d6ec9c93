"""RoPE + KV store and RMSNorm at the sizes where their forms change: head sizes around a warp's 32 pairs and at the
largest, head counts that do not fill a CTA, batches that take one and two heads a thread (with head counts that put a q
and a k head, or a k and a v head, into one thread), rows around what a CTA keeps in registers (8192), unaligned ones, and
more rows than the device has SMs.
RoPE within 2e-5 (rotations of values of a few units in 32 bits), the cache exact given the kernel's own rotation, bf16
rows within one unit in the last place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_head,n_kv,hd", [(1, 1, 2), (2, 1, 64), (3, 1, 34), (6, 2, 66), (5, 5, 130), (4, 2, 256), (32, 8, 128)])
@pytest.mark.parametrize("batch", [1, 3, 500])
def test_rope_and_store(n_head, n_kv, hd, batch):
    import torch
    from oracle import step_oracle as S
    from turbo_lossless_b200 import Split12Engine
    eng, T, theta = Split12Engine(), 8, 10000.0
    rng = np.random.default_rng(hd + batch)
    q, k, v = (rng.standard_normal((batch, n * hd)).astype(np.float32) for n in (n_head, n_kv, n_kv))
    v[0, :hd] = 0.0                                                  # an all-zero head: scale 0, values 0
    pos = rng.integers(0, T, batch).astype(np.int32)
    d = [torch.from_numpy(a).cuda() for a in (q, k, v)]
    kc = torch.full((batch, T, n_kv, hd), 77, dtype=torch.int8, device="cuda"); vc = kc.clone()
    sk = torch.full((batch, T, n_kv), 9.0, device="cuda"); sv = sk.clone()
    pos_d = torch.from_numpy(pos).cuda()
    qr, kr = d[0].clone(), d[1].clone()
    eng.rope_store_kv_batch(*d, kc, vc, sk, sv, pos_d, hd, n_head, n_kv, T * n_kv * hd, theta, batch)
    # the rotation alone and the store alone give the same bits
    eng.rope_batch(qr, kr, pos_d, hd, n_head, n_kv, theta, batch)
    assert torch.equal(qr, d[0]) and torch.equal(kr, d[1])
    alone = [torch.full_like(kc, 77), torch.full_like(vc, 77), torch.full_like(sk, 9.0), torch.full_like(sv, 9.0)]
    eng.store_kv_batch(kr, d[2], *alone, pos_d, n_kv, hd, batch, kv_stride=T * n_kv * hd)
    assert all(torch.equal(a, b) for a, b in zip(alone, (kc, vc, sk, sv)))
    for b in range(0, batch, max(1, batch // 50)):
        np.testing.assert_allclose(d[0][b].cpu().numpy().reshape(-1, hd), S.rope(q[b], int(pos[b]), hd, theta), rtol=0, atol=2e-5)
        rot = d[1][b].cpu().numpy().reshape(-1, hd)
        np.testing.assert_allclose(rot, S.rope(k[b], int(pos[b]), hd, theta), rtol=0, atol=2e-5)
        for cache, scales, src in ((kc, sk, rot), (vc, sv, v[b].reshape(-1, hd))):
            for h in range(n_kv):
                want, scale = S.quantize_head(src[h])
                np.testing.assert_array_equal(cache[b, pos[b], h].cpu().numpy(), want)
                assert scales[b, pos[b], h].item() == scale
            rest = np.arange(T) != pos[b]
            assert (cache[b].cpu().numpy()[rest] == 77).all() and (scales[b].cpu().numpy()[rest] == 9.0).all()


@pytest.mark.parametrize("n,B", [(n, 2) for n in (4, 127, 128, 1020, 4100, 8188, 8192, 8196, 12288)] +
                         [(n, 400) for n in (1020, 1024, 1025, 4100, 8192, 8196)])
@pytest.mark.parametrize("offset", [0, 1])
def test_rms_norm(n, B, offset):
    import torch
    from oracle import step_oracle as S
    from turbo_lossless_b200 import Split12Engine
    eng = Split12Engine()
    rng = np.random.default_rng(n)
    x, r = (rng.standard_normal((B, n)).astype(np.float32) for _ in range(2))
    w = (1 + 0.1 * rng.standard_normal(n)).astype(np.float32)
    for res in (None, r):
        room = torch.zeros(B * n + 4, device="cuda")                 # offset 1: rows off a 16-byte boundary
        xd = room[offset:offset + B * n].view(B, n)
        xd.copy_(torch.from_numpy(x))
        y = torch.zeros(B, n, dtype=torch.int16, device="cuda")
        eng.rms_norm_bf16(xd, torch.from_numpy(w).cuda(), y, 1e-5, B, residual=None if res is None else torch.from_numpy(res).cuda())
        xs, want = S.rms_norm_bf16(x, w, 1e-5, residual=res)
        np.testing.assert_array_equal(xd.cpu().numpy(), xs)
        got, want = S.bf16_to_f32(y.cpu().numpy()).astype(np.float64), S.bf16_to_f32(want).astype(np.float64)
        assert (np.abs(got - want) <= 2.0 ** -7 * np.abs(want) + 1e-30).all()
