"""The tensor-core attention over the forms it takes: head sizes, query heads per kv head, lengths around its 16-position
chunks, its 64-position slices and its splits.  Each call is compared with the float64 statement and with the general
kernel on the same values (a cache that starts 4 bytes off a 16-byte boundary takes that one).

Tolerance: a bf16 output (8 significant bits) is within half a unit in the last place, 2^-8 of the value; the 32-bit sums in
between within 2^-16 of the largest weighted value (a few hundred roundings of 2^-24)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def both(n_head, n_kv, hd, lengths, seed=0, edit=None):
    import torch
    from turbo_lossless_b200 import Split12Engine
    eng = Split12Engine()
    rng = np.random.default_rng(seed)
    B, T = len(lengths), max(lengths)
    c = dict(q=rng.standard_normal((B, n_head * hd)).astype(np.float32),
             k=rng.integers(-127, 128, (B, T, n_kv, hd)).astype(np.int8), v=rng.integers(-127, 128, (B, T, n_kv, hd)).astype(np.int8),
             sk=(rng.random((B, T, n_kv)) * 0.03).astype(np.float32), sv=(rng.random((B, T, n_kv)) * 0.03).astype(np.float32))
    c["k"][..., 0] = -128; c["v"][..., 1] = -128                       # the whole int8 range counts
    if edit:
        edit(c)
    pos = torch.from_numpy(np.array(lengths, np.int32) - 1).cuda()
    d = {n: torch.from_numpy(a).cuda() for n, a in c.items()}
    outs = []
    for off in (0, 4):
        kv = []
        for n in ("k", "v"):
            room = torch.zeros(d[n].numel() + 16, dtype=torch.int8, device="cuda")
            assert room.data_ptr() % 16 == 0
            room[off:off + d[n].numel()] = d[n].flatten()
            kv.append(room[off:])
        out = torch.zeros(B, n_head * hd, dtype=torch.int16, device="cuda")
        eng.attention_all_heads_batch(d["q"], kv[0], kv[1], d["sk"], d["sv"], out, pos, n_head, n_kv, hd, T,
                                      1.0 / float(np.sqrt(hd)), B, T * n_kv * hd)
        outs.append(out.view(torch.bfloat16).double().cpu().numpy())
    return c, outs


def exact(c, b, n, n_head, n_kv, hd):
    g = n_head // n_kv
    k = c["k"][b, :n].astype(np.float64)
    v = c["v"][b, :n].astype(np.float64) * c["sv"][b, :n].astype(np.float64)[..., None]
    s = np.einsum("hgd,thd->hgt", c["q"][b].astype(np.float64).reshape(n_kv, g, hd), k) / np.sqrt(hd)
    s *= c["sk"][b, :n].astype(np.float64).T[:, None, :]              # after the sum, as both kernels do
    p = np.exp(s - s.max(axis=-1, keepdims=True))
    p /= p.sum(axis=-1, keepdims=True)
    return np.einsum("hgt,thd->hgd", p, v).reshape(-1), np.einsum("hgt,thd->hgd", p, np.abs(v)).reshape(-1)


@pytest.mark.parametrize("hd", [64, 96, 128])
@pytest.mark.parametrize("n_head,n_kv", [(1, 1), (4, 2), (8, 2), (16, 2), (32, 8)])
@pytest.mark.parametrize("lengths", [(1,), (15, 16, 17), (63, 64, 65, 1), (127, 130, 2, 33), (1000, 520), (9,) * 40])
def test_against_float64_and_the_general_kernel(hd, n_head, n_kv, lengths):
    c, (new, general) = both(n_head, n_kv, hd, lengths, seed=hd + n_head + len(lengths))
    for b, n in enumerate(lengths):
        want, size = exact(c, b, n, n_head, n_kv, hd)
        bound = 2.0 ** -8 * np.abs(want) * (1 + 2.0 ** -8) + 2.0 ** -16 * size.max()
        assert (np.abs(new[b] - want) <= bound).all(), np.abs(new[b] - want).max()
        assert (np.abs(new[b] - general[b]) <= 2 * bound).all()


@pytest.mark.parametrize("n_head", [8, 16])
@pytest.mark.parametrize("what", ["q", "sk", "sv", "large"])
def test_infinities_and_the_largest_values(what, n_head):
    """One infinite input, and value scales near the end of the 32-bit range.  An invalid 64-bit result is stored as 0x8000
    (what the rounding to bf16 makes of the hardware's NaN) and an infinity as itself, by both kernels; everything else,
    such as the heads that the infinity does not touch, is as near to 64 bits as elsewhere."""
    def edit(c):
        if what == "q":
            c["q"][0, 5] = np.inf
        elif what == "large":
            c["sv"][0, 3, 0] = 2e36
        else:
            c[what][0, 3, 0] = np.inf
    lengths, n_kv, hd = (40, 20), 2, 128
    c, outs = both(n_head, n_kv, hd, lengths, seed=3, edit=edit)
    with np.errstate(invalid="ignore"):
        wants = [exact(c, b, n, n_head, n_kv, hd) for b, n in enumerate(lengths)]
    assert what == "large" or not np.isfinite(wants[0][0]).all()
    assert np.isfinite(wants[0][0]).any() and np.isfinite(wants[1][0]).all()
    for out in outs:
        raw = (out.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
        for b, (want, size) in enumerate(wants):
            bad, fine = np.isnan(want), np.isfinite(want)
            assert (raw[b][bad] == 0x8000).all()
            assert np.array_equal(out[b][~bad & ~fine], want[~bad & ~fine])
            top = np.repeat(size.reshape(n_head, hd).max(axis=1), hd)[fine]
            assert (np.abs(out[b][fine] - want[fine]) <= 2.0 ** -8 * np.abs(want[fine]) * (1 + 2.0 ** -8) + 2.0 ** -16 * top).all()


def on_device(n_kv, gqa, hd, lengths, seed, off=0):
    """The call's outputs, and the float64 statement's with the sums of magnitudes, all on the device."""
    import torch
    from turbo_lossless_b200 import Split12Engine
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, T, n_head = len(lengths), max(lengths), n_kv * gqa
    kv = [torch.randint(-127, 128, (B * T * n_kv * hd + 16,), dtype=torch.int8, device="cuda", generator=g)[off:] for _ in range(2)]
    q = torch.randn(B, n_head * hd, device="cuda", generator=g)
    sk, sv = (0.03 * torch.rand(B, T, n_kv, device="cuda", generator=g) for _ in range(2))
    pos = torch.tensor(lengths, dtype=torch.int32, device="cuda") - 1
    out = torch.zeros(B, n_head * hd, dtype=torch.bfloat16, device="cuda")
    Split12Engine().attention_all_heads_batch(q, kv[0], kv[1], sk, sv, out.view(torch.int16), pos, n_head, n_kv, hd, T, hd ** -0.5, B, T * n_kv * hd)
    k, v = (t[:B * T * n_kv * hd].view(B, T, n_kv, hd) for t in kv)
    want, size = [], []
    for b, n in enumerate(lengths):
        vb = v[b, :n].double() * sv[b, :n].double()[..., None]
        s = torch.einsum("hgd,thd->hgt", q[b].double().view(n_kv, gqa, hd), k[b, :n].double() * sk[b, :n].double()[..., None]) * hd ** -0.5
        p = torch.softmax(s, dim=-1)
        want.append(torch.einsum("hgt,thd->hgd", p, vb).reshape(-1)); size.append(torch.einsum("hgt,thd->hgd", p, vb.abs()).max())
    return out.double(), torch.stack(want), torch.stack(size)[:, None]


@pytest.mark.parametrize("hd", [64, 96, 128])
@pytest.mark.parametrize("gqa", [1, 4, 8])
@pytest.mark.parametrize("lengths", [(2048,), (4099, 2050), (16001,), tuple(range(461, 685)), tuple(range(1500, 1540)) * 3])
def test_long_enough_to_go_round_the_ring(hd, gqa, lengths):
    """Warps with four to sixteen chunks, the last one partial, so that every stage of the ring is filled again: few sequences
    (eight warps a CTA, eight slices), 224 of them (one slice) and 120 (two)."""
    got, want, size = on_device(2, gqa, hd, lengths, hd + gqa)
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() * (1 + 2.0 ** -8) + 2.0 ** -16 * size).all()


@pytest.mark.parametrize("hd,gqa,lengths,off", [(32, 1, (1, 33, 100), 0), (80, 4, (300, 17), 0), (4, 2, (9, 64), 0), (132, 8, (50, 129), 0),
                                                (256, 1, (200, 1), 0), (256, 2, (77,), 0), (256, 4, (1000, 3), 0), (256, 8, (65, 64), 0),
                                                (128, 4, (9000,) * 40, 4), (64, 8, (9000, 5000), 4), (256, 4, (9000,) * 40, 0)])
def test_general_kernel(hd, gqa, lengths, off):
    """What only the general kernel takes: other head sizes, caches off a 16-byte boundary, and contexts whose slices grow in
    number until a CTA's scores fit its shared memory (9000 positions)."""
    got, want, size = on_device(2, gqa, hd, lengths, hd + gqa, off)
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() * (1 + 2.0 ** -8) + 2.0 ** -16 * size).all()


@pytest.mark.parametrize("n_kv,gqa,hd,B,T", [(8, 8, 128, 64, 1000), (8, 8, 64, 256, 128), (8, 8, 96, 64, 1000), (8, 4, 128, 56, 7000),
                                             (8, 1, 64, 112, 3500), (8, 1, 128, 1024, 16), (8, 4, 64, 256, 300), (2, 2, 96, 512, 200)])
def test_as_near_to_64_bits_as_the_general_kernel(n_kv, gqa, hd, B, T):
    """Outputs that are not the bf16 value nearest to the 64-bit result, counted over several hundred thousand of them:
    no more than the general kernel has, within four standard deviations of the two counts' difference (each such output
    is an independent rare event, so a count's variance is the count)."""
    import torch
    from turbo_lossless_b200 import Split12Engine
    eng = Split12Engine()
    g = torch.Generator(device="cuda").manual_seed(T + hd)
    n_head, shape, wrong = n_kv * gqa, (B, T, n_kv, hd), [0, 0]
    for _ in range(max(1, 2000000 // (B * n_head * hd))):
        room = [torch.randint(-127, 128, (B * T * n_kv * hd + 16,), dtype=torch.int8, device="cuda", generator=g) for _ in range(2)]
        q = torch.randn(B, n_head * hd, device="cuda", generator=g)
        sk, sv = (0.01 + 0.02 * torch.rand(B, T, n_kv, device="cuda", generator=g) for _ in range(2))
        pos = torch.randint(T // 2, T, (B,), dtype=torch.int32, device="cuda", generator=g)
        outs = [torch.zeros(B, n_head * hd, dtype=torch.int16, device="cuda") for _ in range(2)]
        # the general kernel on the same bytes, 4 off a 16-byte boundary
        for out, off in zip(outs, (0, 4)):
            if off:
                for r in room:
                    r[off:off + r.numel() - 16] = r[:r.numel() - 16].clone()
            eng.attention_all_heads_batch(q, room[0][off:], room[1][off:], sk, sv, out, pos, n_head, n_kv, hd, T, hd ** -0.5, B, T * n_kv * hd)
        k, v = (r[4:4 + B * T * n_kv * hd].view(shape) for r in room)
        for b in range(B):
            n = int(pos[b]) + 1
            kb, vb = k[b, :n].double() * sk[b, :n].double()[..., None], v[b, :n].double() * sv[b, :n].double()[..., None]
            s = torch.einsum("hgd,thd->hgt", q[b].double().view(n_kv, gqa, hd), kb) * hd ** -0.5
            want = torch.einsum("hgt,thd->hgd", torch.softmax(s, dim=-1), vb).float().to(torch.bfloat16).view(torch.int16).reshape(-1)
            for i in range(2):
                wrong[i] += int((outs[i][b] != want).sum())
    assert wrong[0] <= wrong[1] + 4.0 * (wrong[0] + wrong[1]) ** 0.5, wrong


@pytest.mark.parametrize("hd,off", [(128, 0), (64, 0), (128, 4), (80, 0)])
@pytest.mark.parametrize("bound", [1, 17, 101, 1003])
def test_positions_past_the_bound_read_nothing_past_it(hd, off, bound):
    """Device positions at and past the caller's bound give the result at the bound, in both kernels (a cache 4 bytes off
    a 16-byte boundary and a head size of 80 take the general one).  The cache goes on past the bound, with values that would show."""
    import torch
    from turbo_lossless_b200 import Split12Engine
    eng = Split12Engine()
    g = torch.Generator(device="cuda").manual_seed(bound)
    n_kv, B, room = 2, 3, bound + 64
    kv = [torch.randint(-127, 128, (B * room * n_kv * hd + 16,), dtype=torch.int8, device="cuda", generator=g) for _ in range(2)]
    q = torch.randn(B, 8 * hd, device="cuda", generator=g)
    sk, sv = (0.01 + 0.02 * torch.rand(B, room, n_kv, device="cuda", generator=g) for _ in range(2))
    sv[:, bound:] = 1e9
    outs = []
    for at in (bound - 1, bound, bound + 40):
        out = torch.zeros(B, 8 * hd, dtype=torch.int16, device="cuda")
        pos = torch.full((B,), at, dtype=torch.int32, device="cuda")
        eng.attention_all_heads_batch(q, kv[0][off:], kv[1][off:], sk, sv, out, pos, 8, n_kv, hd, bound, hd ** -0.5, B, room * n_kv * hd)
        outs.append(out)
    assert outs[0].any() and torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("hd,gqa", [(64, 1), (96, 8), (128, 4), (128, 8)])
@pytest.mark.parametrize("length", [20, 130, 600])
def test_output_off_an_eight_byte_boundary(hd, gqa, length):
    """The same bits wherever the output starts: one slice and several, merged one and four elements a thread."""
    import torch
    from turbo_lossless_b200 import Split12Engine
    g = torch.Generator(device="cuda").manual_seed(length)
    k, v = (torch.randint(-127, 128, (length * hd,), dtype=torch.int8, device="cuda", generator=g) for _ in range(2))
    q, sk, sv = torch.randn(gqa * hd, device="cuda", generator=g), *(0.03 * torch.rand(length, device="cuda", generator=g) for _ in range(2))
    room = torch.zeros(3, gqa * hd + 4, dtype=torch.int16, device="cuda")
    pos = torch.full((1,), length - 1, dtype=torch.int32, device="cuda")
    for i in range(3):                                             # rows of a multiple of 8 bytes: 0, 2 and 4 bytes off
        Split12Engine().attention_all_heads_batch(q, k, v, sk, sv, room[i, i:], pos, gqa, 1, hd, length, hd ** -0.5, 1, length * hd)
    assert room[0].any() and all(torch.equal(room[0, :gqa * hd], room[i, i:i + gqa * hd]) for i in (1, 2))
    assert not room[1, 0] and not room[0, gqa * hd:].any()
