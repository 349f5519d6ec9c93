"""Device packer vs the oracle packer (itself pinned to the reference's CPU packer): identical bytes."""
import numpy as np
import pytest
import torch

from conftest import GOLDEN_CASES, golden_packed
from gpu_util import dev

pytestmark = pytest.mark.gpu
FIELDS = (("split_sm", "sm"), ("split_gr", "gr"), ("row_offsets", "row_off"), ("patch_cols", "cols"),
          ("patch_correct", "correct"), ("patch_wrong", "wrong"))


def _check(cw, ref):
    assert (cw.M, cw.K, cw.base_exp, cw.num_patches) == (ref.M, ref.K, ref.base_exp, ref.num_patches)
    for a, b in FIELDS:
        t = getattr(cw, a)
        if t is None:
            assert ref.num_patches == 0
            continue
        assert np.array_equal(t.cpu().numpy(), getattr(ref, b)), a


@pytest.mark.parametrize("name", GOLDEN_CASES)
def test_golden_cases(O, golden, name):
    from turbo_lossless_b200 import CompressedWeight
    w, ref = golden_packed(O, golden, name)
    _check(CompressedWeight.pack_on_device(dev(w)), ref)


@pytest.mark.parametrize("M,K,frac", [(4096, 4096, 5e-4), (3000, 1056, 2e-2), (1, 32, 0.0), (5000, 14336, 2.5e-3)])
def test_matches_oracle_packer(O, M, K, frac):
    from turbo_lossless_b200 import CompressedWeight
    w = O.synth_weights(M, K, M + K, outlier_frac=frac)
    _check(CompressedWeight.pack_on_device(dev(w)), O.pack(w))


def test_pack_then_decompress_roundtrip_full_size():
    """lm_head-sized (128256 x 4096) random bf16 weights generated on the device: pack, decompress,
    compare bit for bit -- the round-trip property at full size, without any host copy."""
    from turbo_lossless_b200 import CompressedWeight, Split12Engine
    g = torch.Generator(device="cuda").manual_seed(1)
    w = (torch.randn(128256, 4096, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    cw = CompressedWeight.pack_on_device(w)
    assert 0 < cw.num_patches < 0.001 * w.numel()
    out = Split12Engine().decompress(cw)
    assert torch.equal(out, w.view(torch.int16))


def test_pack_under_dependent_launch(O, golden):
    """The packer's five kernels each consume their predecessor's output; with programmatic dependent launch
    enabled every one of them waits for it before reading."""
    from turbo_lossless_b200 import CompressedWeight, Split12Engine
    eng = Split12Engine()
    old = eng.set_dependent_launch(True)
    try:
        for name in GOLDEN_CASES:
            w, ref = golden_packed(O, golden, name)
            _check(CompressedWeight.pack_on_device(dev(w)), ref)
        w = O.synth_weights(3000, 4096, 3, outlier_frac=1e-2)
        for _ in range(3):
            _check(CompressedWeight.pack_on_device(dev(w)), O.pack(w))
    finally:
        eng.set_dependent_launch(old)


@pytest.mark.parametrize("M,K,frac", [(1, 2, 1.0), (5, 6, 0.5), (3, 8, 0.3), (7, 24, 0.2), (2, 1032, 0.1), (3, 4104, 1e-2), (1, 16384, 0.9),
                                      (9, 2056, 0.33), (40, 264, 0.34), (40, 248, 0.34), (1023, 16, 0.2), (1025, 16, 0.2), (2049, 8, 0.2), (4097, 6, 0.1), (8191, 8, 0.1), (8192, 34, 0.05), (8193, 16, 0.1), (20000, 40, 0.02)])
@pytest.mark.parametrize("offset", [0, 1, 8])
def test_edges_of_the_passes(O, M, K, frac, offset):
    """Rows around the scan's 1024 to 8192, columns around the fill's 256 and 1024, values off a 16-byte boundary (offset
    elements into a buffer): one call, and the separate passes on the same values."""
    from turbo_lossless_b200 import CompressedWeight, capi
    from turbo_lossless_b200.capi import check
    rng = np.random.default_rng(M + K)
    w = O.synth_weights(M, K, M + K, outlier_frac=0.0)
    w = np.where(rng.random((M, K)) < frac, rng.integers(0, 1 << 16, (M, K), dtype=np.uint16), w)   # any exponent
    ref = O.pack(w)
    room = torch.zeros(M * K + 16, dtype=torch.int16, device="cuda")
    wd = room[offset:offset + M * K].view(M, K)
    wd.copy_(dev(w))
    _check(CompressedWeight.pack_on_device(wd), ref)
    _check(CompressedWeight.pack_on_device(wd, base_exp=ref.base_exp), ref)
    lib = capi.load()
    hist = torch.empty(256, dtype=torch.int64, device="cuda")
    check(lib.s12_pack_histogram_async(wd.data_ptr(), M * K, hist.data_ptr(), None))
    assert np.array_equal(hist.cpu().numpy(), np.bincount((w.reshape(-1) >> 7) & 0xFF, minlength=256))
    if ref.num_patches:
        got = [torch.zeros(ref.num_patches, dtype=d, device="cuda") for d in (torch.int32, torch.int16, torch.int16)]
        check(lib.s12_pack_fill_async(wd.data_ptr(), M, K, ref.base_exp, dev(ref.row_off).data_ptr(), *[t.data_ptr() for t in got], None))
        for t, a in zip(got, (ref.cols, ref.correct, ref.wrong)):
            assert np.array_equal(t.cpu().numpy(), a)


@pytest.mark.parametrize("base_exp", [-1, 0, 100, 112, 239, 240, 241, 254, -9])
def test_given_window_over_every_value(O, base_exp):
    """All 65536 bf16 patterns (their sixteen-element chunks hold neighbouring exponents) with a window given by the caller."""
    from turbo_lossless_b200 import CompressedWeight
    w = np.random.default_rng(1).permutation(np.arange(1 << 16, dtype=np.uint32)).astype(np.uint16).reshape(256, 256)
    cw = CompressedWeight.pack_on_device(dev(w), base_exp=base_exp)
    e = ((w >> 7) & 0xFF).astype(np.int32) - base_exp
    grp = np.where((e >= 1) & (e <= 15), e, 0).astype(np.uint8).reshape(-1)
    assert np.array_equal(cw.split_sm.cpu().numpy(), (((w >> 15) << 7) | (w & 0x7F)).astype(np.uint8).reshape(-1))
    assert np.array_equal(cw.split_gr.cpu().numpy(), grp[0::2] | (grp[1::2] << 4))
    rows, cols = np.nonzero(grp.reshape(w.shape) == 0)
    assert cw.num_patches == len(cols) and np.array_equal(cw.patch_cols.cpu().numpy(), cols)
    assert np.array_equal(cw.row_offsets.cpu().numpy(), np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=256))]))
    assert np.array_equal(cw.patch_correct.cpu().numpy().view(np.uint16), w[rows, cols])


def test_rows_within_a_scan_round_of_the_largest_int():
    """As many rows as a 32-bit count holds, less than the scan's 8192 rows from its end (24 GB of tensors)."""
    from turbo_lossless_b200 import capi
    from turbo_lossless_b200.capi import check
    M, K = 2 ** 31 - 6000, 2
    if torch.cuda.mem_get_info()[0] < 40e9:
        pytest.skip("needs 24 GB of device memory")
    w = torch.full((M * K,), 0x3F80, dtype=torch.int16, device="cuda")            # 1.0: exponent 127
    rows = torch.tensor([0, 1023, 8191, 8192, 5 * 10 ** 8, M - 8192, M - 2, M - 1], device="cuda")
    w[rows * K + 1] = 0
    sm, gr = (torch.empty(M * K // n, dtype=torch.uint8, device="cuda") for n in (1, 2))
    row_off = torch.empty(M + 1, dtype=torch.int32, device="cuda")
    check(capi.load().s12_pack_async(w.data_ptr(), M, K, 120, sm.data_ptr(), gr.data_ptr(), row_off.data_ptr(), None))
    for a in range(0, M + 1, 1 << 28):
        at = torch.arange(a, min(a + (1 << 28), M + 1), device="cuda")
        assert torch.equal(row_off[a:a + (1 << 28)], torch.searchsorted(rows, at, out_int32=True))   # escapes in the rows before
    del w, sm, gr, row_off, at
    torch.cuda.empty_cache()                                                     # later tests watch the driver's allocations
