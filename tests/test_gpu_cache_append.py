"""GPU parity of the latent cache append kernel, through the C ABI: bit-exact int8 codes and fp16 scales."""
import pytest
import torch

from conftest import load_golden
from oracle import quant, attention as oattn
from lsvd_b200 import destindex_copy_quantize_latent, cache_append, LatentCacheLayout
from lsvd_b200 import synth

pytestmark = pytest.mark.gpu


def test_append_matches_reference_fixture_both_roundings():
    g = load_golden("latent_quant")
    x = g["x"].cuda()
    T, H, R = x.shape
    # R = 24 is not a multiple of 16: the kernel wants 16-aligned ranks, so embed into R = 32 with zero padding,
    # which changes neither the absmax nor the codes of the first 24 entries.
    xp = torch.zeros(T, H, 32, dtype=torch.float16, device="cuda")
    xp[:, :, :R] = x
    for rounding, cache_ref, scale_ref in (("triton", g["cache_triton"], g["scale_triton"]), ("torch", None, None)):
        cache = torch.zeros(64, H, 32, dtype=torch.int8, device="cuda")
        scale = torch.zeros(64, H, dtype=torch.float16, device="cuda")
        destindex_copy_quantize_latent(xp, g["dest_loc"].cuda(), cache, scale, rounding=rounding)
        torch.cuda.synchronize()
        if rounding == "triton":
            assert torch.equal(scale.cpu(), scale_ref)
            assert torch.equal(cache.cpu()[:, :, :R], cache_ref)
        else:
            rows = g["dest_loc"].long()
            assert torch.equal(scale.cpu()[rows], g["s_torch"])
            assert torch.equal(cache.cpu()[rows][:, :, :R], g["q_torch"])
        assert (cache.cpu()[:, :, R:] == 0).all()


@pytest.mark.parametrize("rounding", ["torch", "triton"])
def test_append_ragged_k_and_v_one_launch(rounding):
    gen = torch.Generator().manual_seed(5)
    k_ranks, v_ranks = [16, 128, 48, 64, 32], [64, 16, 16, 112, 128]
    lay = LatentCacheLayout(k_ranks, v_ranks)
    T, N = 37, 101
    lk = (torch.randn(T, lay.sum_k, generator=gen) * 2).half()
    lv = (torch.randn(T, lay.sum_v, generator=gen) * 0.01).half()
    lk[0] = 0
    lv[1] = 60000.0
    dest = torch.randperm(N, generator=gen)[:T].to(torch.int32)
    ck = torch.full((N, lay.sum_k), 7, dtype=torch.int8)
    cv = torch.full((N, lay.sum_v), 7, dtype=torch.int8)
    sk = torch.full((N, 5), 3.0, dtype=torch.float16)
    sv = torch.full((N, 5), 3.0, dtype=torch.float16)
    ck_ref, sk_ref, cv_ref, sv_ref = ck.clone(), sk.clone(), cv.clone(), sv.clone()
    oattn.cache_append(lk, dest, lay.k_off, ck_ref, sk_ref, rounding)
    oattn.cache_append(lv, dest, lay.v_off, cv_ref, sv_ref, rounding)
    d = [t.cuda() for t in (lk, lv, dest, ck, sk, cv, sv)]
    cache_append(lay, d[0], d[1], d[2], d[3], d[4], d[5], d[6], rounding=rounding)
    torch.cuda.synchronize()
    assert torch.equal(d[3].cpu(), ck_ref) and torch.equal(d[4].cpu(), sk_ref)      # untouched rows stay untouched
    assert torch.equal(d[5].cpu(), cv_ref) and torch.equal(d[6].cpu(), sv_ref)


def test_append_strided_latent_view_like_the_reference_block():
    # the reference appends latent_kv[:, 0] and latent_kv[:, 1] of one [T, 2, H, R] projection output
    gen = torch.Generator().manual_seed(6)
    T, H, R, N = 16, 32, 64, 64
    kv = torch.randn(T, 2, H, R, generator=gen).half()
    dest = torch.arange(T, dtype=torch.int32) * 3
    for side in (0, 1):
        cache = torch.zeros(N, H, R, dtype=torch.int8, device="cuda")
        scale = torch.zeros(N, H, dtype=torch.float16, device="cuda")
        destindex_copy_quantize_latent(kv.cuda()[:, side], dest.cuda(), cache, scale)
        q, s = quant.latent_quant(kv[:, side])
        assert torch.equal(cache.cpu()[dest.long()], q) and torch.equal(scale.cpu()[dest.long()], s)


def test_append_out_of_range_slot_is_skipped_and_reported():
    lay = LatentCacheLayout.uniform(2, 16)
    lat = torch.ones(3, 32, dtype=torch.float16, device="cuda")
    dest = torch.tensor([1, 99, -4], dtype=torch.int32, device="cuda")
    ck = torch.zeros(8, 32, dtype=torch.int8, device="cuda")
    sk = torch.zeros(8, 2, dtype=torch.float16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    cache_append(lay, lat, None, dest, ck, sk, None, None, status_word=status)
    torch.cuda.synchronize()
    assert status.item() == 6
    assert (ck.cpu()[1] == 127).all() and (ck.cpu()[[0, 2, 3, 4, 5, 6, 7]] == 0).all()


def test_append_prefill_sized_batch_checksum():
    """Full prefill-sized append (32768 tokens x 32 heads x 64): compared with the oracle through a checksum."""
    T, H, R = 32768, 32, 64
    gen = torch.Generator().manual_seed(9)
    lat = torch.randn(T, H * R, generator=gen).half()
    dest = torch.randperm(T, generator=gen).to(torch.int32)
    lay = LatentCacheLayout.uniform(H, R)
    ck = torch.zeros(T, H * R, dtype=torch.int8, device="cuda")
    sk = torch.zeros(T, H, dtype=torch.float16, device="cuda")
    cache_append(lay, lat.cuda(), None, dest.cuda(), ck, sk, None, None)
    q, s = quant.latent_quant(lat.view(T, H, R))
    ck_ref = torch.empty(T, H * R, dtype=torch.int8)
    ck_ref[dest.long()] = q.view(T, -1)
    assert torch.equal(ck.cpu(), ck_ref)
    sk_ref = torch.empty(T, H, dtype=torch.float16)
    sk_ref[dest.long()] = s
    assert torch.equal(sk.cpu(), sk_ref)


@pytest.mark.parametrize("rounding", ["torch", "triton"])
def test_append_many_tokens_ragged_both_sides(rounding):
    """Thousands of tokens with ragged ranks, K and V in one launch, strided latents (views of one wider tensor) and
    slots scattered over a larger cache."""
    gen = torch.Generator().manual_seed(21)
    k_ranks, v_ranks = [16, 128, 48, 64, 32], [64, 16, 16, 112, 128]
    lay = LatentCacheLayout(k_ranks, v_ranks)
    T, N = 4001, 4100
    both = torch.randn(T, lay.sum_k + lay.sum_v, generator=gen).half()
    both[7] = 0
    lk, lv = both[:, :lay.sum_k], both[:, lay.sum_k:]                # views with a row stride of both widths
    dest = torch.randperm(N, generator=gen)[:T].to(torch.int32)
    ck = torch.zeros(N, lay.sum_k, dtype=torch.int8, device="cuda")
    cv = torch.zeros(N, lay.sum_v, dtype=torch.int8, device="cuda")
    sk = torch.zeros(N, 5, dtype=torch.float16, device="cuda")
    sv = torch.zeros(N, 5, dtype=torch.float16, device="cuda")
    gb = both.cuda()
    cache_append(lay, gb[:, :lay.sum_k], gb[:, lay.sum_k:], dest.cuda(), ck, sk, cv, sv, rounding=rounding)
    torch.cuda.synchronize()
    for lat, offs, cache, scale in ((lk, lay.k_off, ck, sk), (lv, lay.v_off, cv, sv)):
        c_ref = torch.zeros(N, lat.shape[1], dtype=torch.int8)
        s_ref = torch.zeros(N, 5, dtype=torch.float16)
        oattn.cache_append(lat.contiguous(), dest, list(offs), c_ref, s_ref, rounding=rounding)
        assert torch.equal(cache.cpu(), c_ref) and torch.equal(scale.cpu(), s_ref)


def test_append_many_tokens_out_of_range_slots_are_skipped_and_reported():
    """The same guard in the form used for thousands of tokens: bad slots are skipped, every other row is written."""
    lay = LatentCacheLayout([16, 64, 128], [32, 48, 16])
    T, N = 6000, 6000
    gen = torch.Generator().manual_seed(33)
    lk = torch.randn(T, lay.sum_k, generator=gen).half()
    lv = torch.randn(T, lay.sum_v, generator=gen).half()
    dest = torch.arange(T, dtype=torch.int32)
    dest[17], dest[4242] = N + 5, -1
    ck = torch.zeros(N, lay.sum_k, dtype=torch.int8, device="cuda")
    cv = torch.zeros(N, lay.sum_v, dtype=torch.int8, device="cuda")
    sk = torch.zeros(N, 3, dtype=torch.float16, device="cuda")
    sv = torch.zeros(N, 3, dtype=torch.float16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    cache_append(lay, lk.cuda(), lv.cuda(), dest.cuda(), ck, sk, cv, sv, status_word=status)
    torch.cuda.synchronize()
    assert status.item() == 6
    good = torch.ones(T, dtype=torch.bool)
    good[17] = good[4242] = False
    for lat, offs, cache, scale in ((lk, lay.k_off, ck, sk), (lv, lay.v_off, cv, sv)):
        q, s = quant.latent_quant_ragged(lat, list(offs))
        assert torch.equal(cache.cpu()[good], q[good]) and torch.equal(scale.cpu()[good], s[good])
        assert (cache.cpu()[~good] == 0).all() and (scale.cpu()[~good] == 0).all()


@pytest.mark.parametrize("tokens", [37, 2100])
def test_head_major_layout_holds_the_same_codes(tokens):
    """LSVD_CACHE_HEAD_MAJOR ([H][N_slots][r_h] + scales [H][N_slots]): the same codes and scales as the slot-major
    cache, in the one-warp-per-unit form (37 tokens x 5 heads x 2 sides) and in the row form (2100 tokens x 16 heads x 2
    sides of 64 chunks)."""
    gen = torch.Generator().manual_seed(tokens)
    heads = 5 if tokens < 100 else 16
    k_ranks = synth.ragged_ranks(heads, 64, seed=1) if heads == 16 else [16, 128, 48, 64, 32]
    v_ranks = synth.ragged_ranks(heads, 64, seed=2) if heads == 16 else [64, 16, 16, 112, 128]
    lay = LatentCacheLayout(k_ranks, v_ranks)
    hm = lay.as_head_major()
    N = tokens + 64
    lk = (torch.randn(tokens, lay.sum_k, generator=gen) * 2).half().cuda()
    lv = (torch.randn(tokens, lay.sum_v, generator=gen) * 0.5).half().cuda()
    dest = torch.randperm(N, generator=gen)[:tokens].to(torch.int32).cuda()
    ck, sk, cv, sv = [t.zero_() for t in lay.alloc(N)]
    hk, hsk, hv, hsv = [t.zero_() for t in hm.alloc(N)]
    cache_append(lay, lk, lv, dest, ck, sk, cv, sv)
    cache_append(hm, lk, lv, dest, hk, hsk, hv, hsv)
    torch.cuda.synchronize()
    k2, sk2 = hm.from_head_major(hk, hsk, "k")
    v2, sv2 = hm.from_head_major(hv, hsv, "v")
    assert torch.equal(k2, ck) and torch.equal(sk2, sk) and torch.equal(v2, cv) and torch.equal(sv2, sv)
    # and the conversion helpers are inverses of each other
    fk, fsk = hm.to_head_major(ck, sk, "k")
    assert torch.equal(fk, hk) and torch.equal(fsk, hsk)


@pytest.mark.parametrize("rounding", ["torch", "triton"])
@pytest.mark.parametrize("head_major", [False, True])
@pytest.mark.parametrize("pad", [0, 8])
def test_row_form_equals_the_per_head_form(rounding, head_major, pad):
    """Every fp16 magnitude, zeros, infinities and NaN through the form for many tokens (four tokens per thread, a remainder
    of two) and, a few tokens at a time, through the one-warp-per-head form: the same codes and scales, rows at 8-byte
    alignment included."""
    k_ranks, v_ranks = [16, 128, 48, 64, 32, 80, 112, 96] * 2, [64, 16, 16, 112, 128, 32, 48, 64] * 2
    lay = LatentCacheLayout(k_ranks, v_ranks, head_major=head_major)
    T, N = 2102, 2200
    gen = torch.Generator().manual_seed(7)
    bits = torch.randint(0, 0x7bff, (T, lay.sum_k + lay.sum_v), generator=gen).to(torch.int16)
    both = bits.view(torch.float16) * torch.where(torch.rand(bits.shape, generator=gen) < 0.5, -1, 1).half()
    both[1::3] = (torch.randn(both[1::3].shape, generator=gen)).half()
    both[5] = 0
    both[6, ::40], both[7, 3::50], both[8, 1::30] = float("inf"), float("-inf"), float("nan")
    both[9, ::2] = float("nan")
    both = both.cuda()
    dest = torch.randperm(N, generator=gen)[:T].to(torch.int32).cuda()

    def fresh():
        if head_major:
            return [t.zero_() for t in lay.alloc(N)]
        flat = [torch.zeros(N * (s + pad), dtype=torch.int8, device="cuda") for s in (lay.sum_k, lay.sum_v)]
        ck, cv = flat[0].view(N, -1)[:, :lay.sum_k], flat[1].view(N, -1)[:, :lay.sum_v]
        return [ck, torch.zeros(N, 16, dtype=torch.float16, device="cuda"), cv, torch.zeros(N, 16, dtype=torch.float16, device="cuda")]

    many, few = fresh(), fresh()
    cache_append(lay, both[:, :lay.sum_k], both[:, lay.sum_k:], dest, *many, rounding=rounding)
    for t in range(0, T, 3):
        cache_append(lay, both[t:t + 3, :lay.sum_k], both[t:t + 3, lay.sum_k:], dest[t:t + 3].contiguous(), *few, rounding=rounding)
    for a, b in zip(many, few):
        assert torch.equal(a.contiguous().view(torch.int8), b.contiguous().view(torch.int8))


def _same_as_per_head_form(append, tokens, fresh):
    """``append(slice, caches)`` once for all tokens and a few at a time, through the one-warp-per-head form."""
    many, few = fresh(), fresh()
    append(slice(0, tokens), many)
    for t in range(0, tokens, 3):
        append(slice(t, t + 3), few)
    for a, b in zip(many, few):
        assert torch.equal(a.view(torch.int8), b.view(torch.int8))


@pytest.mark.parametrize("rounding", ["torch", "triton"])
@pytest.mark.parametrize("heads,rank,pad,tokens", [(1, 16, 0, 8195), (1, 128, 8, 8195), (5, 48, 8, 3333), (8, 64, 8, 2051), (32, 64, 16, 515), (64, 128, 0, 259),
                                                   (128, 128, 8, 259)])
def test_many_tokens_of_gathered_heads(rounding, heads, rank, pad, tokens):
    """``destindex_copy_quantize_latent`` on heads that do not lie back to back (or rows too wide for two stages of shared
    memory), from one 16-latent chunk a token to a block of 1024 threads: the head-by-head form below 16 chunks, register loads
    of the row form above."""
    gen = torch.Generator().manual_seed(heads + rank)
    lat = torch.randn(tokens, heads, rank + pad, generator=gen).half().cuda()[:, :, :rank]
    lat[5], lat[6, 0, 3], lat[7, -1, -1] = 0, float("inf"), float("nan")
    dest = torch.randperm(tokens + 40, generator=gen)[:tokens].int().cuda()

    def append(s, caches):
        destindex_copy_quantize_latent(lat[s], dest[s], *caches, rounding=rounding)
    _same_as_per_head_form(append, tokens, lambda: (torch.zeros(tokens + 40, heads, rank, dtype=torch.int8, device="cuda"),
                                                    torch.zeros(tokens + 40, heads, dtype=torch.float16, device="cuda")))


@pytest.mark.parametrize("head_major", [False, True])
@pytest.mark.parametrize("heads,rank,tokens", [(1, 16, 4097), (2, 64, 2050), (8, 16, 515), (8, 32, 9001), (4, 128, 2051), (32, 64, 130), (32, 64, 194), (64, 128, 131), (128, 128, 33),
                                               (128, 128, 66), (128, 128, 130)])
def test_every_form_of_the_append_writes_the_same(head_major, heads, rank, tokens):
    """Both sides of the lines between the forms: rows of 1 to 1024 chunks, a remainder of tokens, both cache layouts, slots
    out of range (skipped and reported)."""
    lay = LatentCacheLayout.uniform(heads, rank)
    lay = lay.as_head_major() if head_major else lay
    gen = torch.Generator().manual_seed(heads + rank)
    both = torch.randn(tokens, 2, lay.sum_k, generator=gen).half().cuda()
    both[3] = 0
    dest = torch.randperm(tokens + 40, generator=gen)[:tokens].int().cuda()
    dest[1], dest[tokens - 1] = -1, tokens + 40
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    cache_append(lay, both[:, 0], both[:, 1], dest, *[t.zero_() for t in lay.alloc(tokens + 40)], status_word=status)
    assert int(status) == 6

    def append(s, caches):
        cache_append(lay, both[s, 0], both[s, 1], dest[s], *caches)
    _same_as_per_head_form(append, tokens, lambda: [t.zero_() for t in lay.alloc(tokens + 40)])
