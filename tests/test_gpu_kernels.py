"""Each CUDA kernel alone against its plain reference, at sizes other than the engine's
tiny models use: widths and vocabularies that are no power of two, odd head counts, every
head size in steps of 16, pages of several sizes."""

from __future__ import annotations

import math
import random

import pytest
import torch

from plain_llama import apply_rope, causal_attention, plain_inv_freq, processed_probs, rms_norm, rope_cos_sin

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16]


def tol(dtype):
    return 2e-6 if dtype == torch.float32 else 1e-2


@pytest.fixture(scope="module")
def ops():
    from kvforge_b200 import ops as o

    return o


_ERR = None


def err_flag():
    """The device error flag that kernels with bounded waits raise."""
    global _ERR
    if _ERR is None:
        _ERR = torch.zeros(4, dtype=torch.int32, device="cuda")
    return _ERR


def dev(t, dtype=None):
    return t.to(device="cuda", dtype=dtype or t.dtype).contiguous()


@pytest.mark.parametrize("dtype", DTYPES)
def test_embed(ops, dtype):
    table = torch.randn(37, 100).to(dtype)
    ids = torch.tensor([0, 36, 5, 5, 17], dtype=torch.int32)
    out = torch.empty(5, 100, device="cuda")
    ops.embed(dev(table), dev(ids), out)
    assert torch.equal(out.cpu(), table[ids.long()].float())


# widths on every path of the launcher: no multiple of 4; 1, 2, 4 and 8 loads of 16 bytes per thread of the
# kernel that holds a row in registers; just past its limit; the kernel with the row in shared memory
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("h,n", [(6, 7), (24, 7), (100, 7), (1000, 7), (2048, 7), (3000, 300), (4096, 7), (4100, 7), (5120, 7), (1536, 1500)])
def test_add_rmsnorm(ops, dtype, h, n):
    resid = torch.randn(n, h) * 3
    delta = (torch.randn(n, h)).to(dtype)
    w = torch.rand(h) + 0.5
    r = dev(resid)
    out = torch.empty(n, h, device="cuda", dtype=dtype)
    ops.add_rmsnorm(r, dev(delta), dev(w), out, 1e-5)
    summed = resid + delta.float()
    assert torch.allclose(r.cpu(), summed, atol=1e-6)
    ref = rms_norm(summed, w, 1e-5)
    assert torch.allclose(out.float().cpu(), ref, rtol=tol(dtype) * 4, atol=tol(dtype) * 4)
    # gathered rows (a row twice), with a pending sum that must not be written back
    rows = torch.tensor([n - 1, 0, n - 1], dtype=torch.int32)
    r2 = dev(resid)
    out2 = torch.empty(3, h, device="cuda", dtype=dtype)
    ops.add_rmsnorm(r2, dev(delta), dev(w), out2, 1e-5, rows=dev(rows))
    assert torch.equal(r2.cpu(), resid)
    assert torch.allclose(out2.float().cpu(), ref[rows.long()], rtol=tol(dtype) * 4, atol=tol(dtype) * 4)
    # no pending sum
    ops.add_rmsnorm(r2, None, dev(w), out, 1e-6)
    assert torch.allclose(out.float().cpu(), rms_norm(resid, w, 1e-6), rtol=tol(dtype) * 4, atol=tol(dtype) * 4)


@pytest.mark.parametrize("dtype", DTYPES)
def test_silu_mul(ops, dtype):
    gu = (torch.randn(5, 2 * 93) * 3).to(dtype)
    out = torch.empty(5, 93, device="cuda", dtype=dtype)
    ops.silu_mul(dev(gu), out)
    g, u = gu[:, :93].float(), gu[:, 93:].float()
    ref = torch.nn.functional.silu(g) * u
    assert torch.allclose(out.float().cpu(), ref, rtol=tol(dtype) * 4, atol=tol(dtype) * 4)
    with pytest.raises(ValueError):
        ops.silu_mul(dev(gu), out, interleaved=True)  # 93 is no multiple of 8


@pytest.mark.parametrize("m,n,k", [(1, 100, 33), (7, 64, 64), (130, 203, 80), (65, 3, 1000)])
def test_gemm_f32_is_true_float32(ops, m, n, k):
    a, w = torch.randn(m, k), torch.randn(n, k)
    out = torch.empty(m, n, device="cuda")
    ops.gemm_nt_f32(dev(a), dev(w), out)
    ref = (a.double() @ w.double().t())
    # float32 accumulation error grows like sqrt(k) * 2^-24; tf32 or bfloat16 inputs would be ~1e-3
    assert float((out.cpu().double() - ref).abs().max()) < 2e-6 * math.sqrt(k) * float(ref.abs().max())


@pytest.mark.parametrize("n,k", [(150, 96), (2048, 2048), (203, 1000), (64, 8192), (9, 4), (331, 130)])
def test_gemm_f32_rows_do_not_depend_on_the_batch(ops, n, k):
    """Up to 16 rows take a kernel of their own, up to 64 tiles of 64 x 64, more rows tiles of
    128 x 128; all add a row's products in the order of k, so a row has the same bits alone, among
    a handful and among hundreds.  (K = 130 is no multiple of 4: the tiled kernels take every count.)"""
    g = torch.Generator().manual_seed(n + k)
    a, w = torch.randn(200, k, generator=g), torch.randn(n, k, generator=g)
    full = torch.empty(200, n, device="cuda")
    ops.gemm_nt_f32(dev(a), dev(w), full)
    ref = a.double() @ w.double().t()
    assert float((full.cpu().double() - ref).abs().max()) < 2e-6 * math.sqrt(k) * float(ref.abs().max())
    # 1, 16 and 9 rows: the kernel of few rows; 17 and 64 rows: tiles of 64 x 64; all 200 (with more than 64 columns): tiles of 128 x 128
    for lo, hi in ((137, 138), (0, 16), (100, 109), (30, 47), (120, 184)):
        part = torch.full((hi - lo, n), float("nan"), device="cuda")
        ops.gemm_nt_f32(dev(a[lo:hi]), dev(w), part)
        assert torch.equal(part, full[lo:hi]), (lo, hi)


@pytest.mark.parametrize("m,n,k", [(128, 18944, 20), (129, 16500, 36), (300, 16383, 17), (130, 9500, 52), (200, 4101, 130), (65, 20100, 16), (33, 1000, 64), (17, 67, 9)])
def test_gemm_f32_every_tile_shape_gives_the_bits_of_few_rows(ops, m, n, k):
    """Shapes that take each of the four tile shapes (128 x 128, twice 64 x 128, twice 64 x 64, three times 32 x 64), with
    ragged last tiles, odd columns and a K that is no multiple of the tile's depth."""
    g = torch.Generator().manual_seed(m + n + k)
    a, w = torch.randn(m, k, generator=g), torch.randn(n, k, generator=g)
    wide = torch.full((m, n + 3), float("nan"), device="cuda")
    ops.gemm_nt_f32(dev(a), dev(w), wide[:, :n])
    assert torch.isnan(wide[:, n:]).all()
    ref = a.double() @ w.double().t()
    assert float((wide[:, :n].cpu().double() - ref).abs().max()) < 2e-6 * math.sqrt(k) * float(ref.abs().max())
    for lo in (0, (m - 11) // 2, m - 11):
        part = torch.empty(11, n, device="cuda")
        ops.gemm_nt_f32(dev(a[lo : lo + 11]), dev(w), part)
        assert torch.equal(part, wide[lo : lo + 11, :n]), lo


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("many", [False, True])  # a few tokens and many tokens take different kernels
@pytest.mark.parametrize("nh,nkv,d,rot,bs", [(4, 2, 16, 16, 16), (3, 1, 32, 32, 8), (6, 3, 48, 24, 4), (5, 5, 128, 128, 32)])
def test_rope_and_cache_write(ops, dtype, nh, nkv, d, rot, bs, many):
    base = [0, 1, 2, 63, 64, 65, 1000, 4095, 4096, 7, 8]
    positions = torch.tensor(base + ([p + 3 for p in base] + [p + 17 for p in base] + [p + 90 for p in base] if many else []), dtype=torch.int32)
    n = positions.numel()
    nb = -(-n // bs) + 8
    qkv = torch.randn(n, (nh + 2 * nkv) * d).to(dtype)
    inv = plain_inv_freq(rot, 500000.0)
    slots = torch.tensor(random.Random(1).sample(range(nb * bs), n), dtype=torch.int32)
    kc = torch.zeros(nb, nkv, bs, d, device="cuda", dtype=dtype)
    vc = torch.zeros_like(kc)
    x = dev(qkv)
    ops.rope_cache_write(x, dev(positions), dev(inv), dev(slots), kc, vc, nh, nkv, d, bs)
    cos, sin = rope_cos_sin(positions, inv)

    def rotated(t):  # [n, heads, d]; only the first `rot` dims turn
        return torch.cat([apply_rope(t[..., :rot], cos, sin), t[..., rot:]], dim=-1)

    q = qkv[:, : nh * d].view(n, nh, d)
    k = qkv[:, nh * d : (nh + nkv) * d].view(n, nkv, d)
    v = qkv[:, (nh + nkv) * d :].view(n, nkv, d)
    t = tol(dtype) * 8
    assert torch.allclose(x[:, : nh * d].float().cpu().view(n, nh, d), rotated(q).float(), rtol=t, atol=t)
    kc_flat = kc.float().cpu().permute(0, 2, 1, 3).reshape(nb * bs, nkv, d)
    vc_flat = vc.float().cpu().permute(0, 2, 1, 3).reshape(nb * bs, nkv, d)
    assert torch.allclose(kc_flat[slots.long()], rotated(k).float(), rtol=t, atol=t)
    assert torch.equal(vc_flat[slots.long()], v.float())
    untouched = torch.ones(nb * bs, dtype=torch.bool)
    untouched[slots.long()] = False
    assert (kc_flat[untouched] == 0).all() and (vc_flat[untouched] == 0).all()


@pytest.mark.parametrize("m", [1, 3, 8, 9, 16, 31, 64])
@pytest.mark.parametrize("n,k", [(64, 64), (203, 80), (3072, 2048), (100, 1000), (2048, 8192), (16, 8)])
def test_gemm_skinny(ops, m, n, k):
    g = torch.Generator().manual_seed(m * 1000 + n + k)
    x = torch.randn(m, k, generator=g).bfloat16()
    w = (torch.randn(n, k, generator=g) * 0.1).bfloat16()
    ref = x.double() @ w.double().t()
    scale = float(ref.abs().max())
    out16 = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    ops.gemm_skinny(dev(x), dev(w), out16)
    assert float((out16.double().cpu() - ref).abs().max()) < 1e-2 * scale
    out32 = torch.empty(m, n, device="cuda")
    ops.gemm_skinny(dev(x), dev(w), out32)
    assert float((out32.double().cpu() - ref).abs().max()) < 2e-5 * scale * max(1.0, k**0.5 / 8)
    for splits in {1, ops.skinny_splits(n, k), min(3, max(1, k // 64))}:
        part = ops.Partials(torch.full((splits, m, n), float("nan"), device="cuda"))
        ops.gemm_skinny(dev(x), dev(w), part)
        assert float((part.t.double().sum(0).cpu() - ref).abs().max()) < 2e-5 * scale * max(1.0, k**0.5 / 8), splits


def test_gemm_skinny_rows_do_not_depend_on_the_batch(ops):
    x = torch.randn(40, 256).bfloat16()
    w = torch.randn(300, 256).bfloat16()
    full = torch.empty(40, 300, device="cuda")
    ops.gemm_skinny(dev(x), dev(w), full)
    one = torch.empty(1, 300, device="cuda")
    ops.gemm_skinny(dev(x[17:18]), dev(w), one)
    assert torch.equal(one[0], full[17])


@pytest.mark.parametrize("m,i,h", [(5, 96, 64), (64, 8192, 256), (1, 200, 80)])
def test_gemm_skinny_with_the_gate(ops, m, i, h):
    x = torch.randn(m, h).bfloat16()
    wg, wu = (torch.randn(i, h) * 0.2).bfloat16(), (torch.randn(i, h) * 0.2).bfloat16()
    w = ops.interleave_gate_up(dev(wg), dev(wu))
    out = torch.empty(m, i, device="cuda", dtype=torch.bfloat16)
    ops.gemm_skinny(dev(x), w, out, mode="silu")
    ref = torch.nn.functional.silu(x.float() @ wg.float().t()) * (x.float() @ wu.float().t())
    assert float((out.float().cpu() - ref).abs().max()) < 1e-2 * float(ref.abs().max())
    # the library product on the interleaved weight followed by the gate kernel agrees
    gu = (x.float() @ w.float().cpu().t()).bfloat16()
    out2 = torch.empty(m, i, device="cuda", dtype=torch.bfloat16)
    ops.silu_mul(dev(gu), out2, interleaved=True)
    assert float((out2.float().cpu() - ref).abs().max()) < 2e-2 * float(ref.abs().max())


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (128, 128, 128), (200, 384, 2048), (65, 100, 80), (2048, 512, 256), (300, 203, 1000), (1, 16, 8)])
def test_gemm_tcgen05(ops, m, n, k):
    g = torch.Generator().manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g).bfloat16()
    w = (torch.randn(n, k, generator=g) * 0.1).bfloat16()
    ref = x.double() @ w.double().t()
    n_pad = -(-n // 8) * 8  # output rows must be 16-byte aligned
    out = torch.full((m, n_pad), float("nan"), device="cuda", dtype=torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.gemm_tcgen05(dev(x), dev(w), out[:, :n], err=err)
    assert int(err.item()) == 0, "a wait inside the kernel ran out"
    got = out[:, :n].double().cpu()
    assert not torch.isnan(got).any()
    assert float((got - ref).abs().max()) < 1e-2 * float(ref.abs().max())


@pytest.mark.parametrize("m,i,h", [(130, 96, 64), (256, 512, 256), (70, 200, 80)])
def test_gemm_tcgen05_with_the_gate(ops, m, i, h):
    x = torch.randn(m, h).bfloat16()
    wg, wu = (torch.randn(i, h) * 0.2).bfloat16(), (torch.randn(i, h) * 0.2).bfloat16()
    w = ops.interleave_gate_up(dev(wg), dev(wu))
    out = torch.full((m, i), float("nan"), device="cuda", dtype=torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.gemm_tcgen05(dev(x), w, out, mode="silu", err=err)
    assert int(err.item()) == 0
    ref = torch.nn.functional.silu(x.float() @ wg.float().t()) * (x.float() @ wu.float().t())
    assert float((out.float().cpu() - ref).abs().max()) < 1e-2 * float(ref.abs().max())


# (width, slices): one group of threads; two and four groups that share the slices; a width past a CTA's threads
@pytest.mark.parametrize("h,splits", [(100, 3), (2048, 10), (2048, 8), (1024, 9), (512, 16), (3072, 8), (4096, 6), (2048, 5)])
@pytest.mark.parametrize("dtype", DTYPES)
def test_norm_and_rope_sum_the_slices_of_a_split_product(ops, dtype, h, splits):
    n = 6
    resid = torch.randn(n, h)
    parts = torch.randn(splits, n, h)
    w = torch.rand(h) + 0.5
    r = dev(resid)
    out = torch.empty(n, h, device="cuda", dtype=dtype)
    ops.add_rmsnorm(r, ops.Partials(dev(parts)), dev(w), out, 1e-5)
    summed = resid + parts.sum(0)
    assert torch.allclose(r.cpu(), summed, atol=1e-5)
    assert torch.allclose(out.float().cpu(), rms_norm(summed, w, 1e-5), rtol=tol(dtype) * 4, atol=tol(dtype) * 4)
    rows = torch.tensor([5, 5, 0], dtype=torch.int32)
    r2 = dev(resid)
    out2 = torch.empty(3, h, device="cuda", dtype=dtype)
    ops.add_rmsnorm(r2, ops.Partials(dev(parts)), dev(w), out2, 1e-5, rows=dev(rows))
    assert torch.equal(r2.cpu(), resid)
    assert torch.allclose(out2.float().cpu(), rms_norm(summed, w, 1e-5)[rows.long()], rtol=tol(dtype) * 4, atol=tol(dtype) * 4)
    # rotation from slices: the same as from their sum
    nh, nkv, d, bs, nb = 3, 1, 32, 8, 4
    width = (nh + 2 * nkv) * d
    qkv_parts = torch.randn(splits, n, width)
    positions = torch.tensor([0, 1, 7, 8, 100, 4000], dtype=torch.int32)
    slots = torch.tensor([3, 9, 17, 31, 0, 12], dtype=torch.int32)
    inv = plain_inv_freq(d, 10000.0)
    kc1 = torch.zeros(nb, nkv, bs, d, device="cuda", dtype=dtype)
    vc1, kc2, vc2 = torch.zeros_like(kc1), torch.zeros_like(kc1), torch.zeros_like(kc1)
    q1 = torch.empty(n, nh * d, device="cuda", dtype=dtype)
    ops.rope_cache_write(ops.Partials(dev(qkv_parts)), dev(positions), dev(inv), dev(slots), kc1, vc1, nh, nkv, d, bs, q_out=q1)
    whole = dev(qkv_parts.sum(0).to(dtype))
    ops.rope_cache_write(whole, dev(positions), dev(inv), dev(slots), kc2, vc2, nh, nkv, d, bs)
    t = tol(dtype) * 8
    assert torch.allclose(q1.float(), whole[:, : nh * d].float(), rtol=t, atol=t)
    assert torch.allclose(kc1.float(), kc2.float(), rtol=t, atol=t) and torch.allclose(vc1.float(), vc2.float(), rtol=t, atol=t)


# ------------------------------------------------------------------ attention


def paged(kv_per_seq, nkv, d, bs, dtype, seed=0, extra_blocks=5, junk=(1e4, -1e4)):
    """Scatter per-sequence [ctx, nkv, d] keys/values into shuffled pages; stale pages hold junk."""
    rng = random.Random(seed)
    need = [-(-k.shape[0] // bs) for k, _ in kv_per_seq]
    nb = sum(need) + extra_blocks
    order = list(range(nb))
    rng.shuffle(order)
    kc = torch.full((nb, nkv, bs, d), junk[0]).to(dtype)  # junk that would show if it were read
    vc = torch.full((nb, nkv, bs, d), junk[1]).to(dtype)
    width = max(need)
    tables = torch.zeros(len(kv_per_seq), width, dtype=torch.int32)
    for s, (k, v) in enumerate(kv_per_seq):
        for j in range(need[s]):
            blk = order.pop()
            tables[s, j] = blk
            part = slice(j * bs, min((j + 1) * bs, k.shape[0]))
            m = part.stop - part.start
            kc[blk, :, :m] = k[part].transpose(0, 1).to(dtype)
            vc[blk, :, :m] = v[part].transpose(0, 1).to(dtype)
    return kc, vc, tables


def run_attention(ops, dtype, nh, nkv, d, bs, ctx_lens, q_lens, window=0, decode_form=False, seed=0, craft=None, kernel="generic", split=256, junk=(1e4, -1e4), cluster=True, wave_target=0):
    g = torch.Generator().manual_seed(seed)
    kv = [(torch.randn(c, nkv, d, generator=g).to(dtype), torch.randn(c, nkv, d, generator=g).to(dtype)) for c in ctx_lens]
    qs = [torch.randn(ql, nh, d, generator=g).to(dtype) for ql in q_lens]
    if craft:
        craft(kv, qs)
    kc, vc, tables = paged(kv, nkv, d, bs, dtype, seed, junk=junk)
    q = torch.cat(qs, 0).reshape(-1, nh * d)
    qsl = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32)
    out = torch.full((q.shape[0], nh * d), float("nan"), device="cuda", dtype=dtype)
    scale = 1.0 / math.sqrt(d)
    scratch, bound = None, None
    if decode_form:
        bound = max(ctx_lens)
        sa, sm = ops.attention_scratch_shapes(len(ctx_lens), nh, d, bound, split)
        scratch = (torch.full(sa, float("nan"), device="cuda"), torch.full(sm, float("nan"), device="cuda"))
        if decode_form == "fused":  # one launch: the last CTA of a (sequence, kv head) merges
            scratch += (torch.zeros(len(ctx_lens) * nkv, dtype=torch.int32, device="cuda"),)
    for _ in range(2 if decode_form == "fused" else 1):  # the second launch finds the tickets as the first left them
        out.fill_(float("nan"))
        ops.paged_attention(
            dev(q), out, dev(kc), dev(vc), dev(tables), dev(qsl), dev(torch.tensor(ctx_lens, dtype=torch.int32)),
            len(ctx_lens), max(q_lens), nh, nkv, d, scale, window=window, scratch=scratch, max_context=bound,
            split_size=split, kernel=kernel, err=err_flag(), cluster=cluster, wave_target=wave_target,
        )  # fmt: skip
    if decode_form == "fused":
        assert int(scratch[2].abs().sum()) == 0
    refs = []
    for (k, v), qq, c, ql in zip(kv, qs, ctx_lens, q_lens):
        full_q = torch.zeros(c, nh, d, dtype=dtype)
        full_q[c - ql :] = qq
        refs.append(causal_attention(full_q.float(), k.float(), v.float(), scale, window or None)[c - ql :])
    ref = torch.cat(refs, 0).reshape(-1, nh * d)
    return out.float().cpu(), ref, kv


SHAPES = [(4, 2, 16, 16), (3, 1, 32, 8), (6, 3, 48, 4), (8, 2, 64, 16), (5, 5, 80, 32), (32, 1, 128, 16), (2, 2, 256, 16)]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nh,nkv,d,bs", SHAPES)
@pytest.mark.parametrize(
    "ctx_lens,q_lens",
    [([7, 13, 1, 20], [1, 1, 1, 1]), ([9, 16], [9, 16]), ([12, 30, 5], [4, 7, 5]), ([17, 3, 25, 130], [1, 3, 5, 67])],
)
def test_paged_attention_generic(ops, dtype, nh, nkv, d, bs, ctx_lens, q_lens):
    out, ref, _ = run_attention(ops, dtype, nh, nkv, d, bs, ctx_lens, q_lens)
    t = 1e-5 if dtype == torch.float32 else 2e-2
    assert not torch.isnan(out).any()
    assert torch.allclose(out, ref, rtol=t, atol=t)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nh,nkv,d,bs", [(4, 2, 16, 16), (6, 3, 48, 4), (8, 2, 64, 16), (24, 1, 32, 8)])
def test_paged_attention_decode_form(ops, dtype, nh, nkv, d, bs):
    ctx = [700, 1, 256, 257, 33]
    out, ref, _ = run_attention(ops, dtype, nh, nkv, d, bs, ctx, [1] * 5, decode_form=True)
    t = 1e-5 if dtype == torch.float32 else 2e-2
    assert not torch.isnan(out).any()
    assert torch.allclose(out, ref, rtol=t, atol=t)


@pytest.mark.parametrize("decode_form", [False, True])
def test_attention_finds_a_far_key_among_hundreds(ops, decode_form):
    """Random scores are near uniform and would hide a key that is skipped: one far key is
    made to take all the weight, at a page's first and last place and across a range edge."""
    for far in (0, 15, 16, 255, 256, 511, 640):

        def craft(kv, qs, far=far):
            k, v = kv[0]
            k.mul_(0.01)
            k[far, :, 0] = 40.0
            qs[0][-1, :, 0] = 40.0

        out, ref, kv = run_attention(ops, torch.float32, 4, 2, 32, 16, [700], [1], decode_form=decode_form, craft=craft)
        v_far = kv[0][1][far].float().repeat_interleave(2, dim=0).reshape(-1)
        assert torch.allclose(out[-1], v_far, atol=1e-3), far
        assert torch.allclose(out, ref, atol=1e-5), far


@pytest.mark.parametrize("decode_form", [False, True])
@pytest.mark.parametrize("window", [1, 5, 32, 33, 100])
def test_attention_window_edge(ops, window, decode_form):
    """The key just inside the window is seen, the one just outside is not."""
    ctx = 300
    for offset, seen in ((window - 1, True), (window, False)):
        far = ctx - 1 - offset

        def craft(kv, qs, far=far):
            k, v = kv[0]
            k.mul_(0.01)
            k[far, :, 0] = 40.0
            qs[0][-1, :, 0] = 40.0

        q_lens = [1] if decode_form else [9]
        out, ref, kv = run_attention(ops, torch.float32, 2, 1, 16, 8, [ctx], q_lens, window=window, decode_form=decode_form, craft=craft)
        assert torch.allclose(out, ref, atol=1e-5), (window, offset)
        v_far = kv[0][1][far].float().repeat(2, 1).reshape(-1)
        assert torch.allclose(out[-1], v_far, atol=1e-3) == seen, (window, offset)


def test_attention_rows_do_not_depend_on_the_cut(ops):
    """A query's output is bit-identical whether it comes alone, in a portion, or in the whole prompt."""
    nh, nkv, d, bs, ctx = 6, 3, 48, 4, 97
    whole, _, _ = run_attention(ops, torch.float32, nh, nkv, d, bs, [ctx], [ctx], seed=4)
    # same seed -> same keys and values; the queries are drawn after them, so rebuild the tail from `whole`'s inputs
    g = torch.Generator().manual_seed(4)
    k = torch.randn(ctx, nkv, d, generator=g)
    v = torch.randn(ctx, nkv, d, generator=g)
    q = torch.randn(ctx, nh, d, generator=g)
    for ql in (1, 2, 30):
        kc, vc, tables = paged([(k, v)], nkv, d, bs, torch.float32, seed=ql)
        out = torch.empty(ql, nh * d, device="cuda")
        ops.paged_attention_generic(
            dev(q[ctx - ql :].reshape(ql, -1)), out, dev(kc), dev(vc), dev(tables), dev(torch.tensor([0, ql], dtype=torch.int32)),
            dev(torch.tensor([ctx], dtype=torch.int32)), 1, ql, nh, nkv, d, 1.0 / math.sqrt(d),
        )  # fmt: skip
        assert torch.equal(out.cpu(), whole[ctx - ql :]), ql


# ---- the tensor-core kernel (bfloat16, head sizes 64 and 128)

MMA_SHAPES = [(8, 2, 64, 16), (32, 8, 64, 16), (3, 1, 64, 8), (6, 3, 128, 4), (24, 8, 128, 32), (5, 5, 64, 16), (14, 2, 128, 16), (32, 1, 64, 16)]


@pytest.mark.parametrize("nh,nkv,d,bs", MMA_SHAPES)
@pytest.mark.parametrize(
    "ctx_lens,q_lens",
    [([7, 13, 1, 20], [1, 1, 1, 1]), ([9, 16], [9, 16]), ([12, 30, 5], [4, 7, 5]), ([17, 3, 25, 130], [1, 3, 5, 67]), ([300, 64, 65], [300, 2, 65])],
)
def test_paged_attention_mma(ops, nh, nkv, d, bs, ctx_lens, q_lens):
    out, ref, _ = run_attention(ops, torch.bfloat16, nh, nkv, d, bs, ctx_lens, q_lens, kernel="mma")
    assert not torch.isnan(out).any()
    assert torch.allclose(out, ref, rtol=2e-2, atol=2e-2)


# ---- the tcgen05 kernel (bfloat16, head size 64, many queries)

TC_SHAPES = MMA_SHAPES + [(4, 4, 64, 16), (16, 1, 64, 32), (4, 4, 128, 16), (8, 1, 128, 48), (8, 2, 64, 64), (8, 2, 128, 64), (4, 2, 64, 128)]


@pytest.mark.parametrize("nh,nkv,d,bs", TC_SHAPES)
@pytest.mark.parametrize(
    "ctx_lens,q_lens",
    [([9, 16], [9, 16]), ([12, 30, 5], [4, 7, 5]), ([17, 3, 25, 130], [1, 3, 5, 67]), ([300, 64, 65], [300, 2, 65]), ([700, 129], [450, 128])],
)
def test_paged_attention_tcgen05(ops, nh, nkv, d, bs, ctx_lens, q_lens):
    # whatever lies past a context inside its last page must not reach the result
    out, ref, _ = run_attention(ops, torch.bfloat16, nh, nkv, d, bs, ctx_lens, q_lens, kernel="tcgen05", junk=(float("nan"), float("nan")))
    assert not torch.isnan(out).any()
    assert torch.allclose(out, ref, rtol=2e-2, atol=2e-2)


def test_paged_attention_tcgen05_takes_its_tiles_from_a_list(ops):
    # the same batch with the grid spanning sequences x tiles, and with a shuffled list of
    # (sequence, first query) tiles that has dead entries in it
    nh, nkv, d, bs = 8, 2, 64, 16
    ctx_lens, q_lens = [300, 64, 65, 130], [300, 2, 65, 1]
    torch.manual_seed(5)
    dev = "cuda"
    kv = [(torch.randn(c, nkv, d).bfloat16(), torch.randn(c, nkv, d).bfloat16()) for c in ctx_lens]
    kc, vc, bt = (t.to(dev) for t in paged(kv, nkv, d, bs, torch.bfloat16))
    q = torch.cat([torch.randn(n, nh, d).bfloat16() for n in q_lens]).reshape(-1, nh * d).contiguous().to(dev)
    qsl = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32).to(dev)
    cl = torch.tensor(ctx_lens, dtype=torch.int32).to(dev)
    outs = []
    tq = ops.tcgen05_query_tile(nh, nkv)
    pairs = [(b, j * tq) for b, n in enumerate(q_lens) for j in range(-(-n // tq))]
    g = torch.Generator().manual_seed(1)
    pairs = [pairs[i] for i in torch.randperm(len(pairs), generator=g).tolist()]
    listed = pairs[:3] + [(-1, 0)] + pairs[3:] + [(-1, 0), (-1, 0)]
    tiles = torch.tensor(listed, device=dev, dtype=torch.int32).reshape(-1).contiguous()
    for query_tiles in (None, (tiles, len(listed))):
        out = torch.full_like(q, float("nan"))
        err = err_flag()
        ops.paged_attention(q, out, kc, vc, bt, qsl, cl, len(q_lens), max(q_lens), nh, nkv, d, d**-0.5, kernel="tcgen05", err=err, query_tiles=query_tiles)
        assert int(err.sum()) == 0
        outs.append(out)
    assert not torch.isnan(outs[1]).any()
    assert torch.equal(outs[0], outs[1])


def test_tcgen05_attention_finds_a_far_key_and_respects_the_window(ops):
    for far in (0, 15, 16, 127, 128, 255, 256, 511, 640):

        def craft(kv, qs, far=far):
            k, v = kv[0]
            k.mul_(0.01)
            k[far, :, 0] = 40.0
            qs[0][-1, :, 0] = 40.0

        out, ref, kv = run_attention(ops, torch.bfloat16, 8, 2, 64, 16, [700], [5], craft=craft, kernel="tcgen05")
        v_far = kv[0][1][far].float().repeat_interleave(4, dim=0).reshape(-1)
        assert torch.allclose(out[-1], v_far, atol=2e-2), far
    ctx = 300
    for window in (1, 5, 128, 129, 200):
        for offset, seen in ((window - 1, True), (window, False)):
            far = ctx - 1 - offset

            def craft(kv, qs, far=far):
                k, v = kv[0]
                k.mul_(0.01)
                k[far, :, 0] = 40.0
                qs[0][-1, :, 0] = 40.0

            out, ref, kv = run_attention(ops, torch.bfloat16, 4, 1, 64, 8, [ctx], [9], window=window, craft=craft, kernel="tcgen05")
            assert torch.allclose(out, ref, rtol=2e-2, atol=2e-2), (window, offset)
            v_far = kv[0][1][far].float().repeat(4, 1).reshape(-1)
            assert torch.allclose(out[-1], v_far, atol=2e-2) == seen, (window, offset)


def test_tcgen05_attention_rows_do_not_depend_on_the_cut(ops):
    nh, nkv, d, bs, ctx = 8, 2, 64, 16, 297
    whole, _, _ = run_attention(ops, torch.bfloat16, nh, nkv, d, bs, [ctx], [ctx], seed=4, kernel="tcgen05")
    g = torch.Generator().manual_seed(4)
    k = torch.randn(ctx, nkv, d, generator=g).bfloat16()
    v = torch.randn(ctx, nkv, d, generator=g).bfloat16()
    q = torch.randn(ctx, nh, d, generator=g).bfloat16()
    for ql in (2, 30, 170):
        kc, vc, tables = paged([(k, v)], nkv, d, bs, torch.bfloat16, seed=ql)
        out = torch.empty(ql, nh * d, device="cuda", dtype=torch.bfloat16)
        ops.paged_attention(
            dev(q[ctx - ql :].reshape(ql, -1)), out, dev(kc), dev(vc), dev(tables), dev(torch.tensor([0, ql], dtype=torch.int32)),
            dev(torch.tensor([ctx], dtype=torch.int32)), 1, ql, nh, nkv, d, 1.0 / math.sqrt(d), kernel="tcgen05",
        )  # fmt: skip
        assert torch.equal(out.float().cpu(), whole[ctx - ql :]), ql


@pytest.mark.parametrize("nh,nkv,d,bs", [s for s in MMA_SHAPES if s[0] // s[1] <= 16])
@pytest.mark.parametrize("split", [64, 128, 256])
@pytest.mark.parametrize("form", [True, "fused"])
def test_paged_attention_mma_decode_form(ops, nh, nkv, d, bs, split, form):
    ctx = [700, 1, 256, 257, 33, 64, 65]
    out, ref, _ = run_attention(ops, torch.bfloat16, nh, nkv, d, bs, ctx, [1] * len(ctx), decode_form=form, kernel="mma", split=split)
    assert not torch.isnan(out).any()
    assert torch.allclose(out, ref, rtol=2e-2, atol=2e-2)


# ---- the TMA decode kernel (bfloat16, head size 64 or 128, up to 8 heads per kv head, pages of 16 n tokens)

TMA_SHAPES = [(8, 2, 64, 16), (32, 8, 64, 16), (3, 1, 64, 32), (24, 8, 128, 32), (5, 5, 64, 48), (14, 2, 128, 16), (8, 1, 64, 16)]


@pytest.mark.parametrize("nh,nkv,d,bs", TMA_SHAPES)
@pytest.mark.parametrize("split", [64, 128, 256, 1024])
@pytest.mark.parametrize("cluster", [True, False])  # the ranges merged through a cluster's shared memory (up to 16), or by ticket
def test_paged_attention_tma_decode(ops, nh, nkv, d, bs, split, cluster):
    ctx = [700, 1, 256, 257, 33, 64, 65, 1500, 16, 17]
    err_flag().zero_()
    # what lies past a context inside its last page must not reach the result, whatever it is
    out, ref, _ = run_attention(ops, torch.bfloat16, nh, nkv, d, bs, ctx, [1] * len(ctx), decode_form="fused", kernel="tma", split=split, junk=(float("nan"), float("nan")), cluster=cluster)
    assert int(err_flag().sum()) == 0
    assert not torch.isnan(out).any()
    assert torch.allclose(out, ref, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("target", [1, 7, 12, 40, 10000])
@pytest.mark.parametrize("cluster", [False, True])
def test_tma_decode_lengthens_its_ranges_to_the_wave_it_is_given(ops, target, cluster):
    """With a target number of CTAs the kernel doubles the range size from the batch's longest
    context (1,500 keys, 4 pairs: ranges of 64 would be 96 CTAs): whatever size comes out, every
    sequence's result is the plain one, also those whose contexts end inside a lengthened range,
    and a window still cuts where it should."""
    ctx = [700, 1, 256, 257, 33, 64, 65, 1500, 16, 17]
    err_flag().zero_()
    for window in (0, 90):
        out, ref, _ = run_attention(ops, torch.bfloat16, 8, 2, 64, 16, ctx, [1] * len(ctx), decode_form="fused", kernel="tma", split=64,
                                    window=window, junk=(float("nan"), float("nan")), cluster=cluster, wave_target=target)  # fmt: skip
        assert int(err_flag().sum()) == 0
        assert not torch.isnan(out).any()
        assert torch.allclose(out, ref, rtol=2e-2, atol=2e-2), (target, window)


def test_tma_decode_finds_a_far_key_and_respects_the_window(ops):
    err_flag().zero_()
    for far in (0, 15, 16, 63, 64, 255, 256, 511, 640, 699):

        def craft(kv, qs, far=far):
            k, v = kv[0]
            k.mul_(0.01)
            k[far, :, 0] = 40.0
            qs[0][-1, :, 0] = 40.0

        out, ref, kv = run_attention(ops, torch.bfloat16, 8, 2, 64, 16, [700], [1], decode_form="fused", craft=craft, kernel="tma", split=128)
        v_far = kv[0][1][far].float().repeat_interleave(4, dim=0).reshape(-1)
        assert torch.allclose(out[-1], v_far, atol=2e-2), far
    ctx = 300
    for window in (1, 5, 16, 17, 64, 65, 100):
        for offset, seen in ((window - 1, True), (window, False)):
            far = ctx - 1 - offset

            def craft(kv, qs, far=far):
                k, v = kv[0]
                k.mul_(0.01)
                k[far, :, 0] = 40.0
                qs[0][-1, :, 0] = 40.0

            out, ref, kv = run_attention(ops, torch.bfloat16, 4, 1, 64, 16, [ctx], [1], window=window, decode_form="fused", craft=craft, kernel="tma", split=64)
            assert torch.allclose(out, ref, rtol=2e-2, atol=2e-2), (window, offset)
            v_far = kv[0][1][far].float().repeat(4, 1).reshape(-1)
            assert torch.allclose(out[-1], v_far, atol=2e-2) == seen, (window, offset)
    assert int(err_flag().sum()) == 0


@pytest.mark.parametrize("nh,nkv,d,bs", [(8, 2, 64, 16), (24, 8, 128, 32)])
def test_mixed_batch_split_between_the_decode_kernel_and_the_kernel_of_prompts(ops, nh, nkv, d, bs):
    """Of a mixed batch the decode kernel computes the sequences that bring one token and leaves
    the rows of the others alone; the kernel of prompts, given the tiles of the others, fills those."""
    ctx_lens, q_lens = [300, 130, 64, 700, 5, 257], [1, 67, 1, 300, 5, 1]
    g = torch.Generator().manual_seed(11)
    kv = [(torch.randn(c, nkv, d, generator=g).bfloat16(), torch.randn(c, nkv, d, generator=g).bfloat16()) for c in ctx_lens]
    qs = [torch.randn(n, nh, d, generator=g).bfloat16() for n in q_lens]
    kc, vc, tables = paged(kv, nkv, d, bs, torch.bfloat16, seed=2, junk=(float("nan"), float("nan")))
    q = dev(torch.cat(qs, 0).reshape(-1, nh * d))
    starts = [0] + list(torch.tensor(q_lens).cumsum(0))
    qsl, cl = dev(torch.tensor(starts, dtype=torch.int32)), dev(torch.tensor(ctx_lens, dtype=torch.int32))
    out = torch.full((q.shape[0], nh * d), float("nan"), device="cuda", dtype=torch.bfloat16)
    scale, split, nseq = 1.0 / math.sqrt(d), 128, len(ctx_lens)
    sa, sm = ops.attention_scratch_shapes(nseq, nh, d, max(ctx_lens), split)
    scratch = (torch.empty(sa, device="cuda"), torch.empty(sm, device="cuda"), torch.zeros(nseq * nkv, dtype=torch.int32, device="cuda"))
    err_flag().zero_()
    common = (q, out, dev(kc), dev(vc), dev(tables), qsl, cl, nseq)
    ops.paged_attention(*common, 1, nh, nkv, d, scale, scratch=scratch, max_context=max(ctx_lens), split_size=split, kernel="tma", err=err_flag(), cluster=False, single_only=True)
    single = [b for b, n in enumerate(q_lens) if n == 1]
    rows_single = [int(starts[b]) for b in single]
    rows_multi = [r for b, n in enumerate(q_lens) if n > 1 for r in range(int(starts[b]), int(starts[b + 1]))]
    assert not torch.isnan(out[rows_single]).any()
    assert torch.isnan(out[rows_multi]).all()
    assert int(scratch[2].abs().sum()) == 0
    tq = ops.tcgen05_query_tile(nh, nkv)
    pairs = [(b, j * tq) for b, n in enumerate(q_lens) if n > 1 for j in range(-(-n // tq))] + [(-1, 0)]
    tiles = dev(torch.tensor(pairs, dtype=torch.int32).reshape(-1))
    before = out[rows_single].clone()
    ops.paged_attention(*common, max(q_lens), nh, nkv, d, scale, kernel="tcgen05", err=err_flag(), query_tiles=(tiles, len(pairs)))
    assert torch.equal(out[rows_single], before)
    assert int(err_flag().sum()) == 0
    refs = []
    for (k, v), qq, c, ql in zip(kv, qs, ctx_lens, q_lens):
        full_q = torch.zeros(c, nh, d)
        full_q[c - ql :] = qq.float()
        refs.append(causal_attention(full_q, k.float(), v.float(), scale, None)[c - ql :])
    ref = torch.cat(refs, 0).reshape(-1, nh * d)
    assert torch.allclose(out.float().cpu(), ref, rtol=2e-2, atol=2e-2)


def test_tma_decode_reads_zeros_for_pages_that_were_given_back(ops):
    """A table entry of -1 (a page the window has passed) is read as zeros, not as page -1."""
    nh, nkv, d, bs, ctx, window = 8, 2, 64, 16, 200, 40
    g = torch.Generator().manual_seed(3)
    k = torch.randn(ctx, nkv, d, generator=g).bfloat16()
    v = torch.randn(ctx, nkv, d, generator=g).bfloat16()
    q = torch.randn(1, nh, d, generator=g).bfloat16()
    kc, vc, tables = paged([(k, v)], nkv, d, bs, torch.bfloat16, seed=1)
    tables[0, : (ctx - window) // bs] = -1
    out = torch.empty(1, nh * d, device="cuda", dtype=torch.bfloat16)
    sa, sm = ops.attention_scratch_shapes(1, nh, d, ctx, 64)
    scratch = (torch.empty(sa, device="cuda"), torch.empty(sm, device="cuda"), torch.zeros(nkv, dtype=torch.int32, device="cuda"))
    err_flag().zero_()
    ops.paged_attention(
        dev(q.reshape(1, -1)), out, dev(kc), dev(vc), dev(tables), dev(torch.tensor([0, 1], dtype=torch.int32)),
        dev(torch.tensor([ctx], dtype=torch.int32)), 1, 1, nh, nkv, d, 1.0 / math.sqrt(d), window=window, scratch=scratch,
        max_context=ctx, split_size=64, kernel="tma", err=err_flag(),
    )  # fmt: skip
    full_q = torch.zeros(ctx, nh, d)
    full_q[-1] = q[0].float()
    ref = causal_attention(full_q, k.float(), v.float(), 1.0 / math.sqrt(d), window)[-1].reshape(-1)
    assert int(err_flag().sum()) == 0
    assert torch.allclose(out[0].float().cpu(), ref, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("decode_form", [False, True, "fused"])
def test_mma_attention_finds_a_far_key_and_respects_the_window(ops, decode_form):
    for far in (0, 15, 16, 63, 64, 255, 256, 511, 640):

        def craft(kv, qs, far=far):
            k, v = kv[0]
            k.mul_(0.01)
            k[far, :, 0] = 40.0
            qs[0][-1, :, 0] = 40.0

        out, ref, kv = run_attention(ops, torch.bfloat16, 8, 2, 64, 16, [700], [1], decode_form=decode_form, craft=craft, kernel="mma", split=128)
        v_far = kv[0][1][far].float().repeat_interleave(4, dim=0).reshape(-1)
        assert torch.allclose(out[-1], v_far, atol=2e-2), far
    ctx = 300
    for window in (1, 5, 64, 65, 100):
        for offset, seen in ((window - 1, True), (window, False)):
            far = ctx - 1 - offset

            def craft(kv, qs, far=far):
                k, v = kv[0]
                k.mul_(0.01)
                k[far, :, 0] = 40.0
                qs[0][-1, :, 0] = 40.0

            q_lens = [1] if decode_form else [9]
            out, ref, kv = run_attention(ops, torch.bfloat16, 4, 1, 64, 8, [ctx], q_lens, window=window, decode_form=decode_form, craft=craft, kernel="mma", split=64)
            assert torch.allclose(out, ref, rtol=2e-2, atol=2e-2), (window, offset)
            v_far = kv[0][1][far].float().repeat(4, 1).reshape(-1)
            assert torch.allclose(out[-1], v_far, atol=2e-2) == seen, (window, offset)


def test_mma_attention_rows_do_not_depend_on_the_cut(ops):
    nh, nkv, d, bs, ctx = 8, 2, 64, 16, 197
    whole, _, _ = run_attention(ops, torch.bfloat16, nh, nkv, d, bs, [ctx], [ctx], seed=4, kernel="mma")
    g = torch.Generator().manual_seed(4)
    k = torch.randn(ctx, nkv, d, generator=g).bfloat16()
    v = torch.randn(ctx, nkv, d, generator=g).bfloat16()
    q = torch.randn(ctx, nh, d, generator=g).bfloat16()
    for ql in (2, 30, 70):
        kc, vc, tables = paged([(k, v)], nkv, d, bs, torch.bfloat16, seed=ql)
        out = torch.empty(ql, nh * d, device="cuda", dtype=torch.bfloat16)
        ops.paged_attention(
            dev(q[ctx - ql :].reshape(ql, -1)), out, dev(kc), dev(vc), dev(tables), dev(torch.tensor([0, ql], dtype=torch.int32)),
            dev(torch.tensor([ctx], dtype=torch.int32)), 1, ql, nh, nkv, d, 1.0 / math.sqrt(d), kernel="mma",
        )  # fmt: skip
        assert torch.equal(out.float().cpu(), whole[ctx - ql :]), ql


def test_head_dim_is_checked(ops):
    ops.check_head_dim(40)  # the FP32-pipe kernels take heads in steps of 8
    with pytest.raises(ValueError, match="head_dim"):
        ops.check_head_dim(44)
    with pytest.raises(ValueError, match="head_dim"):
        ops.check_head_dim(512)


@pytest.mark.parametrize("m,n,k", [(17, 2048, 2048), (64, 2048, 8192), (100, 3072, 3072), (128, 512, 4096)])
def test_library_product_over_slices_of_k(ops, m, n, k):
    """The batched library product that serves a few dozen tokens: its float slices sum to x W^T."""
    g = torch.Generator().manual_seed(m + n)
    x = (torch.randn(m, k, generator=g) * 0.5).bfloat16()
    w = (torch.randn(n, k, generator=g) * 0.05).bfloat16()
    splits = ops.library_splits(m, n, k)
    assert splits in (2, 4) and ops.library_splits(8, n, k) == 1 and ops.library_splits(m, 4 * k, k) == 1
    part = ops.Partials(torch.full((splits, m, n), float("nan"), device="cuda"))
    ops.linear_split_k(dev(x), dev(w), part)
    got = part.t.sum(0).cpu().double()
    want = x.double() @ w.double().t()
    assert float((got - want).abs().max()) < 1e-5 * float(want.abs().max())
    with pytest.raises(ValueError):
        ops.linear_split_k(dev(x), dev(w), ops.Partials(torch.empty(5, m, n, device="cuda")))


# ------------------------------------------------------------------ sampling


def test_greedy_is_argmax_with_lowest_index_on_ties(ops):
    logits = torch.randn(6, 1003)
    logits[2, 77] = logits[2, 500] = 9.0
    out = torch.empty(6, dtype=torch.int32, device="cuda")
    ops.sample(dev(logits), out)
    want = logits.argmax(-1)
    want[2] = 77
    assert out.cpu().tolist() == want.tolist()


@pytest.mark.parametrize("v", [5, 320, 1003, 128256])
def test_batched_argmax(ops, v):
    logits = torch.randn(9, v + 3)[:, :v]  # a row stride that is not the width
    if v > 100:
        logits[2, 77] = logits[2, v - 1] = 9.0
        logits[5, 0] = 11.0
    out = torch.empty(9, dtype=torch.int32, device="cuda")
    scratch = torch.empty(9 * ops.ARGMAX_CHUNKS, dtype=torch.int64, device="cuda")
    dl = torch.empty(9, v + 3, device="cuda")[:, :v]
    dl.copy_(logits)
    ops.argmax(dl, out, scratch)
    want = logits.argmax(-1)
    if v > 100:
        want[2] = 77
    assert out.cpu().tolist() == want.tolist()


@pytest.mark.parametrize("v", [5, 320, 1003, 128256])
def test_sampling_distribution_matches_the_formula(ops, v):
    g = torch.Generator().manual_seed(v)
    logits = torch.randn(8, v, generator=g) * 3
    cases = [(1.0, 0, 1.0), (0.8, 0, 1.0), (1.0, 3, 1.0), (1.0, 0, 0.9), (0.7, 50, 0.5), (2.0, 1, 1.0), (0.0, 0, 1.0), (1.3, 0, 0.01)]
    temps = torch.tensor([c[0] for c in cases])
    ks = torch.tensor([c[1] for c in cases], dtype=torch.int32)
    ps = torch.tensor([c[2] for c in cases])
    keys = torch.arange(8, dtype=torch.int64) + 12345
    out = torch.empty(8, dtype=torch.int32, device="cuda")
    probs = torch.empty(8, v, device="cuda")
    ops.sample(dev(logits), out, dev(temps), dev(ks), dev(ps), dev(keys), probs)
    probs = probs.cpu()
    for i, (t, k, p) in enumerate(cases):
        # The formula in float64: over 128k entries a float32 running sum moves the top-p cut
        # by a few entries.  What may differ from exact arithmetic: entries whose mass is
        # below the 2^-40 fixed point, and entries that sit exactly on the cut.
        ref = processed_probs(logits[i].double(), t, k, p)
        differ = (probs[i] > 0) != (ref > 0)
        assert float(ref[differ].sum()) + float(probs[i][differ].sum()) < 1e-5, (i, int(differ.sum()))
        assert torch.allclose(probs[i].double()[~differ], ref[~differ], atol=2e-6, rtol=1e-4), i
        ref = ref.float()
        # the draw is the inverse CDF in index order at u = splitmix64(key) / 2^64
        u = ops.splitmix64(int(keys[i])) / 2.0**64
        cdf = ref.double().cumsum(0)
        want = int(torch.searchsorted(cdf, torch.tensor(u * float(cdf[-1]), dtype=torch.float64), right=True))
        tok = int(out[i])
        assert ref[tok] > 0
        if tok != want:  # only a draw that lands within rounding of a CDF step may differ
            lo = float(cdf[tok - 1]) if tok > 0 else 0.0
            assert min(abs(u - lo), abs(u - float(cdf[tok]))) < 1e-5, (i, tok, want)


def test_top_p_on_flat_rows_takes_the_cut_from_one_bucket(ops):
    """Top-p alone on rows with hundreds or thousands of entries over the cut: too many to gather, so
    the cut is looked for among the entries of the one coarse bucket it falls into (or, when that
    bucket is crowded too, or is the catch-all lowest one, by the radix passes).  The distribution
    and the draw are those of the formula whichever way was taken."""
    v = 128256
    g = torch.Generator().manual_seed(17)
    noise = torch.randn(v, generator=g)
    rows = [
        (noise * 3, 0.8, 0.9), (noise * 3, 1.0, 0.5), (noise * 3, 2.0, 0.99), (noise * 3, 0.5, 0.3),
        (noise * 0.05, 1.0, 0.9),       # all within an eighth of a nat: one crowded bucket
        (noise * 3, 1.0, 0.9999999),    # nearly everything stays: the cut lies far below the maximum
        (noise * 12, 1.0, 0.999999),    # ... in the lowest bucket, which holds all that is 32 nats down
        ((noise * 3).round(), 1.0, 0.9),  # many equal values: ties stay or go together
    ]  # fmt: skip
    logits = torch.stack([r[0] for r in rows])
    temps = torch.tensor([r[1] for r in rows])
    ps = torch.tensor([r[2] for r in rows])
    keys = torch.arange(len(rows), dtype=torch.int64) + 4242
    out = torch.empty(len(rows), dtype=torch.int32, device="cuda")
    probs = torch.empty(len(rows), v, device="cuda")
    ops.sample(dev(logits), out, dev(temps), None, dev(ps), dev(keys), probs)
    probs = probs.cpu().double()
    for i, (row, t, p) in enumerate(rows):
        ref = tie_keeping_probs(row, t, 0, p)
        differ = (probs[i] > 0) != (ref > 0)
        assert float(ref[differ].sum()) + float(probs[i][differ].sum()) < 1e-5, (i, int(differ.sum()))
        assert torch.allclose(probs[i][~differ], ref[~differ], atol=2e-6, rtol=1e-4), i
        u = ops.splitmix64(int(keys[i])) / 2.0**64
        cdf = ref.cumsum(0)
        want = int(torch.searchsorted(cdf, torch.tensor(u * float(cdf[-1]), dtype=torch.float64), right=True))
        tok = int(out[i])
        assert ref[tok] > 0
        if tok != want:  # only a draw that lands within rounding of a CDF step may differ
            lo = float(cdf[tok - 1]) if tok > 0 else 0.0
            assert min(abs(u - lo), abs(u - float(cdf[tok]))) < 1e-5, (i, tok, want)
    # and without the probabilities written out the same tokens are drawn
    out2 = torch.empty_like(out)
    ops.sample(dev(logits), out2, dev(temps), None, dev(ps), dev(keys))
    assert torch.equal(out, out2)


def tie_keeping_probs(logits, t, k, p):
    """What the sampling kernel defines: values tied with the k-th largest all stay, and top-p
    treats equal values as one block (it stays if the mass of the strictly larger values is
    below top_p of the mass that top-k kept).  float64."""
    x = logits.double() / t
    v = x.numel()
    kept = torch.ones(v, dtype=torch.bool)
    if 0 < k < v:
        kept = x >= x.sort(descending=True).values[k - 1]
    m = torch.exp(x - x.max()) * kept
    if p < 1.0:
        vals, inv = torch.unique(x, return_inverse=True)  # ascending
        per = torch.zeros_like(vals).index_add_(0, inv, m)
        above = per.flip(0).cumsum(0).flip(0) - per  # mass of the strictly larger values
        m = m * (above < p * m.sum())[inv]
    return m / m.sum()


def test_sampling_with_few_and_with_many_entries_left_by_top_k(ops):
    """Top-k up to 256 finishes in one CTA's shared memory on the entries that passed; more
    entries than that (a larger k, values tied with the k-th largest, a flat row under top-p
    alone) take the passes over the row.  Both must give the same distribution and the same draw."""
    v = 5000
    g = torch.Generator().manual_seed(3)
    base = torch.randn(v, generator=g) * 2
    tied = base.clone()
    tied[torch.randperm(v, generator=g)[:400]] = 7.0  # 400 values tied at the top
    edge = base.clone()
    order = edge.argsort(descending=True)
    edge[order[199:201]] = float(edge[order[199]])  # the 200th and the 201st largest are equal
    many_edge = base.clone()
    many_edge[order[511:514]] = float(many_edge[order[511]])  # 512th..514th equal: 514 entries pass k = 512
    cases = [(base, 1.0, 512, 0.9), (base, 0.7, 600, 0.8), (tied, 1.0, 10, 0.9), (edge, 1.3, 200, 0.5), (many_edge, 1.0, 512, 0.95),
             (base, 1.0, 1, 0.5), (base, 0.9, 40, 1.0), (tied, 0.8, 500, 0.3), (base, 0.5, 0, 0.9), (base, 0.3, 0, 0.5), (tied, 0.6, 0, 0.7),
             (edge * 3, 1.0, 0, 0.99)]  # fmt: skip
    logits = torch.stack([c[0] for c in cases])
    temps = torch.tensor([c[1] for c in cases])
    ks = torch.tensor([c[2] for c in cases], dtype=torch.int32)
    ps = torch.tensor([c[3] for c in cases])
    keys = torch.arange(len(cases), dtype=torch.int64) + 99
    out = torch.empty(len(cases), dtype=torch.int32, device="cuda")
    probs = torch.empty(len(cases), v, device="cuda")
    ops.sample(dev(logits), out, dev(temps), dev(ks), dev(ps), dev(keys), probs)
    probs = probs.cpu().double()
    for i, (row, t, k, p) in enumerate(cases):
        ref = tie_keeping_probs(row, t, k, p)
        differ = (probs[i] > 0) != (ref > 0)
        assert float(ref[differ].sum()) + float(probs[i][differ].sum()) < 1e-5, (i, int(differ.sum()))
        assert torch.allclose(probs[i][~differ], ref[~differ], atol=2e-6, rtol=1e-4), i
        u = ops.splitmix64(int(keys[i])) / 2.0**64
        cdf = ref.cumsum(0)
        want = int(torch.searchsorted(cdf, torch.tensor(u * float(cdf[-1]), dtype=torch.float64), right=True))
        tok = int(out[i])
        assert ref[tok] > 0
        if tok != want:  # only a draw that lands within rounding of a CDF step may differ
            lo = float(cdf[tok - 1]) if tok > 0 else 0.0
            assert min(abs(u - lo), abs(u - float(cdf[tok]))) < 1e-5, (i, tok, want)


def test_sampling_is_reproducible_and_follows_the_distribution(ops):
    logits = torch.tensor([[2.0, 1.0, 0.5, -1.0, 0.0]]).repeat(4000, 1)
    temps = torch.full((4000,), 0.8)
    keys = torch.arange(4000, dtype=torch.int64) * 7919
    out1 = torch.empty(4000, dtype=torch.int32, device="cuda")
    out2 = torch.empty(4000, dtype=torch.int32, device="cuda")
    ops.sample(dev(logits), out1, dev(temps), None, None, dev(keys))
    ops.sample(dev(logits), out2, dev(temps), None, None, dev(keys))
    assert torch.equal(out1, out2)
    freq = torch.bincount(out1.cpu().long(), minlength=5).double() / 4000
    ref = torch.softmax(logits[0].double() / 0.8, -1)
    assert float((freq - ref).abs().max()) < 0.03


# ------------------------------------------------------------------ attention over one row a token, many queries


def paged_latent_case(lens, starts, nh, d, dv, block_size, window, seed, sharp=1.0):
    """Queries, a cache on shuffled pages with NaN wherever no key lies, tables, and the 64-bit result with the bound on
    what rounding the weights (relative 2^-9 each) and the result (2^-9) to bfloat16 may change, times two."""
    g = torch.Generator().manual_seed(seed)
    ctx = [n + s for n, s in zip(lens, starts)]
    per = [-(-c // block_size) for c in ctx]
    order = torch.randperm(sum(per) + 3, generator=g).tolist()
    cache = torch.full((sum(per) + 3, 1, block_size, d), float("nan"))
    tables = torch.zeros((len(lens), max(per)), dtype=torch.int32)
    q = (sharp * torch.randn((sum(lens), nh * d), generator=g)).bfloat16()
    outs, bounds, at, row = [], [], 0, 0
    for b, (n, c) in enumerate(zip(lens, ctx)):
        keys = torch.randn((c, d), generator=g).bfloat16()
        pages = order[at : at + per[b]]
        at += per[b]
        for j in range(c):
            cache[pages[j // block_size], 0, j % block_size] = keys[j].float()
        gone = max(0, c - n - window + 1) // block_size if window else 0  # pages that no query of the step sees come back
        tables[b, : per[b]] = torch.tensor([-1] * gone + pages[gone:], dtype=torch.int32)
        k = keys.double()
        qs = q[row : row + n].double().view(n, nh, d)
        row += n
        i, j = torch.arange(c - n, c)[:, None], torch.arange(c)[None]
        seen = (j <= i) & ((i - j < window) if window else True)
        w = torch.softmax((torch.einsum("nhd,jd->hnj", qs, k) * d**-0.5).masked_fill(~seen, -math.inf), -1)
        o, a = (w @ k[:, :dv]).transpose(0, 1), (w @ k[:, :dv].abs()).transpose(0, 1)
        outs.append(o.reshape(n, -1))
        bounds.append((2**-8 * (a + o.abs())).reshape(n, -1))
    return q, cache.bfloat16(), tables, ctx, torch.cat(outs), torch.cat(bounds)


@pytest.mark.parametrize(
    "nh,d,dv,block_size,window,lens,starts",
    [
        (16, 576, 512, 16, 0, [130, 1, 17], [0, 70, 31]),  # two value halves, four query blocks in tensor memory; a single token among prompts
        (16, 576, 512, 16, 50, [9, 200], [300, 40]),  # a window whose pages have come back
        (5, 576, 512, 32, 0, [26, 51], [0, 13]),  # 125 of the 128 rows, tiles of 25 tokens, an odd last page
        (128, 320, 256, 48, 0, [3, 2], [126, 61]),  # a token a CTA, one value half, pages of three boxes
        (3, 80, 64, 64, 0, [64, 65], [0, 63]),  # a last block of 16 numbers, pages of a whole tile
        (1, 64, 64, 16, 7, [300], [5]),  # a row of one block: nothing of the queries in tensor memory, no part outside the values
        (7, 192, 128, 16, 0, [2], [127]),
        (128, 576, 512, 16, 0, [4, 1], [126, 255]),  # a last tile that is seen whole: 128 and 256 keys
        (16, 512, 512, 16, 0, [8, 16], [120, 112]),  # keys that are values whole
    ],
)
def test_latent_attention_of_many_queries_on_tcgen05(ops, nh, d, dv, block_size, window, lens, starts):
    for sharp in (1.0, 4.0):
        q, cache, tables, ctx, ref, bound = paged_latent_case(lens, starts, nh, d, dv, block_size, window, nh + d, sharp)
        qsl = [0]
        for n in lens:
            qsl.append(qsl[-1] + n)
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        tq = ops.latent_query_tile(nh)
        tiles = [(b, t) for b, n in enumerate(lens) for t in range(0, n, tq)]
        tiles = sorted(tiles, key=lambda t: -(starts[t[0]] + t[1])) + [(-1, 0), (len(lens) + 2, 0)]  # dead entries
        for work in (None, (i32(tiles).reshape(-1), len(tiles))):
            out = torch.full((sum(lens), nh * dv), float("nan"), device="cuda", dtype=torch.bfloat16)
            ops.latent_attention(
                dev(q), out, dev(cache), dev(tables), i32(qsl), i32(ctx), len(lens), max(lens), nh, d, dv, d**-0.5, window=window,
                kernel="tcgen05", err=err, query_tiles=work,
            )  # fmt: skip
            assert int(err.item()) == 0
            over = (out.cpu().double() - ref).abs() - bound
            assert float(over.max()) <= 0.0, (sharp, work is None, float(over.max()))


def test_latent_attention_routes_by_shape(ops):
    """What the tcgen05 kernel does not take stays with the mma.sync kernel, whose result it shares to rounding."""
    assert ops.latent_tcgen05_supported(torch.bfloat16, 16, 576, 512, 16)
    for nh, d, dv, bs in ((16, 640, 512, 16), (16, 576, 96, 16), (129, 576, 512, 16), (16, 576, 512, 8), (16, 72, 64, 16)):
        assert not ops.latent_tcgen05_supported(torch.bfloat16, nh, d, dv, bs)
    q, cache, tables, ctx, ref, bound = paged_latent_case([40], [3], 6, 128, 96, 8, 0, 1)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    out = torch.empty((40, 6 * 96), device="cuda", dtype=torch.bfloat16)
    ops.latent_attention(dev(q), out, dev(cache), dev(tables), i32([0, 40]), i32(ctx), 1, 40, 6, 128, 96, 128**-0.5)
    assert float(((out.cpu().double() - ref).abs() - bound).max()) <= 0.0
    with pytest.raises(ValueError):
        ops.latent_attention(dev(q), out, dev(cache), dev(tables), i32([0, 40]), i32(ctx), 1, 40, 6, 128, 96, 128**-0.5, kernel="tcgen05")


# ------------------------------------------------------------------ shaped scores on tcgen05 (many queries) and by TMA (decoding)


def paged_shaped_case(d, nh, nkv, block_size, window, keep, far, cap, sink, lens, starts):
    """Queries, caches on shuffled pages with NaN wherever no key lies, tables, contexts, biases, sinks, and per (request, head) the
    64-bit result with the bound on what rounding the weights and the result to bfloat16 may change (2^-9 each), times two."""
    g = torch.Generator().manual_seed(d + nh + window)
    ctx = [n + s for n, s in zip(lens, starts)]
    per = [-(-c // block_size) for c in ctx]
    order = torch.randperm(sum(per) + 2, generator=g).tolist()
    kc = torch.full((sum(per) + 2, nkv, block_size, d), float("nan"))
    vc = kc.clone()
    tables = torch.zeros((len(lens), max(per)), dtype=torch.int32)
    q = (1.5 * torch.randn((sum(lens), nh * d), generator=g)).bfloat16()
    rel = 2 * torch.randn((far + 1, nh), generator=g) if far else None
    sinks = torch.randn(nh, generator=g) if sink else None
    ref, bound, at, row = [], [], 0, 0
    for b, (n, c) in enumerate(zip(lens, ctx)):
        keys, vals = (torch.randn((c, nkv, d), generator=g).bfloat16() for _ in range(2))
        pages = order[at : at + per[b]]
        at += per[b]
        for j in range(c):
            kc[pages[j // block_size], :, j % block_size], vc[pages[j // block_size], :, j % block_size] = keys[j].float(), vals[j].float()
        lo, hi = -(-keep // block_size), (max(0, c - n - window + 1) // block_size if window else 0)
        tables[b, : per[b]] = torch.tensor([-1 if lo <= i < hi else p for i, p in enumerate(pages)], dtype=torch.int32)
        i, j = torch.arange(c - n, c)[:, None], torch.arange(c)[None]
        seen = (j <= i) & (((i - j < window) | (j < keep)) if window else True)
        for h in range(nh):
            qs = q[row : row + n, h * d : (h + 1) * d].double()
            s = qs @ keys[:, h // (nh // nkv)].double().T * d**-0.5
            s = cap * torch.tanh(s / cap) if cap else s
            s = s + rel[(i - j).clamp(0, far), h].double() if far else s
            s = s.masked_fill(~seen, -math.inf)
            if sink:
                s = torch.cat([s, sinks[h].double().expand(n, 1)], 1)
            w, v = torch.softmax(s, -1)[:, :c], vals[:, h // (nh // nkv)].double()
            ref.append((row, h, w @ v))
            bound.append(2**-8 * (w @ v.abs() + (w @ v).abs()))
        row += n
    return q, kc.bfloat16(), vc.bfloat16(), tables, ctx, rel, sinks, ref, bound


@pytest.mark.parametrize(
    "d,nh,nkv,block_size,window,keep,far,cap,sink,lens,starts",
    [
        (64, 8, 2, 16, 100, 70, 90, 0.0, False, [33, 1, 130], [300, 200, 0]),  # the bias ends inside the window; a kept tile and a half; a single token
        (64, 4, 4, 16, 64, 3, 4000, 0.0, True, [200], [77]),  # one head a key head, a table beyond every distance, sinks
        (64, 6, 2, 32, 0, 0, 50, 5.0, False, [65, 20], [0, 63]),  # 126 of the 128 rows, a bias on capped scores, no window
        (64, 8, 1, 8, 40, 64, 30, 0.0, False, [90], [140]),  # eight heads a key head, pages that come key by key, kept keys of one tile
        (128, 8, 2, 16, 130, 200, 128, 3.0, True, [70, 3], [250, 0]),  # heads of 128 with everything at once; kept keys reach into the window
        (64, 8, 2, 16, 90, 10, 0, 0.0, False, [64, 64], [64, 128]),  # kept keys alone
        (64, 16, 1, 16, 0, 0, 0, 30.0, True, [150], [10]),  # sixteen heads a key head, capped scores and sinks
        (128, 2, 1, 48, 1, 0, 7, 0.0, False, [129], [0]),  # a window of the query itself
    ],
)
def test_shaped_scores_of_many_queries_on_tcgen05(ops, d, nh, nkv, block_size, window, keep, far, cap, sink, lens, starts):
    """Unused places of the pages and pages that have come back hold nothing the kernel may read."""
    q, kc, vc, tables, ctx, rel, sinks, ref, bound = paged_shaped_case(d, nh, nkv, block_size, window, keep, far, cap, sink, lens, starts)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    qsl = [0]
    for n in lens:
        qsl.append(qsl[-1] + n)
    bias = ops.DistanceBias(dev(rel), i32(list(range(far + 1)))) if far else None
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    tq = ops.tcgen05_query_tile(nh, nkv)
    tiles = sorted([(b, t) for b, n in enumerate(lens) for t in range(0, n, tq)], key=lambda t: -(starts[t[0]] + t[1])) + [(-1, 0)]
    assert ops.shaped_tcgen05_supported(torch.bfloat16, nh, nkv, d, bias is not None)
    for work in (None, (i32(tiles).reshape(-1), len(tiles))):
        out = torch.full((sum(lens), nh * d), float("nan"), device="cuda", dtype=torch.bfloat16)
        ops.paged_attention(
            dev(q), out, dev(kc), dev(vc), dev(tables), i32(qsl), i32(ctx), len(lens), max(lens), nh, nkv, d, d**-0.5,
            window=window, keep_first=keep, bias=bias, softcap=cap, sinks=dev(sinks) if sink else None, err=err, query_tiles=work,
        )  # fmt: skip
        assert int(err.item()) == 0
        got = out.cpu().double()
        for (r0, h, o), e in zip(ref, bound):
            over = (got[r0 : r0 + o.shape[0], h * d : (h + 1) * d] - o).abs() - e
            assert float(over.max()) <= 0.0, (work is None, r0, h, float(over.max()))


@pytest.mark.parametrize(
    "d,nh,nkv,block_size,window,keep,far,cap,sink,ctx",
    [
        (64, 8, 2, 16, 100, 70, 90, 0.0, False, [333, 40, 101, 1]),  # kept keys before the window, inside it, longer than the context
        (64, 4, 4, 16, 64, 3, 4000, 0.0, True, [277, 64]),  # one head a key head, sinks
        (64, 6, 2, 32, 0, 0, 50, 5.0, False, [129, 16]),  # three heads a key head, a bias on capped scores
        (128, 8, 1, 16, 130, 200, 128, 3.0, True, [500, 131, 17]),  # heads of 128 with everything at once
        (64, 8, 2, 16, 16, 130, 0, 0.0, False, [400, 129]),  # kept keys alone, several ranges of them and ranges of none
        (64, 16, 2, 48, 0, 0, 0, 30.0, True, [700]),  # capped scores and sinks
    ],
)
def test_shaped_scores_of_a_decode_step_by_tma(ops, d, nh, nkv, block_size, window, keep, far, cap, sink, ctx):
    """Every form of the ranges' merge: one range, a thread-block cluster, tickets; ranges doubled on the device; and of a mixed
    batch the single tokens alone."""
    b = len(ctx)
    q, kc, vc, tables, _, rel, sinks, ref, bound = paged_shaped_case(d, nh, nkv, block_size, window, keep, far, cap, sink, [1] * b, [c - 1 for c in ctx])
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    bias = ops.DistanceBias(dev(rel), i32(list(range(far + 1)))) if far else None
    for split, cluster, wave in ((64, True, 0), (64, False, 0), (128, False, 2 * nkv * b), (1024, False, 0)):
        splits = -(-max(ctx) // split)
        scratch = (torch.full((b, nh, splits, d), float("nan"), device="cuda"), torch.full((b, nh, splits, 2), float("nan"), device="cuda"), i32([0] * b * nkv))
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        for single in (False, True):
            out = torch.full((b, nh * d), float("nan"), device="cuda", dtype=torch.bfloat16)
            ops.paged_attention(
                dev(q), out, dev(kc), dev(vc), dev(tables), i32(list(range(b + 1))), i32(ctx), b, 1, nh, nkv, d, d**-0.5, window=window, keep_first=keep,
                bias=bias, softcap=cap, sinks=dev(sinks) if sink else None, err=err, scratch=scratch, max_context=max(ctx), split_size=split,
                cluster=cluster, wave_target=wave, kernel="tma" if single else "auto", single_only=single,
            )  # fmt: skip
            assert int(err.item()) == 0 and int(scratch[2].abs().max()) == 0
            for (r0, h, o), e in zip(ref, bound):
                over = (out.cpu().double()[r0, h * d : (h + 1) * d] - o[0]).abs() - e[0]
                assert float(over.max()) <= 0.0, (split, cluster, r0, h, float(over.max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,nh,dv", [(1, 1, 8), (3, 5, 7), (5, 3, 24), (700, 16, 192), (9500, 2, 4), (2, 70, 256), (3, 24, 1), (5, 20, 1), (2, 2100, 1)])
def test_head_gate_widths(ops, dtype, n, nh, dv):
    """Heads that come as 16-byte words and heads that do not, a gate a channel, rows that start off such a word, more tokens than the
    grid has rows."""
    g = torch.Generator().manual_seed(n + dv)
    y, z = torch.randn(n, nh * dv, generator=g).to(dtype), (3.0 * torch.randn(n, nh + 16 + nh % 2, generator=g)).to(dtype)
    at = 8 if dv != 7 else 1
    want = (y.double().view(n, nh, dv) * torch.sigmoid(z[:, at : nh + at].double())[..., None]).view(n, -1)
    for shift in (0, 1):
        buf = torch.zeros(n * nh * dv + 2, dtype=dtype, device="cuda")
        got = buf[shift : shift + n * nh * dv].view(n, -1)
        got.copy_(y)
        ops.head_gate(got, z.cuda()[:, at : nh + at], nh, dv)
        # one rounding of the result, and a few of float on the way
        tol = (2.0**-8 if dtype == torch.bfloat16 else 2.0**-20) * want.abs() + 1e-30
        assert ((got.cpu().double() - want).abs() <= tol).all() and float(buf[:shift].abs().sum()) == 0 and float(buf[shift + n * nh * dv :].abs().sum()) == 0


def run_shaped(ops, d, nh, nkv, block_size, window, keep, far, cap, sink, lens, starts, decode=None, **kw):
    """Runs a case of ``paged_shaped_case`` and returns (output, largest excess over the bound).  ``decode``: (split, cluster)."""
    q, kc, vc, tables, ctx, rel, sinks, ref, bound = paged_shaped_case(d, nh, nkv, block_size, window, keep, far, cap, sink, lens, starts)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    qsl, b = [0], len(lens)
    for n in lens:
        qsl.append(qsl[-1] + n)
    if decode is not None:
        splits = -(-max(ctx) // decode[0])
        scratch = (torch.full((b, nh, splits, d), float("nan"), device="cuda"), torch.full((b, nh, splits, 2), float("nan"), device="cuda"), i32([0] * b * nkv))
        kw = dict(kw, scratch=scratch, max_context=max(ctx), split_size=decode[0], cluster=decode[1])
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.full((sum(lens), nh * d), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.paged_attention(
        dev(q), out, dev(kc), dev(vc), dev(tables), i32(qsl), i32(ctx), b, max(lens), nh, nkv, d, d**-0.5, window=window, keep_first=keep,
        bias=ops.DistanceBias(dev(rel), i32(list(range(far + 1)))) if far else None, softcap=cap, sinks=dev(sinks) if sink else None, err=err, **kw,
    )  # fmt: skip
    assert int(err.item()) == 0
    got = out.cpu().double()
    over = max(float(((got[r0 : r0 + o.shape[0], h * d : (h + 1) * d] - o).abs() - e).max()) for (r0, h, o), e in zip(ref, bound))
    return out.cpu(), over


@pytest.mark.parametrize(
    "d,nh,nkv,block_size,window,keep,far,cap,sink,lens,starts,takes",
    [
        (64, 8, 2, 16, 100, 70, 90, 0.0, False, [33, 1, 130], [300, 200, 0], True),
        (128, 8, 2, 16, 130, 200, 128, 3.0, True, [70, 3], [250, 0], True),
        (64, 16, 1, 16, 0, 0, 0, 30.0, True, [150], [10], True),  # sixteen heads a key head, without a bias
        (64, 16, 1, 16, 60, 20, 40, 0.0, False, [70], [100], False),  # with one: more than a tile's biases have room for
        (128, 9, 1, 8, 0, 0, 50, 5.0, True, [40, 5], [0, 70], False),
    ],
)
def test_shaped_scores_of_many_queries_by_either_kernel(ops, d, nh, nkv, block_size, window, keep, far, cap, sink, lens, starts, takes):
    """The mma.sync tile kernel, which stays for what the tcgen05 kernel's form does not take; and which of them "auto" is."""
    case = (d, nh, nkv, block_size, window, keep, far, cap, sink, lens, starts)
    auto, over = run_shaped(ops, *case)
    assert over <= 0.0, over
    tiles, over = run_shaped(ops, *case, kernel="mma")
    assert over <= 0.0, over
    if takes:
        assert torch.equal(auto, run_shaped(ops, *case, kernel="tcgen05")[0]) and not torch.equal(auto, tiles)
    else:
        assert torch.equal(auto, tiles)
        with pytest.raises(ValueError):
            run_shaped(ops, *case, kernel="tcgen05")
    with pytest.raises(ValueError):
        run_shaped(ops, *case, kernel="tma")


@pytest.mark.parametrize(
    "d,nh,nkv,block_size,window,keep,far,cap,sink,ctx,takes",
    [
        (64, 8, 2, 16, 100, 70, 90, 0.0, False, [333, 40, 101, 1], True),
        (128, 8, 1, 16, 130, 200, 128, 3.0, True, [500, 131, 17], True),
        (64, 16, 1, 16, 60, 20, 40, 0.0, False, [300, 7], False),  # more than eight heads a key head
        (64, 8, 2, 8, 0, 0, 50, 5.0, False, [200, 65], False),  # pages that are no multiple of sixteen
    ],
)
def test_shaped_scores_of_a_decode_step_by_either_kernel(ops, d, nh, nkv, block_size, window, keep, far, cap, sink, ctx, takes):
    case = (d, nh, nkv, block_size, window, keep, far, cap, sink, [1] * len(ctx), [c - 1 for c in ctx])
    for split in (64, 1024):
        auto, over = run_shaped(ops, *case, decode=(split, False))
        assert over <= 0.0, (split, over)
        ranges, over = run_shaped(ops, *case, decode=(split, False), kernel="mma")
        assert over <= 0.0, (split, over)
        if takes:
            assert torch.equal(auto, run_shaped(ops, *case, decode=(split, False), kernel="tma")[0])
            assert split == 64 or not torch.equal(auto, ranges)  # (ranges of 64 keys: both give a warp sixteen)
        else:
            assert torch.equal(auto, ranges)
            with pytest.raises(ValueError):
                run_shaped(ops, *case, decode=(split, False), kernel="tma")
        with pytest.raises(ValueError):
            run_shaped(ops, *case, decode=(split, False), kernel="tcgen05")


def test_latent_attention_of_many_queries_is_the_tcgen05_kernel_s(ops):
    """"auto" takes the tcgen05 kernel where that takes the shape, with and without a list of tiles."""
    q, cache, tables, ctx, ref, bound = paged_latent_case([150, 3], [20, 500], 16, 576, 512, 16, 0, 2)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    outs = {}
    for kernel in ("auto", "tcgen05", "mma"):
        out = outs[kernel] = torch.empty((153, 16 * 512), device="cuda", dtype=torch.bfloat16)
        ops.latent_attention(dev(q), out, dev(cache), dev(tables), i32([0, 150, 153]), i32(ctx), 2, 150, 16, 576, 512, 576**-0.5, kernel=kernel)
        assert float(((out.cpu().double() - ref).abs() - bound).max()) <= 0.0
    assert torch.equal(outs["auto"], outs["tcgen05"]) and not torch.equal(outs["auto"], outs["mma"])


@pytest.mark.parametrize("d,nh,nkv,block_size", [(64, 8, 2, 16), (128, 4, 1, 16), (64, 9, 1, 8), (48, 4, 2, 16)])
@pytest.mark.parametrize("far,cap", [(0, 0.0), (30, 0.0), (0, 5.0)])
def test_kept_keys_without_a_window_change_nothing(ops, d, nh, nkv, block_size, far, cap):
    """Every key before a query is seen anyway: by the tensor-core kernels and, with heads of 48, on the FP32 pipes."""
    for lens, starts, decode in (([70, 3], [90, 0], None), ([1, 1], [300, 20], (64, False)), ([1, 1], [300, 20], (512, True))):
        outs = []
        for keep in (0, 70):
            out, over = run_shaped(ops, d, nh, nkv, block_size, 0, keep, far, cap, False, lens, starts, decode=decode)
            assert over <= 0.0, (lens, keep, over)
            outs.append(out)
        plain_elsewhere = d == 64 and nh == 9 or d == 48  # without kept keys other kernels take plain scores there
        assert torch.equal(*outs) or (plain_elsewhere and not far and not cap)


@pytest.mark.parametrize("shape", [(64, 8, 2, 16), (64, 4, 2, 8), (128, 4, 1, 16)])
@pytest.mark.parametrize("far,cap,window,keep", [(0, 0.0, 0, 0), (30, 0.0, 0, 0), (0, 5.0, 0, 0), (20, 3.0, 90, 70)])
@pytest.mark.parametrize("bad", [5, 70, 133, 199])  # in either of the tiles that two groups of warps take in turn, and in the last
def test_what_is_no_number_shows_in_the_rows_that_see_it(ops, shape, far, cap, window, keep, bad):
    """One key that is NaN: every head of every query that sees it is NaN, the others are what they were."""
    d, nh, nkv, bs = shape
    q, kc, vc, tables, ctx, rel, sinks, ref, bound = paged_shaped_case(d, nh, nkv, bs, window, keep, far, cap, False, [200], [0])
    kc[int(tables[0, bad // bs]), :, bad % bs, 3] = float("nan")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    bias = ops.DistanceBias(dev(rel), i32(list(range(far + 1)))) if far else None
    for kernel in ("auto", "mma"):
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        out = torch.zeros((200, nh * d), device="cuda", dtype=torch.bfloat16)
        ops.paged_attention(
            dev(q), out, dev(kc), dev(vc), dev(tables), i32([0, 200]), i32([200]), 1, 200, nh, nkv, d, d**-0.5, window=window, keep_first=keep,
            bias=bias, softcap=cap, err=err, kernel=kernel,
        )  # fmt: skip
        assert int(err.item()) == 0
        got, i = out.cpu().double(), torch.arange(200)
        sees = (i >= bad) & ((i - bad < window) | (bad < keep) if window else True)
        assert torch.isnan(got[sees]).all() and not torch.isnan(got[~sees]).any(), kernel
        for (r0, h, o), e in zip(ref, bound):
            assert float(((got[:, h * d : (h + 1) * d] - o).abs() - e)[~sees].max()) <= 0.0, (kernel, h)


@pytest.mark.parametrize("d,nh,nkv", [(64, 8, 2), (128, 8, 1)])
@pytest.mark.parametrize("far,cap", [(0, 0.0), (30, 0.0), (0, 5.0)])
def test_what_is_no_number_shows_in_a_decode_step(ops, d, nh, nkv, far, cap):
    """A NaN key in one of three sequences: as the only range of its sequence, among the ranges of a cluster, among ranges that
    merge by tickets, and on the mma.sync kernel."""
    ctx = [40, 200, 130]
    q, kc, vc, tables, _, rel, sinks, ref, bound = paged_shaped_case(d, nh, nkv, 16, 0, 0, far, cap, False, [1] * 3, [c - 1 for c in ctx])
    kc[int(tables[1, 150 // 16]), :, 150 % 16, 3] = float("nan")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    bias = ops.DistanceBias(dev(rel), i32(list(range(far + 1)))) if far else None
    for split, cluster, kernel in ((64, True, "tma"), (64, False, "tma"), (256, False, "tma"), (64, False, "mma")):
        ns = -(-200 // split)
        scratch = (torch.zeros((3, nh, ns, d), device="cuda"), torch.zeros((3, nh, ns, 2), device="cuda"), i32([0] * 3 * nkv))
        out, err = torch.zeros((3, nh * d), device="cuda", dtype=torch.bfloat16), torch.zeros(1, dtype=torch.int32, device="cuda")
        ops.paged_attention(
            dev(q), out, dev(kc), dev(vc), dev(tables), i32([0, 1, 2, 3]), i32(ctx), 3, 1, nh, nkv, d, d**-0.5, bias=bias, softcap=cap, err=err,
            scratch=scratch, max_context=200, split_size=split, cluster=cluster, kernel=kernel,
        )  # fmt: skip
        assert int(err.item()) == 0 and int(scratch[2].abs().max()) == 0
        got = out.cpu().double()
        assert torch.isnan(got[1]).all(), (split, cluster, kernel)
        for (r0, h, o), e in zip(ref, bound):
            if r0 != 1:
                assert float(((got[r0, h * d : (h + 1) * d] - o[0]).abs() - e[0]).max()) <= 0.0, (split, cluster, kernel, r0, h)


@pytest.mark.parametrize("ranges", [1, 8, 255, 256, 257, 3000, 6140, 30000])
def test_latent_decode_merges_any_number_of_ranges(ops, ranges):
    """Scratch of up to 30,000 ranges of 32 keys, and contexts that use all of the first few hundred and their edges."""
    nh, d, dv, bs = 3, 64, 64, 16
    used = min(ranges, 600)
    ctx = [used * 32, max(1, used * 32 - 17), 1]
    q, cache, tables, ctx, ref, bound = paged_latent_case([1] * 3, [c - 1 for c in ctx], nh, d, dv, bs, 0, ranges)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    scratch = (torch.full((3, nh, ranges, dv), float("nan"), device="cuda"), torch.full((3, nh, ranges, 2), float("nan"), device="cuda"))
    out = torch.full((3, nh * dv), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.latent_attention(
        dev(q), out, dev(cache), dev(tables), i32([0, 1, 2, 3]), i32(ctx), 3, 1, nh, d, dv, d**-0.5, scratch=scratch, max_context=max(ctx), split_size=32,
    )  # fmt: skip
    assert float(((out.cpu().double() - ref).abs() - bound).max()) <= 0.0


def test_latent_decode_shows_what_is_no_number_in_any_range(ops):
    """A NaN key in a range whose scores lie so far below the others' that its factor in the merge is zero."""
    nh, d, dv = 2, 64, 64
    q, cache, tables, ctx, ref, bound = paged_latent_case([1, 1], [199, 199], nh, d, dv, 16, 0, 5)
    q = torch.ones_like(q)
    for b in range(2):
        for j in range(200):
            cache[int(tables[b, j // 16]), 0, j % 16] = 20.0 if j >= 64 else -20.0  # scores of 160 and -160
    cache[int(tables[1, 2]), 0, 5, 3] = float("nan")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    scratch = (torch.zeros((2, nh, 4, dv), device="cuda"), torch.zeros((2, nh, 4, 2), device="cuda"))
    out = torch.zeros((2, nh * dv), device="cuda", dtype=torch.bfloat16)
    ops.latent_attention(
        dev(q), out, dev(cache), dev(tables), i32([0, 1, 2]), i32(ctx), 2, 1, nh, d, dv, d**-0.5, scratch=scratch, max_context=200, split_size=64,
    )  # fmt: skip
    assert (out[0] == 20.0).all() and torch.isnan(out[1]).all()


def test_head_gate_of_rows_beyond_32_bits(ops):
    y = torch.ones((1, 2 * (2**30 + 8)), dtype=torch.bfloat16, device="cuda")
    z = torch.tensor([[0.0, 2.0]], dtype=torch.bfloat16, device="cuda")
    ops.head_gate(y, z, 2, 2**30 + 8)
    for h, want in ((0, 0.5), (1, torch.sigmoid(torch.tensor(2.0)).bfloat16().item())):
        half = y[0, h * (2**30 + 8) : (h + 1) * (2**30 + 8)]
        assert float(half.min()) == float(half.max()) == want


@pytest.mark.parametrize("nh,d,dv,block_size", [(16, 576, 512, 16), (16, 576, 512, 64), (4, 208, 128, 48), (5, 64, 64, 32)])
@pytest.mark.parametrize("ctx", [1, 15, 17, 63, 65, 100, 127, 129, 143, 255, 257, 300])
def test_latent_attention_of_contexts_that_end_anywhere(ops, nh, d, dv, block_size, ctx):
    """The last tile's boxes: whole ones, the one that the context ends in, and those past it, whose places hold NaN."""
    n = min(ctx, 40)
    q, cache, tables, ctxs, ref, bound = paged_latent_case([n, 1], [ctx - n, ctx - 1], nh, d, dv, block_size, 0, ctx + d)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.full((n + 1, nh * dv), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.latent_attention(
        dev(q), out, dev(cache), dev(tables), i32([0, n, n + 1]), i32(ctxs), 2, n, nh, d, dv, d**-0.5, kernel="tcgen05", err=err,
    )  # fmt: skip
    assert int(err.item()) == 0
    assert float(((out.cpu().double() - ref).abs() - bound).max()) <= 0.0


def off_by(out, ref, d):
    """Relative error of ``run_shaped``'s output against the 64-bit results of its case."""
    got = out.double()
    num = sum(float((got[r0 : r0 + o.shape[0], h * d : (h + 1) * d] - o).square().sum()) for r0, h, o in ref)
    return math.sqrt(num / sum(float(o.square().sum()) for _, _, o in ref))


@pytest.mark.parametrize("d,nh,nkv,far,cap,sink", [(64, 8, 2, 200, 0.0, False), (64, 8, 2, 0, 30.0, False), (128, 8, 2, 100, 20.0, True)])
def test_shaped_scores_on_tcgen05_are_no_further_off(ops, d, nh, nkv, far, cap, sink):
    """Against 64 bits, as far off as the mma.sync kernel: both round the same weights to bfloat16, with the largest one exact.
    4,000 rows: the ratio of two such errors varies by 1 / sqrt(2 x 4,000), so 4 % are more than three times that."""
    case = (d, nh, nkv, 16, 0, 0, far, cap, sink, [130, 370], [400, 0])
    ref = paged_shaped_case(*case)[7]
    errors = [off_by(run_shaped(ops, *case, kernel=kernel)[0], ref, d) for kernel in ("tcgen05", "mma")]
    assert errors[0] <= 1.04 * errors[1], errors


@pytest.mark.parametrize("d,nh,nkv,far,cap,sink", [(64, 8, 2, 200, 0.0, False), (64, 8, 2, 0, 30.0, False), (128, 8, 2, 100, 20.0, True)])
def test_shaped_scores_of_a_decode_step_by_tma_are_no_further_off(ops, d, nh, nkv, far, cap, sink):
    """With the same ranges a warp has the same keys in either kernel, and both leave the largest weight exact: the errors against
    64 bits differ by the order of float sums alone."""
    case = (d, nh, nkv, 16, 0, 0, far, cap, sink, [1] * 24, [400 - 7 * i for i in range(24)])
    ref = paged_shaped_case(*case)[7]
    errors = [off_by(run_shaped(ops, *case, decode=(256, False), kernel=kernel)[0], ref, d) for kernel in ("tma", "mma")]
    assert errors[0] <= 1.02 * errors[1], errors


@pytest.mark.parametrize("nh,d,dv,lens,starts", [(16, 576, 512, [150, 100], [0, 300]), (8, 320, 256, [300], [200])])
@pytest.mark.parametrize("sharp", [1.0, 3.0])
def test_latent_attention_on_tcgen05_is_no_further_off(ops, nh, d, dv, lens, starts, sharp):
    """Against 64 bits, as far off as the mma.sync kernel.  2,400 and more rows: the ratio of two such errors varies by
    1 / sqrt(2 x 2,400), so 5 % are more than three times that."""
    q, cache, tables, ctx, ref, bound = paged_latent_case(lens, starts, nh, d, dv, 16, 0, 3, sharp)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    qsl, errors = [0], []
    for n in lens:
        qsl.append(qsl[-1] + n)
    for kernel in ("tcgen05", "mma"):
        out = torch.empty((sum(lens), nh * dv), device="cuda", dtype=torch.bfloat16)
        ops.latent_attention(dev(q), out, dev(cache), dev(tables), i32(qsl), i32(ctx), len(lens), max(lens), nh, d, dv, d**-0.5, kernel=kernel)
        errors.append(float((out.cpu().double() - ref).norm() / ref.norm()))
    assert errors[0] <= 1.05 * errors[1], errors


@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("bad", [3, 64, 140, 200, 243])
def test_latent_attention_keeps_what_is_no_number_near(ops, window, bad):
    """A NaN row of the cache: every query that sees it is NaN; of the others only those whose tile of eight queries reaches into
    the sixteen keys around it may be."""
    nh, d, dv, n = 16, 192, 128, 250
    q, cache, tables, ctx, ref, bound = paged_latent_case([n], [0], nh, d, dv, 16, window, bad)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    page = int(tables[0, bad // 16])
    cache[page if page >= 0 else -1, 0, bad % 16] = float("nan")
    for kernel in ("tcgen05", "mma"):
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        out = torch.zeros((n, nh * dv), device="cuda", dtype=torch.bfloat16)
        ops.latent_attention(dev(q), out, dev(cache), dev(tables), i32([0, n]), i32(ctx), 1, n, nh, d, dv, d**-0.5, window=window, kernel=kernel, err=err)
        assert int(err.item()) == 0
        got, i = out.cpu().double(), torch.arange(n)
        sees = (i >= bad) & (i - bad < (window or n))
        first = i // 8 * 8
        near = (first + 7 >= bad // 16 * 16) & (first - (window or n) + 1 <= bad // 16 * 16 + 15)
        assert torch.isnan(got[sees]).all(), kernel
        if kernel == "tcgen05" and bool((~near).any()):
            assert not torch.isnan(got[~near]).any()
            assert float(((got - ref).abs() - bound)[~near].max()) <= 0.0


@pytest.mark.parametrize("longest", [64, 65])
def test_latent_attention_of_short_contexts_stays_with_mma(ops, longest):
    q, cache, tables, ctx, ref, bound = paged_latent_case([longest, 3], [0, 20], 16, 576, 512, 16, 0, 2)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    outs = {}
    for kernel, known in (("auto", longest), ("auto", None), ("tcgen05", longest), ("mma", None)):
        out = outs[kernel, known] = torch.empty((longest + 3, 16 * 512), device="cuda", dtype=torch.bfloat16)
        ops.latent_attention(
            dev(q), out, dev(cache), dev(tables), i32([0, longest, longest + 3]), i32(ctx), 2, longest, 16, 576, 512, 576**-0.5, kernel=kernel, max_context=known,
        )  # fmt: skip
        assert float(((out.cpu().double() - ref).abs() - bound).max()) <= 0.0
    assert torch.equal(outs["auto", None], outs["tcgen05", longest]) and not torch.equal(outs["auto", None], outs["mma", None])
    assert torch.equal(outs["auto", longest], outs["mma", None] if longest == 64 else outs["auto", None])


@pytest.mark.parametrize("n,longest", [(3, 3), (40, 60), (200, 300)])
def test_shaped_scores_of_short_contexts_choose_their_kernel(ops, n, longest):
    case = (64, 8, 2, 16, 0, 0, 50, 5.0, False, [n, 1], [longest - n, 0])
    auto, over = run_shaped(ops, *case, max_context=longest)
    assert over <= 0.0, over
    pays = ops.shaped_tcgen05_pays(64, 4, 2, 2, n + 1, n, longest, True)
    assert pays == (longest == 300)
    assert torch.equal(auto, run_shaped(ops, *case, kernel="tcgen05" if pays else "mma")[0])
    assert torch.equal(run_shaped(ops, *case, kernel="tcgen05", max_context=longest)[0], run_shaped(ops, *case)[0])
