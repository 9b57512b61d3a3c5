"""GPU parity tests of the split-KV decode path.  Tolerance: atol = rtol = 2e-3 vs the fp32 oracle."""
import ctypes

import pytest
import torch

from _util import check_close, load_decode
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def run_decode(kerns, q, kc, vc, lens):
    out = torch.full(q.shape, float("nan"), dtype=q.dtype, device="cuda")
    kerns.flash_attn_decode(q.cuda(), kc.cuda(), vc.cuda(), lens.cuda().to(torch.int32), out)
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("name", ["decode_g4_d128", "decode_g1_d64_bf16", "decode_g6_d128"])
def test_golden_vectors(kerns, name):
    q, k, v, lens, want = load_decode(name)
    check_close(run_decode(kerns, q, k, v, lens), want, name, bf16=q.dtype == torch.bfloat16)


@pytest.mark.parametrize("D,H,Hkv,dtype", [(128, 32, 8, torch.float16), (64, 32, 8, torch.float16),
                                            (128, 16, 2, torch.bfloat16), (128, 5, 5, torch.float16),
                                            (64, 32, 2, torch.float16)])
def test_ragged_lengths(kerns, D, H, Hkv, dtype):
    B, Lmax = 9, 2100
    g = torch.Generator().manual_seed(31 + D + H)
    q = torch.randn(B, H, 1, D, generator=g).to(dtype)
    kc = torch.randn(B, Hkv, Lmax, D, generator=g).to(dtype)
    vc = torch.randn(B, Hkv, Lmax, D, generator=g).to(dtype)
    lens = torch.tensor([1, 2, 15, 16, 17, 511, 512, 513, 2100], dtype=torch.int32)
    want = O.decode_oracle(q, kc, vc, lens)
    check_close(run_decode(kerns, q, kc, vc, lens), want, "ragged", bf16=dtype == torch.bfloat16)


def test_padding_is_never_read(kerns):
    """NaN beyond lens[b] must not reach the output; a zero-length sequence yields zeros."""
    B, H, Hkv, Lmax, D = 3, 8, 2, 700, 128
    g = torch.Generator().manual_seed(77)
    q = torch.randn(B, H, 1, D, generator=g).half()
    kc = torch.randn(B, Hkv, Lmax, D, generator=g).half()
    vc = torch.randn(B, Hkv, Lmax, D, generator=g).half()
    lens = torch.tensor([0, 300, 641], dtype=torch.int32)
    want = O.decode_oracle(q, kc, vc, torch.tensor([1, 300, 641]))
    for b in range(B):
        kc[b, :, int(lens[b]):] = float("nan")
        vc[b, :, int(lens[b]):] = float("nan")
    got = run_decode(kerns, q, kc, vc, lens)
    assert torch.count_nonzero(got[0]) == 0
    check_close(got[1:], want[1:], "padding")


def test_strided_cache_views(kerns):
    """Cache stored [B, Lmax, Hkv, D] and viewed as [B, Hkv, Lmax, D]; batch-sliced shard."""
    B, H, Hkv, Lmax, D = 4, 8, 2, 600, 128
    g = torch.Generator().manual_seed(78)
    q = torch.randn(B, H, 1, D, generator=g).half()
    kc = torch.randn(B, Lmax, Hkv, D, generator=g).half().transpose(1, 2)
    vc = torch.randn(B, Lmax, Hkv, D, generator=g).half().transpose(1, 2)
    lens = torch.tensor([600, 77, 512, 130], dtype=torch.int32)
    want = O.decode_oracle(q, kc, vc, lens)
    qd, kd, vd, ld = q.cuda(), kc.cuda(), vc.cuda(), lens.cuda()
    assert not kd.is_contiguous()
    out = torch.zeros(B, H, 1, D, dtype=torch.float16, device="cuda")
    kerns.flash_attn_decode(qd, kd, vd, ld, out)
    check_close(out, want, "strided cache")
    part = torch.zeros(2, H, 1, D, dtype=torch.float16, device="cuda")
    kerns.flash_attn_decode(qd[2:], kd[2:], vd[2:], ld[2:].contiguous(), part)
    assert torch.equal(part, out[2:])


@pytest.mark.parametrize("chunk", [64, 256, 1024, 8192])
def test_chunk_sizes_through_the_c_abi(chunk):
    """Any chunk (split) size gives the same answer within tolerance: called through the C ABI directly."""
    from minfer.kernels.torch_ext import _lib
    B, H, Hkv, Lmax, D = 5, 8, 2, 1500, 128
    g = torch.Generator().manual_seed(79)
    q = torch.randn(B, H, 1, D, generator=g).half()
    kc = torch.randn(B, Hkv, Lmax, D, generator=g).half()
    vc = torch.randn(B, Hkv, Lmax, D, generator=g).half()
    lens = torch.tensor([1500, 3, 1024, 1025, 64], dtype=torch.int32)
    want = O.decode_oracle(q, kc, vc, lens)
    qd, kd, vd, ld = q.cuda(), kc.cuda(), vc.cuda(), lens.cuda()
    out = torch.zeros(B, H, 1, D, dtype=torch.float16, device="cuda")
    need = _lib.lib.minfer_attn_decode_workspace_bytes(B, H, Lmax, D, chunk)
    ws = torch.full((need,), 0xFF, dtype=torch.uint8, device="cuda")   # the workspace may hold anything
    p = _lib.DecodeParams()
    p.q, p.k_cache, p.v_cache, p.lens, p.out = qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), ld.data_ptr(), out.data_ptr()
    p.workspace, p.workspace_bytes = ws.data_ptr(), need
    p.batch, p.n_heads, p.n_kv_heads, p.max_len, p.head_dim = B, H, Hkv, Lmax, D
    p.dtype, p.chunk, p.softmax_scale = _lib.F16, chunk, 0.0
    for i in range(2):
        p.q_stride[i], p.out_stride[i] = qd.stride(i), out.stride(i)
    for i in range(3):
        p.kv_stride[i] = kd.stride(i)
    rc = _lib.lib.minfer_attn_decode(ctypes.byref(p), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, _lib.strerror(rc)
    torch.cuda.synchronize()
    check_close(out, want, f"chunk={chunk}")
    # repeated calls, back to back on the same workspace, give the same bits
    first = out.clone()
    for _ in range(20):
        out.fill_(float("nan"))
        assert _lib.lib.minfer_attn_decode(ctypes.byref(p), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        assert torch.equal(out, first)
    p.workspace_bytes = need - 1
    assert _lib.lib.minfer_attn_decode(ctypes.byref(p), None) == 5


def test_config3_full_size(kerns):
    """Batch 64, 32/8 heads, D=128, lengths uniform in [512, 8192], cache padded to 8192 and
    filled everywhere (so an over-read would show): every sequence against the oracle."""
    B, H, Hkv, Lmax, D = 64, 32, 8, 8192, 128
    g = torch.Generator().manual_seed(2)
    lens = torch.randint(512, 8193, (B,), generator=g, dtype=torch.int32)
    lens[0], lens[1] = 512, 8192
    q = torch.randn(B, H, 1, D, generator=g).half()
    kd = torch.randn(B, Hkv, Lmax, D, device="cuda", dtype=torch.float16)
    vd = torch.randn(B, Hkv, Lmax, D, device="cuda", dtype=torch.float16)
    out = torch.full((B, H, 1, D), float("nan"), dtype=torch.float16, device="cuda")
    kerns.flash_attn_decode(q.cuda(), kd, vd, lens.cuda(), out)
    torch.cuda.synchronize()
    for b0 in range(0, B, 16):
        want = O.decode_oracle(q[b0:b0 + 16], kd[b0:b0 + 16].cpu(), vd[b0:b0 + 16].cpu(), lens[b0:b0 + 16])
        check_close(out[b0:b0 + 16], want, f"config3 b={b0}")
    out2 = torch.empty_like(out)
    kerns.flash_attn_decode(q.cuda(), kd, vd, lens.cuda(), out2)
    assert torch.equal(out, out2)


def test_argument_errors_raise(kerns):
    q = torch.zeros(2, 8, 1, 128, dtype=torch.float16, device="cuda")
    kc = torch.zeros(2, 2, 256, 128, dtype=torch.float16, device="cuda")
    lens = torch.tensor([5, 6], dtype=torch.int32, device="cuda")
    out = torch.zeros_like(q)
    with pytest.raises(RuntimeError):
        kerns.flash_attn_decode(q, kc, kc, lens.long(), out)
    with pytest.raises(RuntimeError):
        kerns.flash_attn_decode(q, kc, kc, lens[:1], out)
    with pytest.raises(RuntimeError):
        kerns.flash_attn_decode(q.expand(2, 8, 2, 128), kc, kc, lens, out.expand(2, 8, 2, 128))


@pytest.mark.parametrize("seed", range(8))
def test_random_shapes_against_the_oracle(kerns, seed):
    """Seeded random batch, heads, GQA group up to 16, head_dim, type, padded length and lengths (empty sequences
    included), contiguous or [B, Lmax, Hkv, D]-stored caches."""
    g = torch.Generator().manual_seed(7000 + seed)
    r = lambda lo, hi: int(torch.randint(lo, hi + 1, (1,), generator=g))  # noqa: E731
    B, Hkv, group = r(1, 9), r(1, 4), [1, 2, 3, 4, 5, 8, 16][r(0, 6)]
    H, D = Hkv * group, [64, 128][r(0, 1)]
    dtype = [torch.float16, torch.bfloat16][r(0, 1)]
    Lmax = r(1, 3000)
    lens = torch.randint(0, Lmax + 1, (B,), generator=g, dtype=torch.int32)
    lens[r(0, B - 1)] = Lmax
    q = torch.randn(B, H, 1, D, generator=g).to(dtype)
    if r(0, 1):
        kc = torch.randn(B, Lmax, Hkv, D, generator=g).to(dtype).transpose(1, 2)
        vc = torch.randn(B, Lmax, Hkv, D, generator=g).to(dtype).transpose(1, 2)
    else:
        kc = torch.randn(B, Hkv, Lmax, D, generator=g).to(dtype)
        vc = torch.randn(B, Hkv, Lmax, D, generator=g).to(dtype)
    want = O.attention_f64(q, kc, vc, lens=lens)
    got = run_decode(kerns, q, kc, vc, lens)
    assert torch.count_nonzero(got[lens == 0]) == 0
    live = lens > 0
    what = f"seed {seed}: B={B} H={H} Hkv={Hkv} D={D} Lmax={Lmax} {dtype}"
    if dtype == torch.bfloat16:
        from _util import check_close_bf16_by_keys
        check_close_bf16_by_keys(got[live], want[live], lens[live].view(-1, 1, 1, 1), what)
    else:
        check_close(got[live], want[live], what)


@pytest.mark.parametrize("B,Hkv,group,D,Lmax,dtype", [
    (1, 1, 1, 64, 15, torch.float16), (1, 2, 16, 128, 1100, torch.bfloat16),   # one block; clusters of 16, two column tiles
    (9, 2, 9, 64, 1024, torch.float16), (40, 2, 4, 128, 150, torch.float16),   # clusters of 16 and of 2
    (16, 1, 4, 128, 1100, torch.bfloat16), (10, 6, 3, 128, 700, torch.float16),     # clusters of 8 and of 4
    (150, 2, 8, 64, 300, torch.bfloat16),                                      # more pairs than one wave of blocks
    (256, 1, 2, 128, 1300, torch.float16), (257, 1, 2, 128, 1300, torch.float16),   # one block each, a batch that could be ranked and one that could not
    (256, 1, 2, 128, 2048, torch.float16), (257, 1, 2, 128, 2048, torch.float16)])  # two waves, ordered by length and not
def test_block_clusters_and_order_by_length(kerns, B, Hkv, group, D, Lmax, dtype):
    """Every cluster size and both orders, with lengths at the edges of the 16-key tiles and of the shares of a
    cluster's blocks (so that some blocks get nothing), empty sequences and equal lengths among them."""
    g = torch.Generator().manual_seed(B + D)
    H = Hkv * group
    lens = torch.randint(0, Lmax + 1, (B,), generator=g, dtype=torch.int32)
    edges = [Lmax, 0, 1, 16, 17, min(Lmax, 127), min(Lmax, 256), min(Lmax, 256)]
    lens[:min(B, len(edges))] = torch.tensor(edges[:B], dtype=torch.int32)
    q = torch.randn(B, H, 1, D, generator=g).to(dtype)
    kc = torch.randn(B, Hkv, Lmax, D, generator=g).to(dtype)
    vc = torch.randn(B, Hkv, Lmax, D, generator=g).to(dtype)
    want = O.attention_f64(q, kc, vc, lens=lens)
    for b in range(B):
        kc[b, :, int(lens[b]):] = float("nan")
        vc[b, :, int(lens[b]):] = float("nan")
    got = run_decode(kerns, q, kc, vc, lens)
    assert torch.count_nonzero(got[lens == 0]) == 0
    live = lens > 0
    if dtype == torch.bfloat16:
        from _util import check_close_bf16_by_keys
        check_close_bf16_by_keys(got[live], want[live], lens[live].view(-1, 1, 1, 1), f"B={B}")
    else:
        check_close(got[live], want[live], f"B={B} D={D}")
    assert torch.equal(got, run_decode(kerns, q, kc, vc, lens))


@pytest.mark.parametrize("D,H,Hkv,Lmax", [(128, 8, 2, 700), (64, 4, 4, 700), (64, 12, 1, 100), (128, 2, 1, 20)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_infinite_values_and_nan_scores(kerns, D, H, Hkv, Lmax, dtype):
    """A visible infinite value makes its dimension infinite and nothing else NaN, whatever the number of blocks that share
    the sequence; a row whose sum of weights is NaN (a NaN key or query) is zeros, as the merging kernel has it."""
    B = 3
    g = torch.Generator().manual_seed(D + H)
    q = torch.randn(B, H, 1, D, generator=g).to(dtype)
    kc = torch.randn(B, Hkv, Lmax, D, generator=g).to(dtype)
    vc = torch.randn(B, Hkv, Lmax, D, generator=g).to(dtype)
    lens = torch.tensor([Lmax - 1, 11, Lmax // 2], dtype=torch.int32)
    want = O.attention_f64(q, kc, vc, lens=lens)
    vc[:, :, 7, 3] = float("inf")
    kc[1, :, 10] = float("nan")
    q[2] = float("nan")
    got = run_decode(kerns, q, kc, vc, lens).float().cpu()
    assert (got[0, ..., 3] == float("inf")).all()
    keep = [d for d in range(D) if d != 3]
    check_close(got[:1][..., keep], want[:1][..., keep], "finite dimensions", bf16=dtype == torch.bfloat16)
    assert torch.count_nonzero(got[1:]) == 0


@pytest.mark.parametrize("B,Hkv,Lmax", [(6, 8, 8192), (13, 8, 4096), (255, 1, 2048), (256, 1, 2048)])
def test_lengths_outside_the_cache_are_clamped_in_order_by_length(kerns, B, Hkv, Lmax):
    """Calls that take the longest sequences first, batches that are and are not multiples of four: a negative length is an
    empty sequence (zeros), one beyond the cache is max_len, and no sequence is lost - the bits of the same call with clamped lengths."""
    D, dtype = 128, torch.float16
    g = torch.Generator(device="cuda").manual_seed(B)
    q = torch.randn(B, Hkv, 1, D, generator=g, device="cuda", dtype=dtype)
    kc = torch.randn(B, Hkv, Lmax, D, generator=g, device="cuda", dtype=dtype)
    vc = torch.randn(B, Hkv, Lmax, D, generator=g, device="cuda", dtype=dtype)
    lens = torch.randint(1, Lmax, (B,), generator=g, device="cuda", dtype=torch.int32)
    for odd in ([-5, 2 ** 31 - 1], [-2, Lmax + 3, -2 ** 31], [2 ** 31 - 1, -1, -2, -5]):
        bad = lens.clone()
        bad[torch.randperm(B, generator=g, device="cuda")[:len(odd)]] = torch.tensor(odd, device="cuda", dtype=torch.int32)
        outs = []
        for n in (bad, bad.clamp(0, Lmax)):
            out = torch.full((B, Hkv, 1, D), float("nan"), dtype=dtype, device="cuda")
            kerns.flash_attn_decode(q, kc, vc, n, out)
            outs.append(out)
        assert torch.equal(outs[0], outs[1])
        assert torch.count_nonzero(outs[0][bad <= 0]) == 0 and torch.isfinite(outs[0]).all()
        full = bad > Lmax
        if full.any():
            want = O.attention_f64(q[full].cpu(), kc[full].cpu(), vc[full].cpu(), lens=torch.full((int(full.sum()),), Lmax, dtype=torch.int32))
            check_close(outs[0][full], want, f"B={B} beyond the cache")


def test_weights_keep_the_precision_of_512_key_chunks(kerns):
    """Rounding the weights to 16 bits costs least where few keys share a reference maximum: a large call's error against 64
    bits is no more than that of chunks of 512 keys dealt out to four warps in 16-key tiles, each with a running maximum of
    its own.  (The two cut the keys differently; over 2048 rows that moves the error by about 0.5 %.)"""
    B, Hkv, group, D, Lmax = 64, 8, 4, 128, 8192
    g = torch.Generator(device="cuda").manual_seed(1)
    lens = torch.tensor([512 + (Lmax - 512) * i // (B - 1) for i in range(B)], dtype=torch.int32, device="cuda")
    q = torch.randn(B, Hkv * group, 1, D, generator=g, device="cuda", dtype=torch.float16)
    kc = torch.randn(B, Hkv, Lmax, D, generator=g, device="cuda", dtype=torch.float16)
    vc = torch.randn(B, Hkv, Lmax, D, generator=g, device="cuda", dtype=torch.float16)
    out = torch.zeros_like(q)
    kerns.flash_attn_decode(q, kc, vc, lens, out)
    err = chunked = 0.0
    for b in range(B):
        n = int(lens[b])
        s = (q[b].double().view(Hkv, group, D) @ kc[b].double().transpose(1, 2)) * (D ** -0.5 * 1.4426950408889634)
        s[..., n:] = -float("inf")
        v = vc[b].double()
        p = torch.exp2(s - s.amax(-1, keepdim=True))
        want = ((p / p.sum(-1, keepdim=True)) @ v).view(Hkv * group, 1, D)
        tiles = s.view(Hkv, group, Lmax // 512, 8, 4, 16)             # chunk, tile of the warp, warp, key
        ref = tiles.amax(-1).cummax(3).values.unsqueeze(-1)
        w = torch.exp2(tiles - ref).nan_to_num(0.0)                  # (chunks beyond the sequence)
        scale = torch.exp2(ref - s.amax(-1).view(Hkv, group, 1, 1, 1, 1))
        num = (w.half().double() * scale).view(Hkv, group, Lmax) @ v
        emu = (num / (w * scale).sum((2, 3, 4, 5)).unsqueeze(-1)).view(Hkv * group, 1, D).half().double()
        err += float(((out[b].double() - want) ** 2).sum())
        chunked += float(((emu - want) ** 2).sum())
    assert err ** 0.5 <= 1.01 * chunked ** 0.5, (err / chunked) ** 0.5


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("Hkv,group,D", [(1, 4, 128), (40, 9, 64)])
def test_scores_that_fall_or_rise_along_the_sequence(kerns, dtype, Hkv, group, D):
    """The reference maximum of a warp goes down by 2^4 per segment: scores that fall by more than that from segment to segment
    (the sums are then those of the first keys), that rise, and that stay within a segment's reach.  Tolerance: every weight
    and the result carry one 16-bit rounding, and scores of up to 1100 octaves some 2e-4 of a weight in 32 bits."""
    B, L = 3, 6000
    g = torch.Generator().manual_seed(D)
    q = torch.zeros(B, Hkv * group, 1, D)
    q[..., 0] = D ** 0.5
    kc = torch.randn(B, Hkv, L, D, generator=g) * 0.1
    at = torch.arange(L, dtype=torch.float32)
    kc[0, :, :, 0] = -at / 8                 # 11.5 octaves per 64 keys, down
    kc[1, :, :, 0] = (at - L) / 8            # and up
    kc[2, :, :, 0] = -at / 400
    vc = torch.randn(B, Hkv, L, D, generator=g) * 100
    q, kc, vc = q.to(dtype), kc.to(dtype), vc.to(dtype)
    lens = torch.tensor([L, L - 3, L - 7], dtype=torch.int32)
    got = run_decode(kerns, q, kc, vc, lens).float().cpu()
    want = O.attention_f64(q, kc, vc, lens=lens)
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    tol = (u + 3e-4) * O.attention_f64(q, kc, vc.abs(), lens=lens) + u * want.abs()
    assert ((got - want).abs() <= tol).all(), float(((got - want).abs() / tol).max())


@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("B,Hkv,Lmax", [(1, 1, 32768), (1, 3, 32768), (5, 1, 32768), (1, 5, 32768), (16, 1, 8192), (1, 1, 65552)])
def test_few_heads_over_a_long_cache(kerns, B, Hkv, Lmax, paged):
    """Both sides of the lines between clusters of 16 blocks, of 8, and chunks merged by a second kernel, as the library
    chooses them: full, ragged and empty sequences of a padded and of a paged cache."""
    D, group = 128, 2
    g = torch.Generator().manual_seed(B + Hkv)
    q = torch.randn(B, Hkv * group, 1, D, generator=g).half()
    kc = torch.randn(B, Hkv, Lmax, D, generator=g).half()
    vc = torch.randn(B, Hkv, Lmax, D, generator=g).half()
    lens = torch.tensor([Lmax, 0, Lmax // 2 + 3, 1, 700][:B] + [Lmax - 17 * i for i in range(5, B)], dtype=torch.int32)
    want = O.attention_f64(q, kc, vc, lens=lens)
    if not paged:
        got = run_decode(kerns, q, kc, vc, lens)
    else:
        page = 16
        per_seq = Lmax // page
        table = torch.randperm(B * per_seq, generator=g).to(torch.int32).view(B, per_seq)
        pools = []
        for x in (kc, vc):
            pool = torch.empty(B * per_seq, Hkv, page, D, dtype=x.dtype)
            pool[table.long().flatten()] = x.view(B, Hkv, per_seq, page, D).transpose(1, 2).reshape(B * per_seq, Hkv, page, D)
            pools.append(pool.cuda())
        got = torch.full(q.shape, float("nan"), dtype=q.dtype, device="cuda")
        kerns.flash_attn_decode_paged(q.cuda(), *pools, table.cuda(), lens.cuda(), got)
    check_close(got, want, f"{B}x{Hkv} heads, {Lmax} keys")
    assert torch.count_nonzero(got[lens == 0]) == 0
