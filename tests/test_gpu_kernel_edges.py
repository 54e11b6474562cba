"""The attention kernels where their tiles, lists of key tiles and loaders change shape, forward and backward, against the oracle."""
import math
import os

import pytest
import torch

from oracle import hyper_oracle as O

pytestmark = pytest.mark.gpu

T = lambda x: x.transpose(1, 2)
# Outputs and log-sum-exps, gradients: twice what roundings to 16 bits make of them.  Outputs: weights and result, 2^-9 / sqrt(3) each in bf16, with one
# more a merge: 1.6e-3 to 2.6e-3; gradients: weights, dS, output and result: 2.3e-3 to 2.9e-3.  fp32: the reference's merges have
# an eps in their logarithm (2^-23 a merge, which the gradients' exponentials repeat for every row).
TOL = {torch.float32: (2e-6, 5e-5), torch.bfloat16: (5e-3, 6e-3), torch.float16: (6.5e-4, 7.5e-4)}


def rel(a, b):
    a, b = a.detach().float().cpu(), b.detach().float().cpu()
    return ((a - b).norm() / b.norm().clamp_min(1e-30)).item()


def _check(got, want, dtype):
    t_out, t_grad = TOL[dtype]
    errs = [rel(g, w) for g, w in zip(got, want)]
    assert max(errs[:2]) < t_out and max(errs[2:], default=0.) < t_grad, errs


@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float32])
@pytest.mark.parametrize('cfg', [
    # B, H, n, d, dv, block, sample, smooth
    (1, 2, 128, 64, 64, 256, 128, False),      # a single query tile, a window cut to one tile
    (2, 1, 640, 64, 64, 128, 128, False),      # one-tile blocks: the two tiles of a pair have windows of their own
    (1, 3, 896, 64, 64, 384, 0, False),        # three-tile blocks: pairs that straddle two blocks; nothing sampled
    (1, 2, 1152, 128, 128, 384, 128, False),   # ... at head dim 128, last block cut
    (1, 2, 896, 64, 64, 512, 384, True),       # smooth windows of four tiles, an odd number of query tiles
    (1, 2, 640, 128, 128, 256, 256, True),
    (1, 1, 512, 64, 128, 256, 128, False),     # dv != d, both ways
    (1, 1, 512, 128, 64, 256, 128, False),
    (1, 160, 256, 64, 64, 256, 256, False),    # more items than CTAs: every ring wraps
    (1, 84, 512, 128, 128, 256, 256, False),
])
def test_hyper_pattern_edges(dtype, cfg):
    import hyperattention_b200 as ha
    from hyperattention_b200 import _lib as L
    B, H, n, d, dv, block, sample, smooth = cfg
    torch.manual_seed(70)
    q, k, do = torch.randn(B, H, n, d).to(dtype), torch.randn(B, H, n, d).to(dtype), torch.randn(B, H, n, dv).to(dtype)
    v = torch.randn(B, H, n, dv).to(dtype)
    qi, ki = [torch.sort(torch.randint(0, 16, (B, H, n)), dim=2, stable=True)[1] for _ in range(2)]
    qg, kg, vg = [t.cuda().requires_grad_() for t in (q, k, v)]
    o, lse = ha.hyper_attn_func(T(qg), T(kg), T(vg), T(qi.cuda()), T(ki.cuda()), block, sample, None, smooth, None,
                                L.FLAG_BWD_REF_SMOOTH if smooth else 0)
    T(o).backward(do.cuda())
    h = slice(0, 2) if H > 4 else slice(None)           # heads are independent: two of many are enough
    qc, kc, vc = [t[:, h].float().requires_grad_() for t in (q, k, v)]
    ow, lw = O.hyper_attn_func(T(qc), T(kc), T(vc), T(qi[:, h]), T(ki[:, h]), block, sample, None, smooth, None, False)
    T(ow).backward(do[:, h].float())
    _check((T(o)[:, h], lse[:, h], qg.grad[:, h], kg.grad[:, h], vg.grad[:, h]), (T(ow), lw, qc.grad, kc.grad, vc.grad), dtype)


@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float32])
@pytest.mark.parametrize('n', [1, 63, 64, 65, 127, 128, 129, 191, 257, 385, 700])
@pytest.mark.parametrize('causal', [True, False])
@pytest.mark.parametrize('d', [64, 128])
def test_exact_attention_lengths(dtype, n, causal, d):
    import hyperattention_b200 as ha
    torch.manual_seed(71)
    B, H = 2, 2
    q, k, v, do = [torch.randn(B, n, H, d).to(dtype) for _ in range(4)]
    qg, kg, vg = [t.cuda().requires_grad_() for t in (q, k, v)]
    o, lse = ha.flash_attn_func(qg, kg, vg, None, causal, None)
    o.backward(do.cuda())
    qc, kc, vc = [t.float().requires_grad_() for t in (q, k, v)]
    ow, lw = O.flash_attn_func(qc, kc, vc, None, causal, None)
    ow.backward(do.float())
    g = 3 if n > 1 else 1          # one key: dq and dk are zero but for rounding
    _check((o, lse[:, :, :n]) + (vg.grad, qg.grad, kg.grad)[:g], (ow, lw[:, :, :n]) + (vc.grad, qc.grad, kc.grad)[:g], dtype)


@pytest.mark.parametrize('nq,nk', [(300, 77), (77, 300), (128, 1000)])
def test_exact_attention_unequal_lengths_and_layouts(nq, nk):
    """fewer / more keys than queries; K/V heads expanded with stride 0, which no tensor map can describe; sequence-major tensors"""
    import hyperattention_b200 as ha
    torch.manual_seed(72)
    B, H, d = 2, 3, 64
    q = torch.randn(B, nq, H, d).bfloat16()
    k, v = [torch.randn(B, nk, 1, d).bfloat16().expand(-1, -1, H, -1) for _ in range(2)]
    o, lse = ha.flash_attn_func(q.cuda(), k.cuda()[:, :, :1].expand(-1, -1, H, -1), v.cuda()[:, :, :1].expand(-1, -1, H, -1))
    ow, lw = O.flash_attn_func(q.float(), k.float(), v.float())
    _check((o, lse[:, :, :nq]), (ow, lw[:, :, :nq]), torch.bfloat16)
    qs, ks, vs = [t.contiguous().permute(1, 0, 2, 3).contiguous().cuda().permute(1, 0, 2, 3) for t in (q, k, v)]     # [n, B, H, d] memory
    o2, lse2 = ha.flash_attn_func(qs, ks, vs)
    assert torch.equal(o2, o) and torch.equal(lse2, lse)


def test_rows_that_see_no_key_of_a_tile():
    """weighted sampling in which whole sampled tiles are dropped for a query tile (every sampled key lies in its window)"""
    import hyperattention_b200 as ha
    torch.manual_seed(73)
    B, H, n, d = 1, 2, 512, 64
    q, k, v = [torch.randn(B, H, n, d).bfloat16() for _ in range(3)]
    qi, ki = [torch.sort(torch.randint(0, 4, (B, H, n)), dim=2, stable=True)[1] for _ in range(2)]
    sidx = ki[:, :, :128].contiguous()                  # the first window tile's keys: dropped for the first block, kept for the second
    o, lse = ha.hyper_attn_func(T(q.cuda()), T(k.cuda()), T(v.cuda()), T(qi.cuda()), T(ki.cuda()), 256, 128, None, False, sidx.cuda(), 0, True)
    ow, lw = O.hyper_attn_func(T(q.float()), T(k.float()), T(v.float()), T(qi), T(ki), 256, 128, None, False, sidx, False, True)
    _check((o, lse), (ow, lw), torch.bfloat16)


@pytest.mark.parametrize('n,dtype,train', [(1023, torch.bfloat16, True), (2047, torch.float32, True), (1535, torch.bfloat16, False)])
def test_causal_odd_length_runs_the_single_call_schedule(n, dtype, train):
    """an odd length is padded by one zero row and takes the single-call schedule: against the oracle, which pads as the reference does"""
    import hyperattention_b200 as ha
    torch.manual_seed(74)
    B, H, d = 1, 2, 64
    proj = torch.randn(1, 1, d, 8).to(dtype).float()
    q, k, v, do = [torch.randn(B, H, n, d).to(dtype) for _ in range(4)]
    mod = ha.HyperAttention(input_dim=d, block_size=256, sample_size=256, min_seq_len=512)
    mod.lsh.proj_dir.copy_(proj)
    mod = mod.to(device='cuda', dtype=dtype)
    assert mod._regular_causal(n)
    qg, kg, vg = [t.cuda().requires_grad_(train) for t in (q, k, v)]
    o, lse = mod(qg, kg, vg, causal=True, return_lse=True)
    orc = O.HyperAttentionOracle(proj, 256, 256, 512, False)
    qc, kc, vc = [t.float().requires_grad_() for t in (q, k, v)]
    ow, lw = orc(qc, kc, vc, causal=True, return_lse=True)
    assert o.shape == ow.shape and lse.shape == lw.shape
    if not train:
        return _check((o, lse), (ow, lw), dtype)
    o.backward(do.cuda())
    ow.backward(do.float())
    _check((o, lse, qg.grad, kg.grad, vg.grad), (ow, lw, qc.grad, kc.grad, vc.grad), dtype)


@pytest.mark.parametrize('causal', [True, False])
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float32])
def test_strided_tensors_match_contiguous_ones(causal, dtype):
    """[n, B, H, d] and [B, n, H, d] tensors as [B, H, n, d] views: same results, gradients included; the output keeps the order"""
    import hyperattention_b200 as ha
    torch.manual_seed(75)
    B, H, n, d = 2, 3, 1024, 64
    mod = ha.HyperAttention(input_dim=d, min_seq_len=256, sample_size=128, rng=torch.Generator().manual_seed(5)).to(device='cuda', dtype=dtype)
    base = [torch.randn(B, H, n, d, device='cuda').to(dtype) for _ in range(4)]
    res = []
    for order in ((0, 1, 2, 3), (2, 0, 1, 3), (0, 2, 1, 3)):
        inv = tuple(order.index(i) for i in range(4))
        q, k, v, do = [t.permute(order).contiguous().permute(inv) for t in base]
        q, k, v = [t.requires_grad_() for t in (q, k, v)]
        o, lse = mod(q, k, v, causal=causal, return_lse=True)
        if dtype == torch.bfloat16:
            assert o.stride() == q.stride()
        with torch.no_grad():
            o2 = mod(q, k, v, causal=causal)
        res.append((o.detach(), lse.detach(), o2) + torch.autograd.grad(o, (q, k, v), do))
    for r in res[1:]:
        assert torch.equal(r[0], res[0][0]) and torch.equal(r[1], res[0][1]) and torch.equal(r[2], res[0][2])
        for a, b in zip(r[3:], res[0][3:]):
            assert rel(a, b) < 1e-3


@pytest.mark.parametrize('rows,n,span,off,length,bits', [
    (3, 2047, 2047, 0, 2047, 8), (3, 2048, 2048, 0, 2048, 8), (2, 2049, 2049, 0, 2049, 7), (2, 4097, 4097, 0, 4097, 8),
    (1, 8192, 8192, 0, 8192, 8), (2, 8193, 8193, 0, 8193, 1), (1, 70001, 70001, 0, 70001, 8), (150, 1, 1, 0, 1, 8),
    (2, 12288, 4096, 2048, 2048, 8), (2, 4100, 2050, 1025, 1025, 8), (2, 3000, 3000, 0, 3000, 10),
])
def test_segment_sort_at_the_edges_of_its_chunks(rows, n, span, off, length, bits):
    """lengths around the chunk sizes, segments that start inside a span, more key bits than a chunk counts: the stable order"""
    import hyperattention_b200 as ha
    codes = torch.randint(0, 1 << bits, (rows, n), generator=torch.Generator().manual_seed(76), dtype=torch.int32)
    idx = ha.seg_sort(codes.cuda(), bits, span=span, seg_off=off, seg_len=length).cpu()
    segs = codes.view(rows * (n // span), span)[:, off:off + length]
    assert torch.equal(idx.view(segs.shape).long(), torch.sort(segs, dim=1, stable=True)[1])


@pytest.mark.parametrize('dtype,d,n,causal', [(torch.bfloat16, 64, 333, True), (torch.float16, 128, 257, True),
                                              (torch.bfloat16, 64, 130, False), (torch.float32, 64, 200, True)])
def test_exact_attention_with_shared_key_value_heads(dtype, d, n, causal):
    """fewer key/value heads than query heads, never expanded: against the oracle on expanded ones"""
    import hyperattention_b200 as ha
    torch.manual_seed(77)
    B, H, Hk = 2, 6, 2
    q, do = [torch.randn(B, n, H, d).to(dtype) for _ in range(2)]
    k, v = [torch.randn(B, n, Hk, d).to(dtype) for _ in range(2)]
    qg, kg, vg = [t.cuda().requires_grad_() for t in (q, k, v)]
    o, lse = ha.flash_attn_func(qg, kg, vg, None, causal)
    o.backward(do.cuda())
    qc, kc, vc = [t.float().requires_grad_() for t in (q, k, v)]
    s = (qc.transpose(1, 2) @ kc.repeat_interleave(H // Hk, 2).permute(0, 2, 3, 1)) * d ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(n, n, dtype=torch.bool).triu(1), float('-inf'))
    ow = (s.softmax(-1) @ vc.repeat_interleave(H // Hk, 2).transpose(1, 2)).transpose(1, 2)
    ow.backward(do.float())
    _check((o, lse[:, :, :n], qg.grad, kg.grad, vg.grad), (ow, s.logsumexp(-1), qc.grad, kc.grad, vc.grad), dtype)


@pytest.mark.parametrize('rows,n,S', [(3, 1000, 256), (1, 128, 128), (5, 131072, 384)])
def test_uniform_sample_draws_the_oracles_rows(rows, n, S):
    """one row per stratum, whole numbers equal to the oracle's, at sizes that divide evenly and that do not"""
    from hyperattention_b200 import ops
    base = (2024 * 0x9E3779B97F4A7C15 + 3 * 0xD1B54A32D192ED03) & ((1 << 64) - 1)
    got = ops.uniform_sample(rows, n, S, base, 'cuda').cpu().long()
    assert torch.equal(got, torch.as_tensor(O.uniform_sample_idx(2024, 3, rows, S, n)).long())


@pytest.mark.parametrize('n,causal,H', [(1000, False, 1), (2176, True, 1), (384, True, 80)])
def test_exact_backward_by_key_tiles(n, causal, H):
    """head dim 128: many key tiles (shorter sequences: test_exact_attention_lengths), more of them than CTAs"""
    import hyperattention_b200 as ha
    torch.manual_seed(78)
    q, k, v, do = [torch.randn(1, n, H, 128).bfloat16() for _ in range(4)]
    qg, kg, vg = [t.cuda().requires_grad_() for t in (q, k, v)]
    o, lse = ha.flash_attn_func(qg, kg, vg, None, causal)
    o.backward(do.cuda())
    qc, kc, vc = [t.float().requires_grad_() for t in (q, k, v)]
    s = T(qc) @ T(kc).transpose(2, 3) * 128 ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(n, n, dtype=torch.bool).triu(1), float('-inf'))
    ow = T(s.softmax(-1) @ T(vc))
    ow.backward(do.float())
    _check((o, lse[:, :, :n], qg.grad, kg.grad, vg.grad), (ow, s.logsumexp(-1), qc.grad, kc.grad, vc.grad), torch.bfloat16)


@pytest.mark.parametrize('direct', [None, False])
@pytest.mark.parametrize('n,block,S,smooth,weighted', [(896, 384, 128, False, False), (512, 256, 128, False, True), (768, 256, 256, True, True), (512, 512, 0, True, False)])
def test_hyper_backward_by_key_tiles(n, block, S, smooth, weighted, direct):
    """head dim 128: key tiles that one query tile of a pair meets, weighted samples with dropped slots, smooth windows.  direct=False (fp32
    accumulators) is what the kernel by key tiles takes in all of these; the default leaves those without whole blocks to the earlier one."""
    from hyperattention_b200 import _lib as L, ops
    torch.manual_seed(79)
    B, H, d = 1, 2, 128
    q, k, v, do = [torch.randn(B, H, n, d).bfloat16() for _ in range(4)]
    qi, ki = [torch.sort(torch.randint(0, 4, (B, H, n)), dim=2, stable=True)[1] for _ in range(2)]
    sidx = ki[:, :, 64:64 + S].contiguous() if weighted else None
    qc, kc, vc = [t.float().requires_grad_() for t in (q, k, v)]
    ow, lw = O.hyper_attn_func(T(qc), T(kc), T(vc), T(qi), T(ki), block, S, None, smooth, sidx, False, weighted)
    T(ow).backward(do.float())
    qg, kg, vg, og, dg = [T(t.cuda()) for t in (q, k, v, T(ow).detach().bfloat16(), do)]
    qr, kr = [t.cuda().int().view(B * H, n) for t in (qi, ki)]
    sr = sidx.cuda().int().view(B * H, S) if weighted else None
    delta = T((og.float() * dg.float()).sum(-1)).contiguous()
    flags = (L.FLAG_SMOOTH | L.FLAG_BWD_REF_SMOOTH) if smooth else 0
    weights = ops.sample_weights(kr, sr, n, block, S, smooth) if weighted else None
    got = ops.hyper_bwd(qg, kg, vg, qr, kr, sr, og, lw.detach().cuda().contiguous(), dg, delta, block, S, d ** -0.5, flags, weights, direct)
    errs = [rel(T(g), w) for g, w in zip(got, (qc.grad, kc.grad, vc.grad))]
    assert max(errs) < TOL[torch.bfloat16][1], errs


@pytest.mark.parametrize('block,smooth', [(256, True), (384, False), (512, True)])
def test_causal_training_at_head_dim_128(block, smooth):
    """the kernel by key tiles in the causal schedule, which adds to fp32 accumulators: smooth windows of two and four tiles, blocks of three
    tiles (cut at the ends of the rectangles)"""
    import hyperattention_b200 as ha
    torch.manual_seed(91)
    n, d = 2048, 128
    proj = torch.randn(1, 1, d, 8).bfloat16().float()
    q, k, v, do = [torch.randn(1, 2, n, d).bfloat16() for _ in range(4)]
    mod = ha.HyperAttention(input_dim=d, block_size=block, sample_size=128, min_seq_len=512, smooth_block=smooth)
    mod.lsh.proj_dir.copy_(proj)
    mod = mod.to(device='cuda', dtype=torch.bfloat16)
    assert mod._regular_causal(n)
    qg, kg, vg = [t.cuda().requires_grad_() for t in (q, k, v)]
    o, lse = mod(qg, kg, vg, causal=True, return_lse=True)
    o.backward(do.cuda())
    qc, kc, vc = [t.float().requires_grad_() for t in (q, k, v)]
    ow, lw = O.HyperAttentionOracle(proj, block, 128, 512, smooth)(qc, kc, vc, causal=True, return_lse=True)
    ow.backward(do.float())
    _check((o, lse, qg.grad, kg.grad, vg.grad), (ow, lw, qc.grad, kc.grad, vc.grad), torch.bfloat16)


@pytest.mark.parametrize('dtype,B,n,rows,shapes', [(torch.bfloat16, 2, 1023, 1024, ((3, 64), (3, 64), (1, 128))), (torch.float16, 1, 5, 6, ((2, 20),)),
                                                   (torch.float32, 3, 130, 133, ((4, 7), (2, 8))), (torch.bfloat16, 1, 1, 2, ((1, 8), (1, 2), (5, 1), (1, 9)))])
def test_padding_rows(dtype, B, n, rows, shapes):
    """aligned rows, odd widths, strided sources, one to four tensors: bytes equal to torch's padding"""
    from hyperattention_b200 import ops
    ts = [torch.randn(n, B, h, w, device='cuda').to(dtype).permute(1, 2, 0, 3) for h, w in shapes]
    for t, o in zip(ts, ops._padded(ts, rows)):
        assert o.is_contiguous() and torch.equal(o, torch.nn.functional.pad(t, (0, 0, 0, rows - n)))


@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float16])
@pytest.mark.parametrize('count,off', [(1, 0), (7, 0), (8, 0), (100003, 0), (4096, 1)])
def test_cast_from_f32_at_odd_counts(dtype, count, off):
    """whole chunks, a tail, less than a chunk, an unaligned source: torch's rounding"""
    from hyperattention_b200 import _lib as L, ops
    src = torch.randn(count + off, device='cuda')[off:]
    dst = torch.full((count + 1,), 7., dtype=dtype, device='cuda')
    L.check(L.load().ha_cast_from_f32(src.data_ptr(), dst.data_ptr(), count, ops._DT[dtype], ops._stream()), 'ha_cast_from_f32')
    assert torch.equal(dst[:count], src.to(dtype)) and dst[count] == 7.


def test_host_streams_hand_their_streams_on():
    """a triple of streams serves one HostStream at a time and then the next one"""
    import hyperattention_b200 as ha
    from hyperattention_b200.host import HostStream
    mod = ha.HyperAttention(input_dim=64, min_seq_len=128, sample_size=128, rng=torch.Generator().manual_seed(3)).to(device='cuda', dtype=torch.bfloat16)
    q, k, v = [torch.randn(1, 4, 512, 64, dtype=torch.bfloat16).pin_memory() for _ in range(3)]
    a, b = HostStream(mod), HostStream(mod)
    oa, ob = a.forward(q, k, v), b.forward(k, q, v)
    torch.cuda.synchronize()
    first, other = a._streams, b._streams
    assert not set(first) & set(other)
    del a
    c = HostStream(mod)
    oc = c.forward(q, k, v)
    torch.cuda.synchronize()
    assert c._streams == first and torch.equal(oa, oc) and not torch.equal(oa, ob)


@pytest.mark.parametrize('hyper', [False, True])
@pytest.mark.parametrize('d', [64, 128])
def test_the_largest_weight_of_a_row_is_exact(d, hyper):
    """Keys past the first 64 score log(1 + 2^-8) more than those before: weights against the row's maximum are 1 and 0.9961, which a
    bf16 P holds (to 2e-5), so that a constant V comes back.  Against an earlier, smaller reference they are 1.0039, half a bf16 step
    above 1."""
    import hyperattention_b200 as ha
    n, scale = 1024, math.log1p(2 ** -8)
    q, k, v = torch.zeros(1, n, 2, d), torch.zeros(1, n, 2, d), torch.ones(1, n, 2, d)
    q[..., 0] = 1
    k[:, 64:, :, 0] = 1
    q, k, v = [t.bfloat16().cuda() for t in (q, k, v)]
    if hyper:
        idx = torch.arange(n, device='cuda').view(1, n, 1).expand(1, n, 2)
        o, lse = ha.hyper_attn_func(q, k, v, idx, idx, 256, 256, scale)
    else:
        o, lse = ha.flash_attn_func(q, k, v, None, False, scale)
        assert rel(lse, torch.full((1, 2, n), math.log(64 + 960 * math.exp(scale)))) < 1e-6
    assert torch.equal(o, torch.ones_like(o))


@pytest.mark.parametrize('bad', [float('nan'), float('inf')])
@pytest.mark.parametrize('dtype,d,causal', [(torch.bfloat16, 64, False), (torch.float16, 64, True), (torch.bfloat16, 128, False)])
def test_a_key_that_is_not_finite_shows_at_every_position(dtype, d, causal, bad):
    """A NaN key, or one whose score is +infinity, at each of sixteen neighbouring positions (the exponentials of some are polynomials): the
    rows that see it are not finite, the others are."""
    import hyperattention_b200 as ha
    torch.manual_seed(81)
    n, H, first = 256, 16, 70
    q, k, v = [torch.randn(1, n, H, d) for _ in range(3)]
    q[..., 0] = 1
    for h in range(H):
        k[0, first + h, h, 0] = bad
    o, _ = ha.flash_attn_func(*[t.to(dtype).cuda() for t in (q, k, v)], None, causal)
    sees = torch.arange(n)[:, None] >= first + torch.arange(H) if causal else torch.ones(n, H, dtype=torch.bool)
    finite = torch.isfinite(o[0].cpu())
    assert torch.equal(finite.all(-1), ~sees) and torch.equal(finite.any(-1), ~sees)


@pytest.mark.parametrize('n,causal', [(130, False), (193, True), (1, False)])
def test_absent_query_rows_of_many_short_sequences(n, causal):
    """head dim 64, more sequences than CTAs, the last query tile nearly empty: its absent rows add nothing to any key's gradient, in the
    first item of a CTA (their slots hold nothing yet) and in later ones (they hold another sequence's)"""
    import hyperattention_b200 as ha
    torch.manual_seed(82)
    q, k, v, do = [torch.randn(2, n, 200, 64).bfloat16() for _ in range(4)]
    qg, kg, vg = [t.cuda().requires_grad_() for t in (q, k, v)]
    o, lse = ha.flash_attn_func(qg, kg, vg, None, causal)
    o.backward(do.cuda())
    qc, kc, vc = [t.cuda().float().requires_grad_() for t in (q, k, v)]
    s = T(qc) @ T(kc).transpose(2, 3) * 64 ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device='cuda').triu(1), float('-inf'))
    ow = T(s.softmax(-1) @ T(vc))
    ow.backward(do.cuda().float())
    for t, w in ((o, ow), (vg.grad, vc.grad)) + (((qg.grad, qc.grad), (kg.grad, kc.grad)) if n > 1 else ()):
        per_head = (t.float() - w).norm(dim=(1, 3)) / w.norm(dim=(1, 3))
        assert per_head.max() < 2e-2, per_head.max()      # (bf16 rounds to 2^-9; gradients are products of three rounded factors)


@pytest.mark.parametrize('keep,stride,off', [(0, 68, 0), (0, 64, 1), (1, 64, 1), (1, 72, 8)])
def test_causal_outputs_that_vector_stores_do_not_fit(keep, stride, off):
    """C entry point: output rows 136 bytes apart, or starting one element into an allocation (no 16-byte boundaries: the merges run in the
    epilogues), and aligned ones with a gap; against the module's own contiguous call"""
    import ctypes as C
    import hyperattention_b200 as ha
    from hyperattention_b200 import _lib as L, ops
    torch.manual_seed(83)
    B, H, n, d = 1, 2, 1024, 64
    q, k, v = [torch.randn(B, H, n, d, device='cuda').bfloat16() for _ in range(3)]
    mod = ha.HyperAttention(input_dim=d, min_seq_len=512, sample_size=128, rng=torch.Generator().manual_seed(6)).to(device='cuda', dtype=torch.bfloat16)
    want, lse_want = mod(q, k, v, causal=True, return_lse=True)
    mem = torch.full((off + B * H * n * stride + 64,), 7., device='cuda', dtype=torch.bfloat16)
    o, lse = mem[off:off + B * H * n * stride].view(B, H, n, stride)[..., :d], torch.empty(B, H, n, device='cuda')
    p, lib = L.CausalParams(), L.load()
    p.dtype, p.B, p.H, p.n, p.d, p.dv, p.levels, p.block_size, p.sample_size, p.lsh_bits = L.BF16, B, H, n, d, d, 1, 256, 128, 8
    p.keep_parts, p.min_seq_len, p.scale = keep, 512, d ** -0.5
    p.q, p.k, p.v, p.o, p.lse, p.proj = [t.data_ptr() for t in (q, k, v, o, lse, mod.lsh.proj_f32())]
    saved = ops._buffer(p, 'saved', lib.ha_causal_saved_bytes(C.byref(p)), 'cuda')
    scratch = ops._buffer(p, 'scratch', lib.ha_causal_scratch_bytes(C.byref(p), 0), 'cuda')
    st = (C.c_int64 * 15)(*q.stride()[:3], *k.stride()[:3], *v.stride()[:3], *o.stride()[:3], 0, 0, 0)
    L.check(lib.ha_causal_fwd_strided(C.byref(p), st, ops._stream()), 'ha_causal_fwd_strided')
    assert rel(o, want) < 1e-2 and rel(lse, lse_want[..., 0]) < 1e-4        # (bf16 weights on one side, fp32 ones on the other)
    gaps = torch.ones_like(mem, dtype=torch.bool)
    gaps[off:off + B * H * n * stride].view(B, H, n, stride)[..., :d] = False
    assert (mem[gaps] == 7).all()
    del saved, scratch


def test_first_calls_from_many_threads():
    """the first launches of a process, made by eight host threads at once on streams of their own: every thread's results are one thread's"""
    import subprocess
    import sys
    code = '''
import threading, torch, hyperattention_b200 as ha
torch.manual_seed(0)
ts = [torch.randn(1, 2, 1024, 64, device='cuda').bfloat16() for _ in range(4)]
mod = ha.HyperAttention(input_dim=64, min_seq_len=256, sample_size=128, rng=torch.Generator().manual_seed(1)).to(device='cuda', dtype=torch.bfloat16)
torch.cuda.synchronize()
out, gate = [None] * 8, threading.Barrier(8)
def work(i):
    with torch.cuda.stream(torch.cuda.Stream()):
        q, k, v = [t.clone().requires_grad_() for t in ts[:3]]
        gate.wait()
        o = mod(q, k, v, causal=i % 2 == 0)
        out[i] = (o.detach(),) + torch.autograd.grad(o, (q, k, v), ts[3])
        torch.cuda.current_stream().synchronize()
threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
[t.start() for t in threads]
[t.join() for t in threads]
for i in range(2, 8):
    assert torch.equal(out[i][0], out[i % 2][0]), i
    for a, b in zip(out[i][1:], out[i % 2][1:]):
        assert (a.float() - b.float()).norm() < 1e-3 * b.float().norm(), i      # (fp32 additions in no fixed order, rounded to bf16)
ha.check_device_status()
'''
    subprocess.run([sys.executable, '-c', code], check=True, timeout=120, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


@pytest.mark.parametrize('n,causal', [(300, True), (512, False), (1024, True)])
@pytest.mark.parametrize('kind', ['tensor', 'cuda', 'numpy'])
def test_a_scale_that_changes_between_calls(n, causal, kind):
    """a 0-dim tensor or array as the scale, rewritten in place: every call takes its value of that moment, forward and backward"""
    import numpy as np
    import hyperattention_b200 as ha
    torch.manual_seed(84)
    mod = ha.HyperAttention(input_dim=64, min_seq_len=512, sample_size=128, rng=torch.Generator().manual_seed(7)).to(device='cuda', dtype=torch.bfloat16)
    q, k, v = [torch.randn(1, 2, n, 64, device='cuda').bfloat16().requires_grad_() for _ in range(3)]
    scale = np.array(0.) if kind == 'numpy' else torch.zeros((), device='cuda' if kind == 'cuda' else 'cpu')
    for value in (0.0625, 0.25):
        scale[...] = value
        got, want = mod(q, k, v, scale=scale, causal=causal), mod(q, k, v, scale=value, causal=causal)
        with torch.no_grad():
            assert torch.equal(mod(q, k, v, scale=scale, causal=causal), want)
        assert torch.equal(got, want)
        for a, b in zip(torch.autograd.grad(got, (q, k, v), v), torch.autograd.grad(want, (q, k, v), v)):
            assert rel(a, b) < 1e-3        # (fp32 additions in no fixed order, rounded to bf16)


def test_projection_copy_is_there_for_other_streams():
    """the fp32 copy of the projection is made behind other work of one stream; a call on another stream right after it uses the finished one"""
    import hyperattention_b200 as ha
    torch.manual_seed(85)
    q, k, v = [torch.randn(1, 2, 1024, 64, device='cuda').bfloat16() for _ in range(3)]
    new = lambda: ha.HyperAttention(input_dim=64, min_seq_len=256, sample_size=128, rng=torch.Generator().manual_seed(8)).to(device='cuda', dtype=torch.bfloat16)
    want, mod, a, b = new()(q, k, v), new(), torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        stale = torch.full((64, 8), float('nan'), device='cuda')      # (what the copy's memory holds until it is written)
    torch.cuda.synchronize()
    del stale
    with torch.cuda.stream(a):
        torch.cuda._sleep(200_000_000)
        mod(q, k, v)
    with torch.cuda.stream(b):
        got = mod(q, k, v)
    torch.cuda.synchronize()
    assert torch.equal(got, want)


def test_projection_copy_of_a_capture_stays_in_its_graph():
    """a module whose first call is captured: eager calls before a replay have a copy of their own"""
    import hyperattention_b200 as ha
    torch.manual_seed(86)
    q, k, v = [torch.randn(1, 2, 1024, 64, device='cuda').bfloat16() for _ in range(3)]
    new = lambda: ha.HyperAttention(input_dim=64, min_seq_len=256, sample_size=128, rng=torch.Generator().manual_seed(8)).to(device='cuda', dtype=torch.bfloat16)
    want, mod, graph = new()(q, k, v), new(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = mod(q, k, v)
    assert torch.equal(mod(q, k, v), want)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(captured, want)


def test_status_word_is_there_for_other_streams(monkeypatch):
    """the device's status word is made behind other work of one stream; a call on another stream right after it does not take what its memory
    held for a failure"""
    import hyperattention_b200 as ha
    from hyperattention_b200 import ops
    torch.manual_seed(87)
    q, k, v = [torch.randn(1, 300, 2, 64, device='cuda').bfloat16() for _ in range(3)]
    want, a, b = ha.flash_attn_func(q, k, v, None, True)[0], torch.cuda.Stream(), torch.cuda.Stream()
    monkeypatch.setattr(ops, '_STATUS', {})
    monkeypatch.setattr(ops, '_STATUS_RAW', {})
    with torch.cuda.stream(a):
        stale = torch.ones(1, dtype=torch.int32, device='cuda')
    torch.cuda.synchronize()
    del stale
    with torch.cuda.stream(a):
        torch.cuda._sleep(200_000_000)
        first = ha.flash_attn_func(q, k, v, None, True)[0]
    with torch.cuda.stream(b):
        got = ha.flash_attn_func(q, k, v, None, True)[0]
    torch.cuda.synchronize()
    assert torch.equal(got, want) and torch.equal(first, want)
    ha.check_device_status()


@pytest.mark.parametrize('n,causal', [(300, True), (512, False), (1024, True)])
def test_forward_mode_and_transforms_are_refused(n, causal):
    """there is no rule for tangents or batches: an error, also where no input requires a gradient; other tensors in a dual level pass"""
    import torch.autograd.forward_ad as fwd
    import hyperattention_b200 as ha
    torch.manual_seed(88)
    mod = ha.HyperAttention(input_dim=64, min_seq_len=512, sample_size=128, rng=torch.Generator().manual_seed(9)).to(device='cuda', dtype=torch.bfloat16)
    q, k, v = [torch.randn(1, 2, n, 64, device='cuda').bfloat16() for _ in range(3)]
    call = lambda t: mod(t, k, v, causal=causal)
    want = call(q)
    with torch.no_grad(), fwd.dual_level():
        with pytest.raises(NotImplementedError):
            call(fwd.make_dual(q, torch.ones_like(q)))
        assert torch.equal(call(q), want)
    for run in (lambda: torch.func.jvp(call, (q,), (torch.ones_like(q),)), lambda: torch.func.vmap(call)(q[None])):
        with pytest.raises(RuntimeError):
            run()


@pytest.mark.parametrize('m,causal', [(200, True), (72, False), (330, True)])
@pytest.mark.parametrize('d', [64, 128])
def test_segments_of_any_length_keep_to_themselves(d, m, causal):
    """C entry points: two segments a head that end inside a tile; the second one's rows are all NaN, the first one's results are not"""
    import ctypes as C
    from hyperattention_b200 import _lib as L, ops
    torch.manual_seed(89)
    H, n, lib = 3, 2 * m, L.load()
    q, k, v, do = [torch.randn(1, n, H, d, device='cuda').bfloat16() for _ in range(4)]
    for t in (q, k, v, do):
        t[:, m:] = float('nan')
    o, lse = torch.empty_like(q), torch.empty(1, H, n, device='cuda')
    acc, delta = torch.zeros(3, 1, H, n, d, device='cuda'), torch.empty(1, H, n, device='cuda')
    p = ops._flash_params(q, k, v, o, lse, causal, d ** -0.5, 0)
    p.segs_per_head, p.span, p.m_q, p.m_k = 2, m, m, m
    L.check(lib.ha_attn_fwd(C.byref(p), ops._stream()), 'ha_attn_fwd')
    L.check(lib.ha_delta(o.data_ptr(), *ops._bhn(o), do.data_ptr(), *ops._bhn(do), 1, H, n, d, L.BF16, delta.data_ptr(), ops._stream()), 'ha_delta')
    p.d_o, p.delta, p.dq_acc, p.dk_acc, p.dv_acc = do.data_ptr(), delta.data_ptr(), acc[0].data_ptr(), acc[1].data_ptr(), acc[2].data_ptr()
    p.do_sb, p.do_sh, p.do_sn = ops._bhn(do)
    L.check(lib.ha_attn_bwd(C.byref(p), ops._stream()), 'ha_attn_bwd')
    ref = [t[:, :m].float().cpu().requires_grad_() for t in (q, k, v)]
    ow, lw = O.flash_attn_func(*ref, None, causal)
    ow.backward(do[:, :m].float().cpu())
    _check((o[:, :m], lse[:, :, :m]) + tuple(T(a[:, :, :m]) for a in acc), (ow, lw[:, :, :m]) + tuple(t.grad for t in ref), torch.bfloat16)
    assert torch.isnan(o[:, m:]).all()


@pytest.mark.parametrize('d', [64, 128])
def test_fp32_sums_are_made_of_short_chains(d):
    """exact attention in fp32 against 64 bits.  A chain of L roundings of 2^-24 is off by about 2^-24 / sqrt(3) sqrt(L / 2): 2.2e-7 where tiles of
    64 are summed by themselves and then added (L = 64 + 16 here), 7.7e-7 where a sum runs over all 1000 keys.  Two products in a row: 3.1e-7."""
    import hyperattention_b200 as ha
    torch.manual_seed(90)
    q, k, v, do = [torch.randn(1, 1000, 4, d, device='cuda') for _ in range(4)]
    qg, kg, vg = [t.clone().requires_grad_() for t in (q, k, v)]
    o, _ = ha.flash_attn_func(qg, kg, vg)
    o.backward(do)
    qe, ke, ve = [t.double().requires_grad_() for t in (q, k, v)]
    oe = T((T(qe) @ T(ke).transpose(2, 3) * d ** -0.5).softmax(-1) @ T(ve))
    oe.backward(do.double())
    err = [((a.double() - b).norm() / b.norm()).item() for a, b in ((o, oe), (qg.grad, qe.grad), (kg.grad, ke.grad), (vg.grad, ve.grad))]
    assert max(err) < 4.5e-7, err


@pytest.mark.parametrize('d', [64, 128])
@pytest.mark.parametrize('n,H', [(600, 5), (512, 230), (640, 250), (330, 300)])
def test_causal_items_are_dealt_out_once_each(d, n, H):
    """exact causal attention with fewer items than CTAs, whole rounds of segments and a rest (even and odd numbers of pairs), more than two segments
    a CTA (the segments' own order): every head's outputs and gradients"""
    import hyperattention_b200 as ha
    torch.manual_seed(95)
    q, k, v, do = [torch.randn(1, n, H, d, device='cuda').bfloat16() for _ in range(4)]
    qg, kg, vg = [t.clone().requires_grad_() for t in (q, k, v)]
    o, lse = ha.flash_attn_func(qg, kg, vg, None, True)
    o.backward(do)
    qc, kc, vc = [T(t).double().requires_grad_() for t in (q, k, v)]
    s = (qc @ kc.transpose(2, 3) * d ** -0.5).masked_fill(torch.ones(n, n, dtype=torch.bool, device='cuda').triu(1), float('-inf'))
    ow = s.softmax(-1) @ vc
    ow.backward(T(do).double())
    for got, want, tol in ((o, ow, 0), (qg.grad, qc.grad, 1), (kg.grad, kc.grad, 1), (vg.grad, vc.grad, 1)):
        err = (T(got).double() - want).flatten(2).norm(dim=2) / want.flatten(2).norm(dim=2)
        assert err.max() < TOL[torch.bfloat16][tol], (err.max(), err.argmax())
    assert (lse[:, :, :n].double() - s.logsumexp(-1)).abs().max() < 1e-4


@pytest.mark.parametrize('dtype,d', [(torch.bfloat16, 64), (torch.bfloat16, 128), (torch.float32, 64)])
@pytest.mark.parametrize('n', [1, 515, 640])
def test_exact_causal_call_without_a_gradient(dtype, d, n):
    """short causal calls that keep nothing for a backward hand [batch, heads, rows, width] tensors to the kernel as they are: fewer K/V heads than query
    heads, tensors that lie as [n, B, heads, d] in memory, rows padded and not; the same bits as the call that keeps them"""
    import hyperattention_b200 as ha
    torch.manual_seed(96)
    B, H, Hk = 2, 6, 2
    q, k, v = [torch.randn(n, B, h, d, device='cuda').to(dtype).permute(1, 2, 0, 3) for h in (H, Hk, Hk)]
    mod = ha.HyperAttention(input_dim=d, min_seq_len=2048, rng=torch.Generator().manual_seed(10)).to(device='cuda', dtype=dtype)
    with torch.no_grad():
        o, lse = mod(q, k, v, causal=True, return_lse=True)
        assert torch.equal(mod(q, k, v, causal=True), o)
        assert torch.equal(mod(*[t.contiguous() for t in (q, k, v)], causal=True), o)
    og, lg = mod(*[t.detach().requires_grad_() for t in (q, k, v)], causal=True, return_lse=True)
    assert torch.equal(o, og) and torch.equal(lse, lg) and o.stride() == og.stride() and lse.shape == (B, H, -(-n // 128) * 128)
    s = (q.double() @ k.double().repeat_interleave(H // Hk, 1).transpose(2, 3) * d ** -0.5).masked_fill(torch.ones(n, n, dtype=torch.bool, device='cuda').triu(1), float('-inf'))
    assert rel(o, s.softmax(-1) @ v.double().repeat_interleave(H // Hk, 1)) < TOL[dtype][0]
    assert (lse[:, :, :n].double() - s.logsumexp(-1)).abs().max() < 1e-4 and not lse[:, :, n:].any()


@pytest.mark.parametrize('causal,smooth,dtype,d', [(True, False, torch.bfloat16, 64), (True, False, torch.bfloat16, 128), (False, False, torch.bfloat16, 64),
                                                   (False, True, torch.float16, 64), (False, False, torch.bfloat16, 128), (True, False, torch.float32, 64)])
def test_captured_step_repeats_the_eager_one(causal, smooth, dtype, d):
    """forward alone, forward and backward, recorded as graphs (a side stream and its join, zero-fills and launches that overlap the one before) and replayed
    on other inputs, several times in a row"""
    import hyperattention_b200 as ha
    torch.manual_seed(97)
    n = 2048
    mod = ha.HyperAttention(input_dim=d, min_seq_len=512, sample_size=128, smooth_block=smooth, rng=torch.Generator().manual_seed(11)).to(device='cuda', dtype=dtype)
    new = lambda: [torch.randn(1, 3, n, d, device='cuda').to(dtype) for _ in range(4)]
    held = new()
    q, k, v = [t.requires_grad_() for t in held[:3]]
    do = held[3]

    def forward():
        with torch.no_grad():
            return mod(q, k, v, causal=causal, return_lse=True)

    def step():
        o = mod(q, k, v, causal=causal)
        return (o.detach(),) + torch.autograd.grad(o, (q, k, v), do)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        forward(), step()
    torch.cuda.current_stream().wait_stream(side)
    graphs = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graphs[0]):
        kept = forward()
    with torch.cuda.graph(graphs[1]):
        grads = step()
    for times in (1, 3):
        with torch.no_grad():
            for t, x in zip(held, new()):
                t.copy_(x)
        for _ in range(times):
            for g in graphs:
                g.replay()
        torch.cuda.synchronize()
        for got, want in zip(kept, forward()):
            assert torch.equal(got, want)
        want = step()
        assert torch.equal(grads[0], want[0])
        for got, w in zip(grads[1:], want[1:]):       # (fp32 additions in no fixed order, rounded to 16 bits)
            assert rel(got, w) < (1e-3 if dtype != torch.float32 else 1e-6)
