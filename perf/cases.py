"""The attention calls that a user of this package makes, as cases that can be timed and compared.

A case is a dict of plain values:

  call      'module'  HyperAttention.forward on [B, H, n, d] tensors (and, with train, its backward through autograd)
            'core'    FastCoreAttention, the attention core of a ChatGLM2-style decoder block, on [n, B, H, d] tensors
            'host'    HostStream.forward_backward on pinned host tensors
  batch, heads, kv_heads, n, dim, dtype
  causal    decoder attention (recursive half-splits down to exact leaves) or bidirectional attention
  train     forward and backward, or the forward alone
  smooth    smooth_block=True
  sampling  'reference' (the first rows) or 'uniform' (importance-weighted draws)
  data      'clusters': queries and keys around 64 shared unit-norm centroids per head; 'normal': N(0, 1)

Every case uses the benchmark configurations' block_size 256, sample_size 256, 8 projections and min_seq_len 2048.
"""
import math

import torch

import hyperattention_b200 as ha
from hyperattention_b200.host import HostStream
from hyperattention_b200.llm import FastCoreAttention, chatglm2_config

BLOCK, SAMPLE, MIN_SEQ, BITS = 256, 256, 2048, 8
DTYPES = {'bf16': torch.bfloat16, 'fp16': torch.float16, 'fp32': torch.float32}
BASE = dict(call='module', batch=1, heads=32, kv_heads=32, n=4096, dim=64, dtype='bf16', causal=False, train=True, smooth=False,
            sampling='reference', data='normal')


def _case(**over):
    c = dict(BASE, **over)
    if 'kv_heads' not in over:
        c['kv_heads'] = c['heads']
    return c


def listed():
    return [
        # a short chat prompt through a patched decoder block: exact attention, two K/V heads; latency of one call
        _case(name='prompt_515', call='core', n=515, kv_heads=2, dim=128, causal=True, train=False),
        # shortest point of the sequence-length sweep, one training step of a bidirectional layer
        _case(name='layer_4k_train', n=4096),
        # the single-layer benchmark (configuration 1)
        _case(name='layer_131k_train', n=131072, data='clusters'),
        # the decoder benchmark (configuration 2), the largest case
        _case(name='decoder_131k_train', n=131072, causal=True, data='clusters'),
        # prefill of a decoder layer of ordinary length, output and log-sum-exp
        _case(name='decoder_16k_prefill', n=16384, causal=True, train=False, dtype='fp16'),
        # the attention of one block of the long-context decoder prefill (configuration 4), heads expanded by the caller
        _case(name='core_32k_prefill', call='core', n=32768, dim=128, causal=True, train=False),
        # fine-tuning a decoder with 128-wide heads, small batch
        _case(name='decoder_8k_d128_train', batch=2, heads=16, n=8192, dim=128, causal=True),
        # the sweep's smooth_block option
        _case(name='smooth_16k_train', n=16384, smooth=True),
        # importance-weighted uniform sampling
        _case(name='uniform_32k_train', heads=16, n=32768, sampling='uniform', data='clusters'),
        # a decoder sequence of odd length (padded by one row at the first split)
        _case(name='decoder_12287_train', heads=16, n=12287, causal=True),
        # single precision at the size of the correctness configuration (configuration 0)
        _case(name='layer_4k_fp32_train', heads=4, n=4096, dtype='fp32'),
        # tensors that live in host memory, streamed through the GPU
        _case(name='host_16k_train', call='host', n=16384),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['layer', 'layer', 'decoder', 'decoder', 'decoder', 'prefill', 'prefill', 'exact', 'core', 'core', 'smooth', 'uniform',
                       'fp32', 'host'])
    dtype = rng.choice(['bf16', 'bf16', 'bf16', 'fp16'])
    heads = rng.choice([4, 8, 12, 16, 24, 32])
    dim = rng.choice([64, 64, 128])
    data = rng.choice(['normal', 'clusters'])
    c = dict(heads=heads, dim=dim, dtype=dtype, data=data)
    # rows x width of the largest listed case
    most = 32 * 131072 * 64

    def split_length(top):
        """A decoder length: leaves of 1152 .. 2048 rows (a multiple of 128) doubled one to six times; at times one row short."""
        leaf, levels = 128 * rng.randint(9, 16), rng.randint(1, 6)
        while levels > 1 and (leaf << levels) > top:
            levels -= 1
        return (leaf << levels) - (1 if rng.random() < 0.25 else 0)

    if kind == 'layer':
        n = 128 * _log_int(rng, MIN_SEQ // 128, 1024)
        c['heads'] = min(heads, max(1, most // (n * dim)))
        return _case(**c, n=n, train=rng.random() < 0.7)
    if kind in ('decoder', 'prefill'):
        n = split_length(most // (heads * dim * (1 if dim == 64 else 2)))
        batch = rng.choice([1, 1, 2, 4])
        batch = batch if 2 * batch * heads * n * dim <= most else 1
        return _case(**c, batch=batch, n=n, causal=True, train=kind == 'decoder')
    if kind == 'exact':                      # short sequences of any length
        return _case(**c, batch=rng.choice([1, 2, 4, 8]), n=_log_int(rng, 64, MIN_SEQ - 1), causal=rng.random() < 0.7, train=rng.random() < 0.5)
    if kind == 'core':
        n = _log_int(rng, 64, MIN_SEQ) if rng.random() < 0.4 else split_length(40000)
        return _case(call='core', n=n, kv_heads=rng.choice([2, 32]), dim=128, dtype='bf16', causal=True, train=False, data='normal')
    if kind == 'smooth':
        return _case(**c, n=128 * _log_int(rng, MIN_SEQ // 128, 256), smooth=True, train=rng.random() < 0.7)
    if kind == 'uniform':
        return _case(**c, n=128 * _log_int(rng, MIN_SEQ // 128, 256), sampling='uniform', train=rng.random() < 0.7)
    if kind == 'fp32':
        return _case(heads=rng.choice([2, 4, 8]), dim=dim, dtype='fp32', n=128 * _log_int(rng, MIN_SEQ // 128, 64), train=rng.random() < 0.7)
    return _case(call='host', heads=heads, dtype=dtype, data=data, n=128 * _log_int(rng, MIN_SEQ // 128, 160))


def _inputs(c, seed):
    """q, k, v, do as [B, H, n, d] device tensors (k and v with kv_heads heads)."""
    g = torch.Generator(device='cuda').manual_seed(seed)
    B, H, Hk, n, d, dt = c['batch'], c['heads'], c['kv_heads'], c['n'], c['dim'], DTYPES[c['dtype']]

    def normal(h):
        return torch.randn(B, h, n, d, generator=g, device='cuda', dtype=torch.float32)

    if c['data'] == 'clusters':
        cent = torch.randn(B, H, 64, d, generator=g, device='cuda')
        cent = cent / cent.norm(dim=-1, keepdim=True)

        def near(h):
            a = torch.randint(0, 64, (B, h, n, 1), generator=g, device='cuda')
            return (cent[:, :h].gather(2, a.expand(-1, -1, -1, d)) + normal(h) * (0.3 / math.sqrt(d))).to(dt)
        q, k = near(H), near(Hk)
    else:
        q, k = normal(H).to(dt), normal(Hk).to(dt)
    return q, k, normal(Hk).to(dt), normal(H).to(dt)


def prepare(case, seed):
    c = case
    q, k, v, do = _inputs(c, seed)
    rng = torch.Generator().manual_seed(seed)
    opts = dict(lsh_num_projs=BITS, block_size=BLOCK, sample_size=SAMPLE, min_seq_len=MIN_SEQ, smooth_block=c['smooth'], rng=rng)
    if c['call'] == 'core':
        cfg = chatglm2_config(num_attention_heads=c['heads'], kv_channels=c['dim'], hidden_size=c['heads'] * c['dim'],
                              multi_query_group_num=c['kv_heads'])
        core = FastCoreAttention(cfg, 1, attn_method='hyper', grouped_kv=c['kv_heads'] != c['heads'], **opts).to(device='cuda', dtype=q.dtype)
        q, k, v = [t.permute(2, 0, 1, 3).contiguous() for t in (q, k, v)]       # a decoder block holds [n, B, heads, d]
        return dict(case=c, mod=core, q=q, k=k, v=v)
    mod = ha.HyperAttention(input_dim=c['dim'], sampling=c['sampling'], sample_seed=seed, **opts).to(device='cuda', dtype=q.dtype)
    if c['call'] == 'host':
        q, k, v, do = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t) for t in (q, k, v, do)]
        return dict(case=c, mod=mod, stream=HostStream(mod), q=q, k=k, v=v, do=do)
    if c['train']:
        q, k, v = [t.requires_grad_() for t in (q, k, v)]
    return dict(case=c, mod=mod, q=q, k=k, v=v, do=do)


def run(state):
    c, q, k, v = state['case'], state['q'], state['k'], state['v']
    if c['call'] == 'host':
        return state['stream'].forward_backward(q, k, v, state['do'], causal=c['causal'])
    if c['call'] == 'core':
        with torch.no_grad():
            return state['mod'](q, k, v, None)
    if not c['train']:
        with torch.no_grad():
            return state['mod'](q, k, v, causal=c['causal'], return_lse=True)
    o = state['mod'](q, k, v, causal=c['causal'])
    return (o.detach(),) + torch.autograd.grad(o, (q, k, v), state['do'])


def work(case):
    c = case
    B, H, Hk, n, d = c['batch'], c['heads'], c['kv_heads'], c['n'], c['dim']
    # (query, key) pairs of one head
    if c['causal']:
        pairs, span, spans = 0, n + (n > MIN_SEQ and n % 2), 1
        while span > MIN_SEQ:
            m = span // 2                                     # rectangle: second half against the first
            pairs += spans * m * (m if m < MIN_SEQ else BLOCK + SAMPLE)
            span, spans = m, 2 * spans
        pairs += spans * span * (span + 1) // 2
    else:
        pairs = n * (n if n < MIN_SEQ else BLOCK + SAMPLE)
    products = 7 if c['train'] or c['call'] == 'host' else 2   # of 2 d operations per pair: S, O | S, dP, dV, dK, dQ
    hashed = 2 * (H + Hk) * n * d * BITS if n > MIN_SEQ or (n == MIN_SEQ and not c['causal']) else 0
    es = 4 if c['dtype'] == 'fp32' else 2
    tensors = (2 * H + 2 * Hk) * es                            # q, k, v, o
    if products == 7:
        tensors += (2 * H + 2 * Hk) * es                       # do, dq, dk, dv
    nbytes = B * n * d * tensors
    if products == 2 and c['call'] == 'module':
        nbytes += B * H * n * 4                                # log-sum-exp
    return {'bytes': nbytes, 'flops': B * (2 * products * d * H * pairs + hashed)}


def tolerance(case):
    return {'rel': 2e-5} if case['dtype'] == 'fp32' else {'rel': 1e-2}
