"""The work this package is measured on: what a user's program asks of it, through its public entry points.

Four kinds of calls:
  attend    `native_sparse_attend`, forward and backward: the selected-block operator on its own
  train     one `SparseAttention` layer, forward and backward: input gradient and the flat parameter gradient
  prefill   one layer over a prompt without gradients, returning the cache that decoding starts from
  generate  some decoding steps of one layer from such a cache, each step handing its cache to the next

Sizes come from the configurations of bench.py, from the tests, or are generic; all inputs and weights are synthetic.
Keys, queries and compressed keys are of unit size, as in the operator benchmark (N(0,1)), so that attention is neither
uniform nor one-hot and the block selection has something to choose."""
import math

import torch

import native_sparse_attention_pytorch_b200 as nsa

DEV = 'cuda'
DTYPES = {'bf16': torch.bfloat16, 'fp32': torch.float32}

# the three-branch settings of the long configurations, and of the small example (window and blocks of a few tokens)
LONG = dict(cbs=32, stride=16, block=64, window=512)
BYTES = dict(cbs=16, stride=8, block=16, window=32)
README = dict(cbs=4, stride=2, block=4, window=2)


def _attend(name, batch, seq, heads, kv_heads, d, nsel, dtype='bf16', block=64):
    return dict(name=name, kind='attend', dtype=dtype, batch=batch, seq=seq, heads=heads, kv_heads=kv_heads, d=d,
                block=block, nsel=nsel)


def _layer(kind, name, batch, seq, dim, heads, kv_heads, d, nsel, sizes, dtype='bf16', causal=True, diff_topk=False,
           shared=True, steps=0):
    c = dict(name=name, kind=kind, dtype=dtype, batch=batch, seq=seq, dim=dim, heads=heads, kv_heads=kv_heads, d=d,
             nsel=nsel, causal=causal, diff_topk=diff_topk, shared=shared, **sizes)
    if kind == 'generate':
        c['steps'] = steps
    return c


def listed():
    return [
        # the operator: a short sequence where launches and host work count; a ragged length in the head size and
        # grouping of long-context models; the kernel benchmark
        _attend('attend_small', 1, 1024, 8, 2, 64, 4),
        _attend('attend_ragged_d128', 1, 3001, 16, 2, 128, 8),
        _attend('attend_large', 4, 8192, 32, 4, 64, 16),
        # the README example: non-causal, fp32, 31 tokens -- the smallest training step
        _layer('train', 'train_readme', 2, 31, 512, 8, 8, 64, 2, README, dtype='fp32', causal=False),
        # a byte-level language model trained in fp32 with short blocks and a differentiable top-k
        _layer('train', 'train_bytes_diff_topk', 4, 512, 512, 8, 4, 64, 4, BYTES, dtype='fp32', diff_topk=True),
        # bf16 training: a small layer, the language model's layer on a ragged batch, the full-layer benchmark
        _layer('train', 'train_small', 1, 1024, 256, 4, 2, 64, 4, dict(LONG, window=128)),
        _layer('train', 'train_lm_ragged', 3, 4997, 512, 8, 4, 64, 16, LONG),
        _layer('train', 'train_large', 2, 16384, 1024, 16, 4, 64, 16, LONG),
        # prompts: an ordinary one of odd length, and the long-context configuration (64 / 8 heads of 128)
        _layer('prefill', 'prefill_ragged', 2, 3333, 1024, 16, 4, 64, 16, LONG),
        _layer('prefill', 'prefill_long', 1, 65536, 4096, 64, 8, 128, 16, LONG),
        # decoding: a chat-sized cache of one user, and long caches of a small batch
        _layer('generate', 'generate_short', 1, 300, 512, 8, 4, 64, 4, LONG, steps=16),
        _layer('generate', 'generate_long', 4, 32768, 2048, 16, 2, 128, 16, LONG, steps=8),
    ]


def _log_int(rng, lo, hi):
    """Spread over the logarithm of the range, both ends included."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(['attend', 'attend', 'train', 'train', 'train_short', 'prefill', 'generate'])
    if kind == 'attend':
        heads, kv = rng.choice([(8, 2), (16, 4), (32, 4), (16, 2), (8, 4), (4, 4)])
        seq = _log_int(rng, 256, 8192)
        batch = rng.randint(1, max(1, min(4, 16384 // seq)))
        c = _attend('', batch, seq, heads, kv, rng.choice([64, 128]), rng.randint(2, 16))
    elif kind == 'train':
        dim, heads, kv, d = rng.choice([(256, 4, 2, 64), (512, 8, 4, 64), (1024, 16, 4, 64), (1024, 16, 2, 64),
                                        (1024, 8, 2, 128)])
        seq = _log_int(rng, 256, 16384)
        batch = rng.randint(1, max(1, min(8, 32768 // seq)))
        c = _layer('train', '', batch, seq, dim, heads, kv, d, rng.randint(2, 16), dict(LONG, window=rng.choice([128, 256, 512])))
    elif kind == 'train_short':
        heads, kv = rng.choice([(8, 8), (8, 4), (8, 2)])
        sizes = rng.choice([README, BYTES])
        seq = _log_int(rng, 24, 1024)
        batch = rng.randint(1, max(1, min(8, 4096 // seq)))
        causal = rng.random() < 0.75
        c = _layer('train', '', batch, seq, 512, heads, kv, 64, rng.randint(1, 4), sizes, dtype=rng.choice(['fp32', 'fp32', 'bf16']),
                   causal=causal, diff_topk=causal and rng.random() < 0.4, shared=rng.random() < 0.75)
    elif kind == 'prefill':
        dim, heads, kv, d = rng.choice([(512, 8, 4, 64), (1024, 16, 4, 64), (2048, 16, 2, 128), (4096, 32, 4, 128)])
        seq = _log_int(rng, 256, 65536)
        batch = rng.randint(1, max(1, min(4, 16384 // seq)))
        c = _layer('prefill', '', batch, seq, dim, heads, kv, d, 16, LONG)
    else:
        dim, heads, kv, d = rng.choice([(512, 8, 4, 64), (512, 8, 8, 64), (1024, 16, 4, 64), (2048, 16, 2, 128)])
        seq = _log_int(rng, 64, 32768)
        batch = rng.randint(1, max(1, min(16, 131072 // seq)))
        c = _layer('generate', '', batch, seq, dim, heads, kv, d, rng.choice([4, 8, 16]), LONG,
                   dtype=rng.choice(['bf16', 'bf16', 'bf16', 'fp32']) if seq <= 4096 else 'bf16', steps=rng.randint(4, 24))
    del c['name']
    return c


# ---- what a program has in hand ------------------------------------------------------------------------------------

def _blocks(batch, kv_heads, seq, block, nsel, gen):
    """Top-k over seeded N(0,1) block scores, past blocks only (the own block is always attended): indices and mask."""
    nb = -(-seq // block)
    k = min(nsel, nb)
    idx = torch.empty(batch, kv_heads, seq, k, dtype=torch.int64, device=DEV)
    mask = torch.empty(batch, kv_heads, seq, k, dtype=torch.bool, device=DEV)
    own = torch.arange(seq, device=DEV) // block
    past = torch.arange(nb, device=DEV)[None, :] < own[:, None]
    for b in range(batch):
        scores = torch.randn(kv_heads, seq, nb, device=DEV, generator=gen).masked_fill_(~past, -1e9)
        top, at = scores.topk(k, dim=-1)
        idx[b], mask[b] = at, top > -1e8
    return idx, mask


def _build(c, gen):
    """A layer whose weights are of the sizes training leaves them at: unit queries, keys, values and compressed rows,
    gates that depend on the token, memory slots and intra-block positions that are not zero."""
    with torch.device(DEV):
        layer = nsa.SparseAttention(
            dim=c['dim'], dim_head=c['d'], heads=c['heads'], kv_heads=c['kv_heads'], causal=c['causal'],
            sliding_window_size=c['window'], compress_block_size=c['cbs'], compress_block_sliding_stride=c['stride'],
            selection_block_size=c['block'], num_selected_blocks=c['nsel'], use_diff_topk=c['diff_topk'],
            query_heads_share_selected_kv=c['shared'], use_triton_kernel=True)

    def normal(p, std):
        p.copy_(torch.randn(p.shape, device=DEV, generator=gen) * std)

    with torch.no_grad():
        for name, p in layer.named_parameters():
            if name == 'norm.weight':
                normal(p, 0.1)
                p.add_(1.)
            elif name in ('compress_mem_kv', 'k_intrablock_positions', 'v_intrablock_positions'):
                normal(p, 0.5)
            elif name.endswith('bias'):
                normal(p, 0.5 if name.startswith('to_strategy_combine') else 0.1)
            elif name.endswith('compress.3.weight'):      # behind a ReLU that halves the second moment
                normal(p, (p.shape[-1] / 2) ** -0.5)
            else:
                normal(p, p.shape[-1] ** -0.5)
    return layer.to(DTYPES[c['dtype']])


def prepare(case, seed):
    c = case
    gen = torch.Generator(DEV).manual_seed(seed)
    dt = DTYPES[c['dtype']]

    def randn(*shape):
        return torch.randn(shape, device=DEV, generator=gen).to(dt)

    if c['kind'] == 'attend':
        q = randn(c['batch'], c['heads'], c['seq'], c['d']).requires_grad_()
        k = randn(c['batch'], c['kv_heads'], c['seq'], c['d']).requires_grad_()
        v = randn(c['batch'], c['kv_heads'], c['seq'], c['d']).requires_grad_()
        idx, mask = _blocks(c['batch'], c['kv_heads'], c['seq'], c['block'], c['nsel'], gen)
        return dict(kind='attend', block=c['block'], q=q, k=k, v=v, idx=idx, mask=mask, dout=randn(*q.shape))

    layer = _build(c, gen)
    if c['kind'] == 'train':
        x = randn(c['batch'], c['seq'], c['dim']).requires_grad_()
        return dict(kind='train', layer=layer, x=x, params=list(layer.parameters()), dout=randn(*x.shape))
    layer.requires_grad_(False)
    x = randn(c['batch'], c['seq'], c['dim'])
    if c['kind'] == 'prefill':
        return dict(kind='prefill', layer=layer, x=x)
    with torch.no_grad():
        _, cache = layer(x, return_cache=True)
    return dict(kind='generate', layer=layer, cache=cache,
                tokens=[randn(c['batch'], 1, c['dim']) for _ in range(c['steps'])])


# ---- one pass ------------------------------------------------------------------------------------------------------

def run(state):
    s = state
    if s['kind'] == 'attend':
        out = nsa.native_sparse_attend(s['q'], s['k'], s['v'], s['block'], s['idx'], s['mask'])
        dq, dk, dv = torch.autograd.grad(out, (s['q'], s['k'], s['v']), s['dout'])
        return out, dq, dk, dv
    if s['kind'] == 'train':
        out = s['layer'](s['x'])
        dx, *grads = torch.autograd.grad(out, [s['x'], *s['params']], s['dout'])
        # one flat gradient, as the data-parallel loop reduces it
        return dict(out=out, dx=dx, grads=torch.cat([g.reshape(-1) for g in grads]))
    with torch.no_grad():
        if s['kind'] == 'prefill':
            return s['layer'](s['x'], return_cache=True)
        cache, outs = s['cache'], []
        for token in s['tokens']:
            out, cache = s['layer'](token, cache=cache, return_cache=True)
            outs.append(out)
        return outs, cache


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def _selected_pairs(seq, block, nsel, causal=True):
    """(query, key) pairs of the selected branch of one (batch, query head)."""
    if not causal:
        return seq * (min(nsel, max(1, seq // block)) * block + block)
    i = torch.arange(seq, dtype=torch.int64)
    return int((block * torch.clamp(i // block, max=nsel) + i % block + 1).sum())


def _layer_pairs(c, seq):
    """(query, key) pairs of the three branches of one (batch, query head)."""
    ncb = seq // c['stride']
    if not c['causal']:
        return seq * (ncb + 1) + _selected_pairs(seq, c['block'], c['nsel'], False) + seq * min(seq, 2 * c['window'] + 1)
    i = torch.arange(seq, dtype=torch.int64)
    compressed = int((i // c['stride'] + 1).sum())
    sliding = int(torch.clamp(i + 1, max=c['window'] + 1).sum())
    return compressed + sliding + _selected_pairs(seq, c['block'], c['nsel'])


def _layer_parameters(c):
    """(parameters of the projections, of the two compress networks, of the rest)."""
    h, hkv, d, dim = c['heads'], c['kv_heads'], c['d'], c['dim']
    proj = dim * (h + 2 * hkv) * d + h * d * dim + dim * 3 * h
    width = c['cbs'] * d
    return proj, 2 * (width * width + width * d + width + d), dim + 3 * h + 2 * hkv * d + 2 * hkv * c['cbs'] * d


def work(case):
    c = case
    el = 2 if c['dtype'] == 'bf16' else 4
    b, n, h, hkv, d = c['batch'], c['seq'], c['heads'], c['kv_heads'], c['d']
    if c['kind'] == 'attend':
        k = min(c['nsel'], -(-n // c['block']))
        qs, kv, sel = b * h * n * d * el, 2 * b * hkv * n * d * el, b * hkv * n * k * 9
        return dict(bytes=qs * 4 + kv * 2 + sel, flops=14 * d * b * h * _selected_pairs(n, c['block'], k))
    proj, comp, rest = _layer_parameters(c)
    ncb, params = n // c['stride'], (proj + comp + rest) * el
    if c['kind'] == 'train':
        gemm = 6 * b * (n * proj + hkv * ncb * (comp // 2) * 2)
        return dict(bytes=2 * params + 4 * b * n * c['dim'] * el, flops=gemm + 14 * d * b * h * _layer_pairs(c, n))
    cache = 2 * b * hkv * (n + ncb) * d * el
    if c['kind'] == 'prefill':
        gemm = 2 * b * (n * proj + hkv * ncb * (comp // 2) * 2)
        return dict(bytes=params + 2 * b * n * c['dim'] * el + cache, flops=gemm + 4 * d * b * h * _layer_pairs(c, n))
    # a decoding step reads the compressed cache, the selected blocks and the window; the weights of the projections
    keys = ncb + 1 + min(c['nsel'], n // c['block']) * c['block'] + c['block'] + min(n, c['window'] + 1)
    step = (proj + rest) * el + 2 * b * c['dim'] * el + 2 * b * hkv * keys * d * el
    return dict(bytes=c['steps'] * step, flops=c['steps'] * (2 * b * proj + 4 * d * b * h * keys))


def tolerance(case):
    """fp32 is computed in fp32: sums of a few thousand terms, some through atomics.  bf16: inputs, probabilities and
    results carry 8 significant bits; a layer chains several such roundings, and its flat gradient mixes all of them."""
    if case['dtype'] == 'fp32':
        return dict(rel=1e-4)
    return dict(rel=1e-2 if case['kind'] == 'attend' else 2e-2)
