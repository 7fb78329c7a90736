"""Padding rows of the sliding backward (a chunk of a key block has fewer queries than rows) see no column: not even one
whose key is infinite, which they would multiply with their zeros."""
import pytest
import torch

import recipe
from oracle import nsa_oracle as O
from util import assert_close_bf16

import native_sparse_attention_pytorch_b200 as nsa

pytestmark = pytest.mark.gpu


# (window, key): the index of a padding entry is 0xffffff, its first column 255 - window - 64 j in eight bits: 0 and 63 here
@pytest.mark.parametrize('window, at', [(255, 10), (255, 290), (512, 255)])
@pytest.mark.parametrize('d', [64, 128])
def test_an_infinite_key_that_every_query_gives_probability_zero(d, window, at):
    n, heads, kv_heads = 301, 8, 2                   # 32 queries per chunk
    q = recipe.randn((1, heads, n, d), 1)
    q[..., 3] = q[..., 3].abs() + 0.1
    k, v = (recipe.randn((1, kv_heads, n, d), s) for s in (2, 3))
    k[:, :, at, 3] = float('-inf')
    up = recipe.randn(q.shape, 4)
    q, k, v, up = (t.bfloat16() for t in (q, k, v, up))
    ref_in = [t.float().requires_grad_() for t in (q, k, v)]
    ref = O.sliding_attend(*ref_in, window, True)
    want = torch.autograd.grad(ref, ref_in[1:], up.float())
    ins = [t.to('cuda').requires_grad_() for t in (q, k, v)]
    out = nsa.sliding_window_attend(*ins, window, True, impl='sm100')
    assert_close_bf16(out, ref, 'out')
    for g, w, name in zip(torch.autograd.grad(out, ins[1:], up.to('cuda')), want, ('dk', 'dv')):
        assert w.isfinite().all()
        assert_close_bf16(g, w, name)
