"""The CUDA-core kernels of the compressed and the sliding branch at the edges of their tiles (8 queries, 32 keys) against the
oracle, and with a key that is not finite: a block of queries stages the keys of all of them, so a query must not meet the
one that only its neighbours see.  fp32 1e-4 relative, as every operator."""
import pytest
import torch

import recipe
from oracle import nsa_oracle as O
from util import assert_close_f32

import native_sparse_attention_pytorch_b200 as nsa

pytestmark = pytest.mark.gpu
DEV = 'cuda'


def gpu(*ts):
    return [t.to(DEV).requires_grad_() for t in ts]


@pytest.mark.parametrize('causal', [True, False])
@pytest.mark.parametrize('n, window, heads, kv_heads, d', [(1, 1, 1, 1, 64), (8, 32, 4, 2, 8), (9, 31, 8, 1, 64), (33, 24, 4, 4, 128),
                                                           (71, 33, 2, 1, 72), (40, 1, 16, 1, 16)])
def test_sliding_tiles(n, window, heads, kv_heads, d, causal):
    q = recipe.randn((2, heads, n, d), 1)
    k, v = (recipe.randn((2, kv_heads, n, d), s) for s in (2, 3))
    up = recipe.randn(q.shape, 4)
    ref_in = [t.clone().requires_grad_() for t in (q, k, v)]
    ref = O.sliding_attend(*ref_in, window, causal)
    want = torch.autograd.grad(ref, ref_in, up)
    ins = gpu(q, k, v)
    out = nsa.sliding_window_attend(*ins, window, causal)
    assert_close_f32(out, ref, 'out')
    for g, w, name in zip(torch.autograd.grad(out, ins, up.to(DEV)), want, ('dq', 'dk', 'dv')):
        assert_close_f32(g, w, name)


@pytest.mark.parametrize('n, stride, mem, heads, kv_heads, d', [(7, 2, 1, 1, 1, 64), (62, 2, 1, 8, 2, 64), (64, 2, 2, 4, 1, 128), (67, 1, 1, 2, 2, 24)])
def test_compressed_tiles(n, stride, mem, heads, kv_heads, d):
    ncb = n // stride
    q = recipe.randn((2, heads, n, d), 1)
    k, v = (recipe.randn((2, kv_heads, ncb, d), s) for s in (2, 3))
    m = recipe.randn((2, kv_heads, mem, d), 4)
    up = recipe.randn(q.shape, 5)
    ref_in = [t.clone().requires_grad_() for t in (q, k, v)]
    ref, _ = O.compressed_attend(*ref_in, m[0], m[1], stride, True)
    want = torch.autograd.grad(ref, ref_in, up)
    ins = gpu(q, k, v)
    joint = [torch.cat((m[j].to(DEV).expand(2, -1, -1, -1), ins[1 + j]), dim=-2) for j in range(2)]
    out, _ = nsa.compressed_attend(ins[0], *joint, mem, stride, True, sel_heads=kv_heads)
    assert_close_f32(out, ref, 'out')
    for g, w, name in zip(torch.autograd.grad(out, ins, up.to(DEV)), want, ('dq', 'dk', 'dv')):
        assert_close_f32(g, w, name)


@pytest.mark.parametrize('bad', [float('nan'), float('inf')])
def test_a_key_that_is_not_finite_stays_with_the_queries_that_see_it(bad):
    n, window, at = 45, 5, 21                   # queries at .. at + window see it, inside two blocks of queries
    q, k, v, up = (recipe.randn((1, 2, n, 64), s) for s in (1, 2, 3, 4))
    clean = gpu(q, k, v)
    want = nsa.sliding_window_attend(*clean, window, True)
    want_dq, = torch.autograd.grad(want, clean[:1], up.to(DEV))
    k, v = k.clone(), v.clone()
    k[:, :, at, 3] = bad
    v[:, :, at, 5] = bad
    dirty = gpu(q, k, v)
    out = nsa.sliding_window_attend(*dirty, window, True)
    dq, dk = torch.autograd.grad(out, dirty[:2], up.to(DEV))
    others = torch.ones(n, dtype=torch.bool)
    others[at:at + window + 1] = False
    assert torch.equal(out[:, :, others], want[:, :, others])
    assert torch.equal(dq[:, :, others], want_dq[:, :, others])
    assert not out[:, :, at].isfinite().all()
    assert dk[:, :, :at - window].isfinite().all() and dk[:, :, at + window + 1:].isfinite().all()
