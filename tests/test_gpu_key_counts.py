"""CUDA-core kernels of the compressed and the sliding branch on either side of the lines between a warp per query and tiles that
the queries of a block share (by the number of keys, the heads per KV head and dim_head), against the oracle."""
import pytest
import torch

import recipe
from oracle import nsa_oracle as O
from util import assert_close_f32

import native_sparse_attention_pytorch_b200 as nsa

pytestmark = pytest.mark.gpu


def check(want_of, got_of, tensors, up):
    ref_in = [t.clone().requires_grad_() for t in tensors]
    ref = want_of(*ref_in)
    want = torch.autograd.grad(ref, ref_in, up)
    ins = [t.to('cuda').requires_grad_() for t in tensors]
    out = got_of(*ins)
    assert_close_f32(out, ref, 'out')
    for g, w, name in zip(torch.autograd.grad(out, ins, up.to('cuda')), want, ('dq', 'dk', 'dv')):
        assert_close_f32(g, w, name)


# windows of 10 | 11 keys; eight heads per KV head (19 | 20 keys); sixteen (8 | 9), with blocks that fill the GPU, and of 128 (23 | 24)
@pytest.mark.parametrize('batch, n, window, heads, kv_heads, d, causal', [
    (2, 45, 9, 4, 2, 64, True), (2, 45, 10, 4, 2, 64, True), (2, 45, 4, 4, 4, 40, False), (2, 45, 5, 4, 4, 40, False), (1, 3, 0, 2, 1, 64, True),
    (1, 50, 18, 8, 1, 64, True), (1, 50, 19, 8, 1, 64, True), (1, 50, 9, 8, 1, 128, False), (1, 50, 10, 8, 1, 128, False),
    (1, 60, 7, 16, 1, 64, True), (1, 60, 8, 12, 1, 64, True), (2, 593, 10, 16, 1, 16, True), (1, 60, 9, 16, 1, 128, True),
    (1, 60, 10, 16, 1, 128, True), (4, 297, 22, 16, 1, 128, True), (4, 297, 23, 16, 1, 128, True)])
def test_sliding(batch, n, window, heads, kv_heads, d, causal):
    q, up = (recipe.randn((batch, heads, n, d), s) for s in (1, 4))
    k, v = (recipe.randn((batch, kv_heads, n, d), s) for s in (2, 3))
    check(lambda *t: O.sliding_attend(*t, window, causal), lambda *t: nsa.sliding_window_attend(*t, window, causal), (q, k, v), up)


# (positions, stride, memory slots): two keys | three; heads of 128 with sixteen per KV head: eleven | twelve
@pytest.mark.parametrize('n, stride, mem, heads, kv_heads, d', [(9, 8, 1, 4, 2, 64), (19, 8, 1, 4, 2, 64), (9, 8, 2, 4, 4, 24), (5, 8, 1, 2, 1, 64),
                                                                (47, 4, 1, 1, 1, 128), (650, 60, 1, 16, 1, 128), (650, 59, 1, 16, 1, 128)])
def test_compressed(n, stride, mem, heads, kv_heads, d):
    q, up = (recipe.randn((2, heads, n, d), s) for s in (1, 5))
    k, v = (recipe.randn((2, kv_heads, n // stride, d), s) for s in (2, 3))
    m = recipe.randn((2, kv_heads, mem, d), 4)
    def ours(q, k, v):
        joint = [torch.cat((m[j].to('cuda').expand(2, -1, -1, -1), t), dim=-2) for j, t in enumerate((k, v))]
        return nsa.compressed_attend(q, *joint, mem, stride, True, sel_heads=kv_heads)[0]
    check(lambda *t: O.compressed_attend(*t, m[0], m[1], stride, True)[0], ours, (q, k, v), up)


@pytest.mark.parametrize('bad', [float('nan'), float('inf')])
def test_a_key_that_is_not_finite_stays_with_the_queries_that_see_it(bad):
    """As in test_gpu_dense_tiles.py, with a window of shared tiles."""
    n, window, at = 75, 13, 31
    q, k, v, up = (recipe.randn((1, 2, n, 64), s) for s in (1, 2, 3, 4))
    def run(k, v):
        ins = [t.to('cuda').requires_grad_() for t in (q, k, v)]
        out = nsa.sliding_window_attend(*ins, window, True)
        return out, *torch.autograd.grad(out, ins[:2], up.to('cuda'))
    want, want_dq, _ = run(k, v)
    k, v = k.clone(), v.clone()
    k[:, :, at, 3] = bad
    v[:, :, at, 5] = bad
    out, dq, dk = run(k, v)
    others = torch.ones(n, dtype=torch.bool)
    others[at:at + window + 1] = False
    assert torch.equal(out[:, :, others], want[:, :, others]) and torch.equal(dq[:, :, others], want_dq[:, :, others])
    assert not out[:, :, at].isfinite().all()
    assert dk[:, :, :at - window].isfinite().all() and dk[:, :, at + window + 1:].isfinite().all()
