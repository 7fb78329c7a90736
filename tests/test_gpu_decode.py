"""The native decoding step (three launches, caches that grow in place) against the same layer run module by module:
a forward hook on a submodule makes the layer take that path."""
import pytest
import torch

import recipe
from util import assert_close_bf16, assert_close_f32

from native_sparse_attention_pytorch_b200 import SparseAttention

pytestmark = pytest.mark.gpu
DEV = 'cuda'


def build(dtype, heads, kv_heads, d, dim=256, stride=16, nsel=4, window=100, norm=True):
    layer = SparseAttention(dim=dim, dim_head=d, heads=heads, kv_heads=kv_heads, causal=True, sliding_window_size=window,
                            compress_block_size=2 * stride, compress_block_sliding_stride=stride, selection_block_size=64,
                            num_selected_blocks=nsel, norm=norm, use_triton_kernel=True)
    recipe.fill_weights(layer, seed=3)
    return layer.to(DEV).to(dtype).requires_grad_(False)


def steps(layer, tokens, cache):
    outs = []
    for i in range(tokens.shape[1]):
        out, cache = layer(tokens[:, i:i + 1], cache=cache, return_cache=True)
        outs.append(out)
    return torch.cat(outs, dim=1), cache


def flat(cache):
    (k, v), ((ck, cv), (rk, rv)) = cache
    return k, v, ck, cv, rk, rv


# batch (one token row to more than the projection kernels take), group size, head size, cache length: no compressed block
# yet, one tile, several tiles per warp; a head size without a tensor form
CASES = [(1, 4, 4, 64, 3, torch.bfloat16), (2, 8, 2, 64, 300, torch.bfloat16), (3, 16, 1, 128, 1100, torch.bfloat16),
         (17, 4, 2, 64, 200, torch.bfloat16), (2, 6, 2, 40, 150, torch.bfloat16), (9, 8, 8, 64, 500, torch.bfloat16),
         (2, 8, 4, 64, 130, torch.float32), (18, 2, 1, 128, 90, torch.float32)]


@pytest.mark.parametrize('case', CASES)
def test_native_steps_equal_the_module_by_module_steps(case):
    b, hq, hkv, d, n, dtype = case
    layer = build(dtype, hq, hkv, d)
    x = recipe.randn((b, n, 256), 5).to(dtype).to(DEV)
    tokens = recipe.randn((b, 20, 256), 6).to(dtype).to(DEV)
    with torch.no_grad():
        _, cache = layer(x, return_cache=True)
        got, got_cache = steps(layer, tokens, cache)
        hook = layer.combine_heads.register_forward_hook(lambda *_: None)
        want, want_cache = steps(layer, tokens, cache)
        hook.remove()
    close = assert_close_f32 if dtype == torch.float32 else assert_close_bf16
    close(got, want.float().cpu(), 'outputs')
    for g, w, name in zip(flat(got_cache), flat(want_cache), ('keys', 'values', 'ck', 'cv', 'window k', 'window v')):
        assert g.shape == w.shape and g.dtype == w.dtype, name
        close(g, w.float().cpu(), name)


def test_continuations_of_one_cache_do_not_disturb_each_other():
    layer = build(torch.bfloat16, 8, 2, 64)
    x = recipe.randn((2, 200, 256), 5).bfloat16().to(DEV)
    a, b = (recipe.randn((2, 40, 256), s).bfloat16().to(DEV) for s in (6, 7))
    with torch.no_grad():
        _, cache = layer(x, return_cache=True)
        base, mid = steps(layer, a[:, :5], cache)
        out_a, cache_a = steps(layer, a[:, 5:], mid)               # grows in place
        kept = [t.clone() for t in flat(cache_a)]
        out_b, cache_b = steps(layer, b, mid)                      # another continuation while the first is alive
        assert all(torch.equal(t, k) for t, k in zip(flat(cache_a), kept))
        tail = cache_a[0][0][:, :, -1:]                            # a view outlives the cache it was taken from
        tail_copy = tail.clone()
        del cache_a, cache_b
        again, _ = steps(layer, b, mid)
        assert torch.equal(again, out_b) and torch.equal(tail, tail_copy)
        del tail
        again, _ = steps(layer, a[:, 5:], mid)                     # and once more when the others are gone
        assert torch.equal(again, out_a)
        # a cache from elsewhere, its rows cut off in front: positions count from its own first row
        cut = ((mid[0][0][:, :, 64:], mid[0][1][:, :, 64:]), ((mid[1][0][0][:, :, 4:], mid[1][0][1][:, :, 4:]), mid[1][1]))
        got, _ = steps(layer, b[:, :3], cut)
        want, _ = steps(layer, b[:, :3], ((cut[0][0].clone(), cut[0][1].clone()), cut[1]))
        assert torch.equal(got, want)


def test_step_refuses_weights_off_the_16_byte_boundary():
    """Below the layer's own check: the native call reports NSA_ERR_ALIGN instead of loading from such addresses."""
    from native_sparse_attention_pytorch_b200 import _lib as L
    from native_sparse_attention_pytorch_b200.rotary import inverse_frequencies
    layer = build(torch.bfloat16, 8, 2, 64)
    x = recipe.randn((2, 200, 256), 5).bfloat16().to(DEV)
    with torch.no_grad():
        _, cache = layer(x, return_cache=True)
    (w, eps) = layer._native_weights(x[:, :1])

    def step(norm, qkv, gate, gate_b, out, mem):
        return L.host().layer_decode(x[:, :1], norm, eps, qkv, gate, gate_b, out, inverse_frequencies(64, 10000., x.device), mem,
                                     *flat(cache), 8, 16, 64, 32, 4, 100)
    want = step(*w)[0]
    for i in (0, 1, 2, 4, 5):
        buf = torch.empty(w[i].numel() + 4, dtype=w[i].dtype, device=DEV)
        moved = buf[4:].view(w[i].shape).copy_(w[i])
        with pytest.raises(L.NsaError, match='16-byte'):
            step(*w[:i], moved, *w[i + 1:])
    assert torch.equal(step(*w)[0], want)


def storages(cache):
    return [t.untyped_storage().data_ptr() for t in (*cache[0], *cache[1][1])]     # the tensors a step appends to


def test_a_row_is_appended_in_place_only_where_nobody_ever_was():
    layer = build(torch.bfloat16, 8, 2, 64)
    x = recipe.randn((2, 203, 256), 5).bfloat16().to(DEV)
    a, b = (recipe.randn((2, 6, 256), s).bfloat16().to(DEV) for s in (6, 7))
    with torch.no_grad():
        _, mid = layer(x, return_cache=True)
        out_a, first = steps(layer, a, mid)
        assert storages(first) == storages(mid)                    # the prefill's buffers, their only continuation so far
        del first
        out_b, second = steps(layer, b, mid)                       # the rows behind `mid` were given out once
        assert not set(storages(second)) & set(storages(mid))
        # a continuation on another stream gets tensors of that stream
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            out_c, third = steps(layer, a, second)
            assert not set(storages(third)) & set(storages(second))
            more, fourth = steps(layer, a, third)
            assert storages(fourth) == storages(third)             # and goes on in place there
        torch.cuda.current_stream().wait_stream(side)
        want, _ = steps(layer, a, tuple(tuple(t.clone() for t in pair) if isinstance(pair[0], torch.Tensor) else
                                        tuple(tuple(t.clone() for t in p) for p in pair) for pair in second))
        assert torch.equal(out_c, want)


def test_a_recorded_step_leaves_the_caches_of_eager_steps_alone():
    layer = build(torch.bfloat16, 8, 2, 64)
    x = recipe.randn((2, 203, 256), 5).bfloat16().to(DEV)
    a, b = (recipe.randn((2, 4, 256), s).bfloat16().to(DEV) for s in (6, 7))
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.no_grad(), torch.cuda.stream(stream):
        _, mid = layer(x, return_cache=True)
        want, _ = steps(layer, a, tuple((t[0], t[1]) for t in mid))
        _, mid = layer(x, return_cache=True)                       # buffers nothing has been appended to
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out, recorded = steps(layer, a, mid)
            assert not set(storages(recorded)) & set(storages(mid))
        eager_out, eager = steps(layer, b, mid)
        kept = [t.clone() for t in flat(eager)]
        for _ in range(2):
            graph.replay()
            assert torch.equal(out, want)
        assert all(torch.equal(t, k) for t, k in zip(flat(eager), kept))
        after, grown = steps(layer, b, recorded)                   # an eager continuation of what the graph returned
        assert not set(storages(grown)) & set(storages(recorded))
        kept = [t.clone() for t in flat(grown)]
        graph.replay()
        assert all(torch.equal(t, k) for t, k in zip(flat(grown), kept))
        torch.cuda.synchronize()
    del recorded, out, graph


# caches whose compressed logits nearly fill a CTA's shared memory, by type, group and head size: just below what the step
# has always served.  (heads, kv heads, head size, dtype, stride, block, compressed blocks, own rows behind the last one)
@pytest.mark.parametrize('case', [(1, 1, 64, torch.bfloat16, 1, 1, 25100, 3), (2, 1, 128, torch.bfloat16, 1, 2, 31800, 2),
                                  (8, 1, 128, torch.float32, 1, 1, 18800, 1), (16, 1, 128, torch.float32, 1, 1, 12150, 5),
                                  (3, 1, 40, torch.float32, 1, 4, 39220, 7)])
def test_step_on_caches_as_long_as_shared_memory_allows(case):
    from native_sparse_attention_pytorch_b200 import ops
    hq, hkv, d, dtype, stride, block, ncb, rest = case
    t, nsel, window, g = ncb * stride + rest, 5, 37, hq // hkv
    gen = torch.Generator(DEV).manual_seed(ncb)

    def randn(*shape):
        return torch.randn(shape, device=DEV, generator=gen).to(dtype)
    q, qr, keys, vals = randn(1, hq, d), randn(1, hq, d), randn(1, hkv, t, d), randn(1, hkv, t, d)
    ck, cv, mem, gates = randn(1, hkv, ncb, d), randn(1, hkv, ncb, d), randn(2, hkv, 1, d), torch.rand(1, hq, 3, device=DEV, generator=gen).to(dtype)
    got = ops.decode_step(q, qr, keys, vals, ck, cv, mem[0], mem[1], gates, stride=stride, block=block, num_selected=nsel, window=window)

    f = lambda x: x.double().squeeze(0)
    def attend(query, k, v):
        sim = query @ k.transpose(-1, -2) * d ** -0.5
        return sim.softmax(-1) @ v, sim
    k, v, c = f(keys)[0], f(vals)[0], block // stride
    o_cmp, sim = attend(f(q), torch.cat((mem[0, 0].double(), f(ck)[0])), torch.cat((mem[1, 0].double(), f(cv)[0])))
    logits = sim[:, 1:].mean(0)[:ncb // c * c].view(-1, c).mean(1)
    picks = torch.cat((torch.tensor([-1e3], device=DEV, dtype=torch.double), logits)).softmax(0)[1:].topk(nsel)
    assert picks.values[-1] > 1e-10
    rows = [torch.arange(i * block, (i + 1) * block, device=DEV) for i in picks.indices.tolist()] + [torch.arange((t - 1) // block * block, t, device=DEV)]
    o_sel, _ = attend(f(qr), k[torch.cat(rows)], v[torch.cat(rows)])
    o_swa, _ = attend(f(qr), k[-window - 1:], v[-window - 1:])
    gate = f(gates)
    want = (gate[:, 0:1] * o_cmp + gate[:, 1:2] * o_sel + gate[:, 2:3] * o_swa).reshape(1, -1)
    (assert_close_f32 if dtype == torch.float32 else assert_close_bf16)(got, want.float().cpu(), 'merged row')


# (batch, heads, rows, head size, dtype): one piece per row and many, runs of less and more than a block's share, one head and
# many; then views whose heads are not runs, or not on 16-byte boundaries
@pytest.mark.parametrize('case', [(1, 1, 1, 8, torch.bfloat16), (2, 3, 5, 40, torch.float32), (1, 1, 255, 64, torch.bfloat16), (3, 2, 129, 64, torch.bfloat16),
                                  (1, 2, 70000, 128, torch.bfloat16), (64, 8, 33, 64, torch.float32)])
@pytest.mark.parametrize('form', ['dense', 'front cut', 'batch part', 'positions first', 'odd offset'])
def test_a_cache_that_cannot_grow_in_place_is_copied_whole(case, form):
    b, h, rows, d, dtype = case
    layer = build(dtype, 2 * h, h, d, dim=64)
    gen = torch.Generator(DEV).manual_seed(rows)

    def cache(n):
        shape = {'dense': (b, h, n, d), 'front cut': (b, h, n + 2, d), 'batch part': (b + 1, h, n, d), 'positions first': (b, n, h, d)}.get(form)
        if form == 'odd offset':
            return torch.randn(b * h * n * d + 1, device=DEV, generator=gen).to(dtype)[1:].view(b, h, n, d)
        t = torch.randn(shape, device=DEV, generator=gen).to(dtype)
        return {'dense': t, 'front cut': t[:, :, 2:], 'batch part': t[1:], 'positions first': t.transpose(1, 2)}[form]
    k, v, run_k, run_v = cache(rows), cache(rows), cache(7), cache(7)
    empty = torch.zeros(b, h, 0, d, device=DEV, dtype=dtype)
    with torch.no_grad():
        _, got = layer(torch.randn(b, 1, 64, device=DEV, generator=gen).to(dtype), cache=((k, v), ((empty, empty), (run_k, run_v))), return_cache=True)
    for old, new in ((k, got[0][0]), (v, got[0][1]), (run_k, got[1][1][0]), (run_v, got[1][1][1])):
        assert new.shape[2] == old.shape[2] + 1 and torch.equal(new[:, :, :-1], old)
