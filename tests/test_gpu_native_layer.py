"""The layer as one native call per direction against the same layer run module by module: a forward hook on a submodule
makes the layer take that path."""
import pytest
import torch

import recipe
from util import assert_close_bf16, assert_close_f32

from native_sparse_attention_pytorch_b200 import SparseAttention

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32

# (batch, length, heads, kv heads, head size, dtype, options): gates whose rows are not whole 16-byte pieces, lengths that
# end inside a block, one block, a length below the overlap of the windows, head sizes without a tensor form, every option
CASES = [
    (2, 257, 4, 4, 64, BF16, {}),
    (1, 1000, 8, 2, 64, BF16, dict(use_diff_topk=True)),
    (3, 130, 16, 1, 128, BF16, dict(compress_block_size=16, selection_block_size=16)),
    (1, 20, 4, 2, 64, BF16, dict(compress_block_size=64)),
    (2, 96, 6, 2, 40, BF16, dict(norm=False)),
    (1, 515, 4, 2, 64, BF16, dict(num_selected_blocks=0)),
    (2, 200, 8, 4, 64, BF16, dict(query_heads_share_selected_kv=False, causal=False, use_diff_topk=True)),
    (2, 140, 6, 3, 64, F32, dict(use_diff_topk=True)),
    (1, 333, 2, 1, 128, F32, dict(causal=False, num_compressed_mem_kv=3)),
    (2, 75, 4, 4, 40, F32, dict(query_heads_share_selected_kv=False, norm=False)),
]


def run(layer, x, dout):
    x = x.clone().requires_grad_()
    out = layer(x)
    out.backward(dout)
    grads = {n: p.grad for n, p in layer.named_parameters()}
    for p in layer.parameters():
        p.grad = None
    return out, x.grad, grads


@pytest.mark.parametrize('case', CASES)
def test_native_layer_equals_the_module_by_module_layer(case):
    b, n, heads, kv_heads, d, dtype, options = case
    kw = dict(dim=256, dim_head=d, heads=heads, kv_heads=kv_heads, causal=True, sliding_window_size=70, compress_block_size=32,
              compress_block_sliding_stride=16, selection_block_size=64, num_selected_blocks=3, use_triton_kernel=True)
    layer = SparseAttention(**{**kw, **options})
    recipe.fill_weights(layer, seed=3)
    layer = layer.to('cuda').to(dtype)
    layer.to_strategy_combine[0].bias.requires_grad_(False)
    x, dout = (recipe.randn((b, n, 256), seed).to(dtype).to('cuda') for seed in (5, 6))

    out, dx, grads = run(layer, x, dout)
    assert 'NativeLayer' in out.grad_fn.name()
    hook = layer.combine_heads.register_forward_hook(lambda *_: None)
    want, want_dx, want_grads = run(layer, x, dout)
    hook.remove()
    assert 'NativeLayer' not in want.grad_fn.name()

    def close(got, ref, what):
        if dtype == F32:
            assert_close_f32(got, ref, what)
        else:   # the layer's gradients sum in fp32 what the modules add in bf16
            assert_close_bf16(got, ref, what, roundings=2, rel_to_max=1e-2)
    close(out, want, 'out')
    close(dx, want_dx, 'd input')
    assert grads.keys() == want_grads.keys()
    for name, ref in want_grads.items():
        # without selected blocks, or with hard picks, some parameters get no gradient or a zero one
        if ref is None or grads[name] is None:
            assert all(g is None or not g.any() for g in (ref, grads[name])), name
        else:
            assert grads[name].shape == ref.shape and grads[name].dtype == ref.dtype, name
            close(grads[name], ref, name)

    if layer.causal:
        with torch.no_grad():
            _, cache = layer(x, return_cache=True)
            hook = layer.combine_heads.register_forward_hook(lambda *_: None)
            _, ref = layer(x, return_cache=True)
            hook.remove()
        for got, want in zip((*cache[0], *cache[1][0], *cache[1][1]), (*ref[0], *ref[1][0], *ref[1][1])):
            assert got.shape == want.shape and got.dtype == want.dtype
            close(got, want, 'cache')


def test_parameters_packed_into_one_buffer_take_the_module_path():
    """Four heads in bf16: the gate bias is 24 bytes long, so the projections packed behind it start at 8 mod 16 and the
    layer has to take the path whose operators read such weights."""
    layer = SparseAttention(dim=256, dim_head=64, heads=4, kv_heads=2, causal=True, sliding_window_size=70, compress_block_size=32,
                            compress_block_sliding_stride=16, selection_block_size=64, num_selected_blocks=3, use_triton_kernel=True)
    recipe.fill_weights(layer, seed=3)
    layer = layer.to('cuda').to(BF16)
    x, dout, token = (recipe.randn((2, n, 256), seed).to(BF16).to('cuda') for n, seed in ((257, 5), (257, 6), (1, 7)))

    def everything():
        out, dx, grads = run(layer, x, dout)
        with torch.no_grad():
            _, cache = layer(x, return_cache=True)
            step = layer(token, cache=cache)
        return [out, dx, step, *grads.values()]
    hook = layer.combine_heads.register_forward_hook(lambda *_: None)
    want = everything()
    hook.remove()
    flat, at = torch.cat([p.detach().reshape(-1) for p in layer.parameters()]), 0
    for name, p in list(layer.named_parameters()):
        owner, _, leaf = name.rpartition('.')
        layer.get_submodule(owner)._parameters[leaf] = torch.nn.Parameter(flat[at:at + p.numel()].view(p.shape))
        at += p.numel()
    assert any(p.data_ptr() % 16 for p in layer.parameters()) and layer.norm.weight.data_ptr() % 16 == 0
    for got, ref in zip(everything(), want):
        assert (got is None) == (ref is None)
        if ref is not None:
            assert_close_bf16(got, ref, 'packed parameters')


@pytest.mark.parametrize('how', ['native', 'module by module'])
def test_graphs_and_eager_steps_of_one_shape_do_not_share_an_index(how):
    """Two graphs of one shape, recorded on a stream that never ran this shape before; an eager step on that stream before
    either graph was replayed; then replays after so many other shapes that every index kept for eager steps is gone."""
    from native_sparse_attention_pytorch_b200 import ops
    layer = SparseAttention(dim=256, dim_head=64, heads=8, kv_heads=2, causal=True, sliding_window_size=128, compress_block_size=32,
                            compress_block_sliding_stride=16, selection_block_size=64, num_selected_blocks=4, use_triton_kernel=True)
    recipe.fill_weights(layer, seed=7)
    layer = layer.to('cuda').to(BF16)
    if how != 'native':
        layer.combine_heads.register_forward_hook(lambda *_: None)
    params = list(layer.parameters())

    def step(x, dout):
        out = layer(x)
        return [g for g in torch.autograd.grad(out, [x, *params], dout) if g is not None]

    def inputs(n, seed):
        x, dout = (recipe.randn((1, n, 256), seed + i).to(BF16).to('cuda') for i in range(2))
        return x.requires_grad_(), dout

    def same(got, want):
        torch.cuda.synchronize()
        ops.check_device_status()
        for g, w in zip(got, want):
            assert_close_bf16(g, w, 'gradient', roundings=2, rel_to_max=1e-2)

    warm, other = torch.cuda.Stream(), torch.cuda.Stream()
    warm.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(warm):
        x, dout = inputs(700, 11)
        want = step(x, dout)
        step(x, dout)
    torch.cuda.synchronize()
    graphs = []
    with torch.cuda.stream(other):
        for _ in range(2):
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=other):
                got = step(x, dout)
            graphs.append((graph, got))
        same(step(x, dout), want)
        for graph, got in reversed(graphs):
            graph.replay()
            same(got, want)
        for i in range(20):
            step(*inputs(200 + 10 * i, 31))
        for graph, got in graphs:
            for g in got:
                g.zero_()
            graph.replay()
            same(got, want)
    del graphs, graph, got


@pytest.mark.parametrize('dtype', [BF16, F32])
def test_kept_gradients_do_not_keep_the_scratch_of_the_backward(dtype):
    layer = SparseAttention(dim=256, dim_head=64, heads=4, kv_heads=2, causal=True, sliding_window_size=70, compress_block_size=32,
                            compress_block_sliding_stride=16, selection_block_size=64, num_selected_blocks=3, use_triton_kernel=True)
    recipe.fill_weights(layer, seed=3)
    layer = layer.to('cuda').to(dtype)
    sizes = []
    for n in (64, 2048):
        x, dout = (recipe.randn((2, n, 256), seed).to(dtype).to('cuda') for seed in (5, 6))
        out, dx, grads = run(layer, x, dout)
        assert 'NativeLayer' in out.grad_fn.name()
        sizes.append({name: g.untyped_storage().nbytes() for name, g in grads.items()})
    assert sizes[0] == sizes[1]


def test_a_tangent_is_refused_and_not_dropped():
    from native_sparse_attention_pytorch_b200 import native_sparse_attend
    layer = SparseAttention(dim=256, dim_head=64, heads=4, kv_heads=2, causal=True, sliding_window_size=70, compress_block_size=32,
                            compress_block_sliding_stride=16, selection_block_size=64, num_selected_blocks=3, use_triton_kernel=True).to('cuda')
    x, t = (recipe.randn((1, 130, 256), seed).to('cuda') for seed in (5, 6))
    q, dq = (recipe.randn((1, 4, 130, 64), seed).to('cuda') for seed in (7, 8))
    k = recipe.randn((1, 2, 130, 64), 9).to('cuda')
    idx, mask = torch.zeros(1, 2, 130, 1, dtype=torch.int64, device='cuda'), torch.zeros(1, 2, 130, 1, dtype=torch.bool, device='cuda')
    fwd = torch.autograd.forward_ad
    with fwd.dual_level():
        for grad in (True, False):
            with torch.set_grad_enabled(grad):
                with pytest.raises(RuntimeError, match='jvp'):
                    layer(fwd.make_dual(x, t))
                with pytest.raises(RuntimeError, match='jvp'):
                    native_sparse_attend(fwd.make_dual(q, dq), k, k, 64, idx, mask)
        weight = layer.to_qkv.weight.detach()
        with pytest.raises(RuntimeError, match='jvp'):
            torch.func.functional_call(layer, {'to_qkv.weight': fwd.make_dual(weight, weight)}, (x,))
        assert native_sparse_attend(q, k, k, 64, idx, mask).shape == q.shape


# one slice and many, one and several groups of 256 columns, rows of whole 16-byte pieces and not
@pytest.mark.parametrize('b, n, heads, d, dtype', [(1, 40, 2, 64, F32), (2, 4096, 8, 64, F32), (5, 700, 6, 40, F32), (2, 2000, 96, 8, BF16)])
def test_the_gradient_of_the_gate_bias_repeats_to_the_bit(b, n, heads, d, dtype):
    """Nothing in front of it depends on the order of atomics."""
    layer = SparseAttention(dim=256, dim_head=d, heads=heads, kv_heads=heads // 2, causal=True, sliding_window_size=70, compress_block_size=32,
                            compress_block_sliding_stride=16, selection_block_size=64, num_selected_blocks=3, use_triton_kernel=True)
    recipe.fill_weights(layer, seed=3)
    layer = layer.to('cuda').to(dtype)
    x, dout = (recipe.randn((b, n, 256), seed).to(dtype).to('cuda') for seed in (5, 6))
    out, _, grads = run(layer, x, dout)
    assert 'NativeLayer' in out.grad_fn.name()
    hook = layer.combine_heads.register_forward_hook(lambda *_: None)
    _, _, want = run(layer, x, dout)
    hook.remove()
    for name in ('to_strategy_combine.0.bias', 'k_compress.1.bias'):
        if dtype == F32:
            assert_close_f32(grads[name], want[name], name)
    for _ in range(4):
        _, _, again = run(layer, x, dout)
        assert torch.equal(again['to_strategy_combine.0.bias'], grads['to_strategy_combine.0.bias'])


@pytest.mark.parametrize('options', [{}, dict(dim_head=128, heads=8)])
def test_the_native_layer_needs_no_more_memory_than_the_modules(options):
    kw = dict(dim=512, dim_head=64, heads=16, kv_heads=4, causal=True, sliding_window_size=128, compress_block_size=32,
              compress_block_sliding_stride=16, selection_block_size=64, num_selected_blocks=8, use_triton_kernel=True)
    layer = SparseAttention(**{**kw, **options})
    recipe.fill_weights(layer, seed=3)
    layer, n = layer.to('cuda').to(BF16), 4096
    x, dout = (recipe.randn((2, n, 512), seed).to(BF16).to('cuda') for seed in (5, 6))

    def peaks():
        def peak(call):
            call()
            torch.cuda.synchronize()
            before = torch.cuda.memory_allocated()
            torch.cuda.reset_peak_memory_stats()
            call()
            return torch.cuda.max_memory_allocated() - before

        def prefill():
            with torch.no_grad():
                layer(x, return_cache=True)
        return peak(lambda: run(layer, x, dout)), peak(prefill)
    native = peaks()
    hook = layer.combine_heads.register_forward_hook(lambda *_: None)
    modules = peaks()
    hook.remove()
    # the caches of the native prefill have room for 64 to 1024 more rows
    rows = 4 * 2 * layer.kv_heads * (n // 8 + 64) * layer.dim_head * x.element_size()
    # the backward gives up what the forward saved at its end, where the modules release theirs one by one
    assert native[0] <= 1.03 * modules[0] and native[1] <= 1.03 * modules[1] + rows, (native, modules)
