"""The gradient of the differentiable top-k in the native layer against the same layer run module by module, at the edges of
its 64 x 64 tiles: one column, one more than a tile, rows that end inside one; one and several columns per block."""
import pytest
import torch

import recipe
from test_gpu_native_layer import run
from util import assert_close_f32

from native_sparse_attention_pytorch_b200 import SparseAttention

pytestmark = pytest.mark.gpu


# (batch, length, heads, kv heads, head size, options)
@pytest.mark.parametrize('b, n, heads, kv_heads, d, options', [
    (1, 1040, 4, 2, 64, {}),                                        # 65 columns
    (2, 65, 2, 2, 128, {}),                                         # 4 columns, one row past a tile
    (1, 80, 4, 1, 40, dict(selection_block_size=16)),               # one column per block, the own block takes part
    (3, 130, 8, 2, 72, dict(query_heads_share_selected_kv=False)),  # several selections per KV head, two tiles of features
    (1, 264, 4, 4, 64, dict(causal=False, selection_block_size=32)),
    (2, 70, 8, 8, 64, dict(compress_block_sliding_stride=2, compress_block_size=4, selection_block_size=4)),
])
def test_gradient_through_the_topk(b, n, heads, kv_heads, d, options):
    kw = dict(dim=128, dim_head=d, heads=heads, kv_heads=kv_heads, causal=True, sliding_window_size=20, compress_block_size=32,
              compress_block_sliding_stride=16, selection_block_size=64, num_selected_blocks=2, use_diff_topk=True, use_triton_kernel=True)
    layer = SparseAttention(**{**kw, **options})
    recipe.fill_weights(layer, seed=3)
    layer = layer.to('cuda')
    x, dout = (recipe.randn((b, n, 128), seed).to('cuda') for seed in (5, 6))
    out, dx, grads = run(layer, x, dout)
    assert 'NativeLayer' in out.grad_fn.name()
    hook = layer.combine_heads.register_forward_hook(lambda *_: None)
    want, want_dx, want_grads = run(layer, x, dout)
    hook.remove()
    assert 'NativeLayer' not in want.grad_fn.name()
    assert_close_f32(out, want, 'out')
    assert_close_f32(dx, want_dx, 'd input')
    for name, ref in want_grads.items():
        assert (ref is None) == (grads[name] is None), name
        if ref is not None and grads[name] is not None:
            assert_close_f32(grads[name], ref, name)
