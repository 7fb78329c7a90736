"""What the layer checks on the host before it hands raw pointers to the native calls.  No GPU: the checks look at
tensors, the calls behind them are never reached."""
import pytest
import torch

from native_sparse_attention_pytorch_b200 import SparseAttention
from native_sparse_attention_pytorch_b200 import _lib as L

BF16, F32 = torch.bfloat16, torch.float32
DIM, HEADS, KV_HEADS, D, CBS = 64, 4, 2, 64, 16


def build(dtype=BF16, **options):
    kw = dict(dim=DIM, dim_head=D, heads=HEADS, kv_heads=KV_HEADS, causal=True, sliding_window_size=32, compress_block_size=CBS,
              compress_block_sliding_stride=8, selection_block_size=16, num_selected_blocks=2, use_triton_kernel=True)
    return SparseAttention(**{**kw, **options}).to(dtype)


def off_by(t, elements):
    """A dense copy of t that starts `elements` elements behind a 16-byte boundary."""
    buf = torch.empty(t.numel() + 16, dtype=t.dtype)
    lead = (-buf.data_ptr() % 16) // t.element_size()
    view = buf[lead + elements:lead + elements + t.numel()].view(t.shape)
    view.copy_(t)
    assert view.is_contiguous() and view.data_ptr() % 16 == elements * t.element_size() % 16
    return view


@pytest.mark.parametrize('dtype', [BF16, F32])
def test_parameters_off_the_16_byte_boundary_take_the_module_path(dtype):
    """A parameter that is a view into a flat buffer may start anywhere; the native kernels load 16 bytes at a time."""
    layer, x = build(dtype), torch.zeros(2, 32, DIM, dtype=dtype)
    assert layer._native_parameters(x) is not None
    for name, p in list(layer.named_parameters()):
        owner = layer.get_submodule(name.rpartition('.')[0])
        owner._parameters[name.rpartition('.')[2]] = torch.nn.Parameter(off_by(p.detach(), 2))
        assert layer._native_parameters(x) is None, name
        owner._parameters[name.rpartition('.')[2]] = torch.nn.Parameter(off_by(p.detach(), 16 // p.element_size()))
        assert layer._native_parameters(x) is not None, name


@pytest.mark.parametrize('dtype', [BF16, F32])
def test_parameters_packed_into_one_buffer(dtype):
    """Four heads in bf16: the gate bias is 24 bytes, so what is packed behind it starts at 8 mod 16."""
    layer, x = build(dtype), torch.zeros(1, 32, DIM, dtype=dtype)
    flat = torch.cat([p.detach().reshape(-1) for p in layer.parameters()])
    at, aligned = 0, True
    for name, p in list(layer.named_parameters()):
        view = flat[at:at + p.numel()].view(p.shape)
        aligned = aligned and view.data_ptr() % 16 == 0
        layer.get_submodule(name.rpartition('.')[0])._parameters[name.rpartition('.')[2]] = torch.nn.Parameter(view)
        at += p.numel()
    assert (layer._native_parameters(x) is not None) == aligned
    assert aligned == (dtype == F32)


def test_an_input_at_an_odd_offset_takes_the_module_path():
    layer, x = build(), torch.zeros(1, 32, DIM, dtype=BF16)
    assert layer._native_parameters(x) is not None
    assert layer._native_parameters(off_by(x, 1)) is None


def decode_arguments(layer, **changes):
    b, t, ncb, r = 2, 20, 2, 5
    cache = dict(past_k=(b, KV_HEADS, t, D), past_v=(b, KV_HEADS, t, D), ck=(b, KV_HEADS, ncb, D), cv=(b, KV_HEADS, ncb, D),
                 run_k=(b, KV_HEADS, r, D), run_v=(b, KV_HEADS, r, D))
    x = torch.zeros(changes.pop('x', (b, 1, DIM)), dtype=BF16)
    (norm, qkv, gate, gate_b, out, mem), eps = layer._native_weights(x)
    w = dict(qkv=qkv, gate=gate, gate_b=gate_b, out=out, mem=mem)
    for name, shape in changes.items():
        (cache if name in cache else w)[name] = shape if name in cache else torch.zeros(shape, dtype=BF16)
    return (x, norm, eps, w['qkv'], w['gate'], w['gate_b'], w['out'], torch.zeros(D // 2), w['mem'],
            *(torch.zeros(s, dtype=BF16) for s in cache.values()), HEADS, 8, 16, CBS, 2, 32)


@pytest.mark.parametrize('changes', [
    dict(x=(3, 1, DIM)), dict(x=(1, 1, DIM)), dict(x=(2, 2, DIM)),
    dict(past_k=(3, KV_HEADS, 20, D)), dict(past_v=(2, KV_HEADS, 19, D)), dict(past_k=(2, HEADS, 20, D)), dict(past_v=(2, KV_HEADS, 20, 32)),
    dict(ck=(1, KV_HEADS, 2, D)), dict(cv=(2, KV_HEADS, 1, D)), dict(cv=(2, 1, 2, D)), dict(ck=(2, KV_HEADS, 2, 32)),
    dict(run_k=(1, KV_HEADS, 5, D)), dict(run_v=(2, KV_HEADS, 4, D)), dict(run_v=(2, 1, 5, D)), dict(run_k=(2, KV_HEADS, D)),
    dict(out=(DIM, 2 * HEADS * D)), dict(out=(2 * DIM, HEADS * D)), dict(mem=(2, 1, 1, D)), dict(gate_b=(3,))],
    ids=lambda c: '-'.join(f'{k}{list(v)}' for k, v in c.items()))
def test_a_step_refuses_caches_of_another_shape(changes):
    """Batch, heads and row length are taken from one tensor and address all others, so each has to agree."""
    with pytest.raises(L.NsaError, match='decode step'):
        L.host().layer_decode(*decode_arguments(build(), **changes))


def test_forward_mode_differentiation_takes_the_module_path():
    """The native calls have no tangents to give; the modules' operators say so."""
    layer, x = build(), torch.zeros(2, 32, DIM, dtype=BF16)
    assert layer._native_weights(x) is not None
    with torch.autograd.forward_ad.dual_level():
        assert layer._native_weights(x) is None
    assert layer._native_weights(x) is not None


def test_parameters_that_became_plain_tensors_take_the_module_path():
    """A wrapper that shards parameters may delete them from their modules and put views of its own buffer there."""
    x = torch.zeros(2, 32, DIM, dtype=BF16)
    for name, _ in build().named_parameters():
        layer = build()
        owner, _, leaf = name.rpartition('.')
        owner = layer.get_submodule(owner)
        value = getattr(owner, leaf).detach().clone()
        delattr(owner, leaf)
        setattr(owner, leaf, value)
        assert layer._native_parameters(x) is None, name


@pytest.mark.parametrize('name, module', [
    ('combine_heads', torch.nn.Linear(HEADS * D, 2 * DIM, bias=False)), ('combine_heads', torch.nn.Linear(HEADS * D, DIM)),
    ('to_qkv', torch.nn.Linear(DIM, (HEADS + 2 * KV_HEADS) * D)), ('to_strategy_combine.0', torch.nn.Linear(DIM, 3 * HEADS, bias=False)),
    ('k_compress.3', torch.nn.Linear(CBS * D, D, bias=False)), ('v_compress.1', torch.nn.Linear(CBS * D, 2 * CBS * D))])
def test_replaced_submodules_take_the_module_path(name, module):
    x = torch.zeros(2, 32, DIM, dtype=BF16)
    for norm in (True, False):
        layer = build(norm=norm)
        assert layer._native_parameters(x) is not None
        owner, _, leaf = name.rpartition('.')
        setattr(layer.get_submodule(owner), leaf, module.to(BF16))
        assert layer._native_parameters(x) is None


def test_a_layer_pickled_before_it_had_native_calls_still_runs():
    layer, x = build(), torch.zeros(2, 32, DIM, dtype=BF16)
    before = {'heads', 'kv_heads', 'dim_head', 'num_grouped_queries', 'scale', 'causal', 'kernel_impl', 'qkv_split', 'sliding_window_size',
              'compress_block_size', 'compress_block_sliding_stride', 'num_mem_compress_kv', 'use_diff_topk', 'query_heads_share_selected_kv',
              'selection_block_size', 'num_selected_blocks', 'use_triton_kernel', 'training'}
    for name in [n for n in layer.__dict__ if not n.startswith(('_parameters', '_modules', '_buffers', '_backward', '_forward', '_is_full',
                                                                '_non_persistent', '_state_dict', '_load_state')) and n not in before]:
        del layer.__dict__[name]
    assert layer._native_parameters(x) is not None
