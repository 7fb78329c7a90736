"""Drop-in ``SparseAttention`` layer whose hot path -- compressed attention,
block selection, selected-block attention, sliding window and the gated
combine -- runs on the B200 kernels of libnsa_b200.so.

Constructor arguments, parameter names and the forward signature follow
upstream's module (NSA:189-209, NSA:549-557), so a state_dict moves between
the two.  Only the accelerated path exists here: the layer must be built with
``use_triton_kernel=True`` (upstream's name for "use the fused kernel", kept
for compatibility) and called on CUDA tensors; anything else raises instead of
silently computing somewhere else."""
from copy import deepcopy

import torch
import torch.nn.functional as F
from torch import nn
from torch.autograd import forward_ad
from torch.nn import Module

from . import _lib as L
from . import ops
from .norm import MAX_PIECES, RMSNorm
from .rotary import RotaryEmbedding, inverse_frequencies

_has_any_global_hook = nn.modules.module._has_any_global_hook
_F32_EPS = torch.finfo(torch.float32).eps
_PLAIN = (nn.Parameter, torch.Tensor)


def _plain(*params):
    """All are tensors of the ordinary classes (a parameter that is missing is not)."""
    for p in params:
        if p.__class__ not in _PLAIN:
            return False
    return True


def _untouched(module, cls):
    """`module` is exactly a `cls` that runs its own forward: no subclass, no hooks, no replaced forward."""
    d = module.__dict__
    return module.__class__ is cls and not (d['_forward_hooks'] or d['_forward_pre_hooks'] or d['_backward_hooks'] or
                                            d['_backward_pre_hooks'] or 'forward' in d)


class _Windows(Module):
    """[B,H,N,d] -> [B,H,ncb,cbs,d]: window w holds tokens (w+1)*stride-cbs .. (w+1)*stride-1,
    zero where that is negative (same result as upstream's pad + unfold, NSA:270-275)."""

    def __init__(self, block, stride):
        super().__init__()
        self.block, self.stride = block, stride

    def forward(self, t):
        t = F.pad(t, (0, 0, self.block - self.stride, 0))
        return t.unfold(2, self.block, self.stride).permute(0, 1, 2, 4, 3)


class SparseAttention(Module):
    def __init__(
        self,
        dim,
        dim_head,
        heads,
        sliding_window_size,
        compress_block_size,
        compress_block_sliding_stride,
        selection_block_size,
        num_selected_blocks,
        kv_heads=None,
        num_compressed_mem_kv=1,
        causal=False,
        norm=True,
        use_diff_topk=False,
        use_triton_kernel=False,
        query_heads_share_selected_kv=True,
        compress_mlp: Module | None = None,
        compress_mlp_expand_factor=1.,
        strategy_combine_mlp: Module | None = None,
        kernel_impl='auto',
    ):
        super().__init__()
        kv_heads = heads if kv_heads is None else kv_heads
        assert kv_heads <= heads and heads % kv_heads == 0
        self.heads, self.kv_heads, self.dim_head = heads, kv_heads, dim_head
        self.num_grouped_queries = heads // kv_heads
        self.scale = dim_head ** -0.5
        self.causal = causal
        self.kernel_impl = kernel_impl

        self.norm = RMSNorm(dim) if norm else nn.Identity()
        self.rotary_emb = RotaryEmbedding(dim_head)
        self.qkv_split = (dim_head * heads, dim_head * kv_heads, dim_head * kv_heads)
        self.to_qkv = nn.Linear(dim, sum(self.qkv_split), bias=False)

        self.sliding_window_size = sliding_window_size

        self.compress_block_size = compress_block_size
        self.compress_block_sliding_stride = compress_block_sliding_stride
        assert compress_block_size >= compress_block_sliding_stride, 'compress_block_size must be >= compress_block_sliding_stride'
        assert compress_block_sliding_stride > 0, 'compress_block_sliding_stride must be greater than 0'
        assert selection_block_size % compress_block_sliding_stride == 0, \
            f'selection_block_size {selection_block_size} must be divisible by compress_block_sliding_stride {compress_block_sliding_stride}'
        self.split_compress_window = _Windows(compress_block_size, compress_block_sliding_stride)

        assert num_compressed_mem_kv > 0
        self.num_mem_compress_kv = num_compressed_mem_kv
        self.compress_mem_kv = nn.Parameter(torch.zeros(2, kv_heads, num_compressed_mem_kv, dim_head))
        self.k_intrablock_positions = nn.Parameter(torch.zeros(kv_heads, compress_block_size, dim_head))
        self.v_intrablock_positions = nn.Parameter(torch.zeros(kv_heads, compress_block_size, dim_head))

        if compress_mlp is None:
            compress_dim = compress_block_size * dim_head
            hidden = int(compress_mlp_expand_factor * compress_dim)
            # index 0 flattens (n d) so the Linear layers sit at indices 1 and 3 as upstream's do
            compress_mlp = nn.Sequential(nn.Flatten(-2), nn.Linear(compress_dim, hidden), nn.ReLU(),
                                         nn.Linear(hidden, dim_head))
        self.k_compress = deepcopy(compress_mlp)
        self.v_compress = deepcopy(compress_mlp)

        self.use_diff_topk = use_diff_topk
        self.query_heads_share_selected_kv = query_heads_share_selected_kv
        self.selection_block_size = selection_block_size
        assert num_selected_blocks >= 0
        if num_selected_blocks == 0:
            print('`num_selected_blocks` should be set greater than 0, unless if you are ablating it for experimental purposes')
        self.num_selected_blocks = num_selected_blocks
        self.use_triton_kernel = use_triton_kernel

        if strategy_combine_mlp is None:
            strategy_combine_mlp = nn.Linear(dim, 3 * heads)
            nn.init.zeros_(strategy_combine_mlp.weight)
            strategy_combine_mlp.bias.data.copy_(torch.tensor([-2., -2., 2.] * heads))
        self.to_strategy_combine = nn.Sequential(strategy_combine_mlp, nn.Sigmoid())

        self.combine_heads = nn.Linear(dim_head * heads, dim, bias=False)

    def _native_weights(self, x):
        """The parameters the native layer calls take, or None where the layer has to run module by module: a replaced
        or hooked submodule, a parameter that is not one any more (a wrapper put a plain tensor in its place), autocast,
        forward-mode differentiation (the modules refuse it).  Whether the calls can take them as they are is for
        `layer_takes` to say."""
        if (x.dtype is not torch.bfloat16 and x.dtype is not torch.float32) or torch.is_autocast_enabled('cuda') or \
                _has_any_global_hook() or torch.compiler.is_compiling() or forward_ad._current_level >= 0:
            return None
        m = self._modules
        norm, gate, qkv, out = m['norm'], m['to_strategy_combine'], m['to_qkv'], m['combine_heads']
        gate_linear = gate._modules.get('0')
        norm_w, eps = None, 0.
        if _untouched(norm, RMSNorm):
            norm_w, eps = norm._parameters.get('weight'), norm.eps
            if not _plain(norm_w):
                return None
            eps = _F32_EPS if eps is None else eps
        elif not _untouched(norm, nn.Identity):
            return None
        if not (_untouched(m['rotary_emb'], RotaryEmbedding) and _untouched(gate, nn.Sequential) and len(gate._modules) == 2 and
                _untouched(gate._modules['1'], nn.Sigmoid) and _untouched(qkv, nn.Linear) and _untouched(out, nn.Linear) and
                _untouched(gate_linear, nn.Linear)):
            return None
        if qkv.bias is not None or out.bias is not None:
            return None
        w = (qkv._parameters.get('weight'), gate_linear._parameters.get('weight'), gate_linear._parameters.get('bias'),
             out._parameters.get('weight'), self._parameters.get('compress_mem_kv'))
        return ((norm_w, *w), eps) if _plain(*w) else None

    def _layer_takes(self, x, weights):
        return L.host().layer_takes(x, weights, self.heads, self.kv_heads, self.dim_head, self.compress_block_size, self.num_mem_compress_kv)

    def _native_parameters(self, x):
        """All parameters of a native layer call, in its order, and the norm's epsilon; or None where the layer has to run
        module by module (`_native_weights`, another compress network, or an input or parameters that do not fit: of another
        type, device or shape, or off the 16-byte boundaries the kernels load from)."""
        native, k_net, v_net = self._native_weights(x), self._default_network('k_compress'), self._default_network('v_compress')
        pos = (self._parameters.get('k_intrablock_positions'), self._parameters.get('v_intrablock_positions'))
        if native is None or k_net is None or v_net is None or not _plain(*pos):
            return None
        weights = (*native[0], *pos, *k_net, *v_net)
        return (weights, native[1]) if self._layer_takes(x, weights) else None

    def _native_layer(self, x, return_cache):
        """The whole forward natively, or None where the layer has to run module by module (a chosen kernel family, a
        plug-in or hooked submodule, a sequence shorter than a compressed block, a cache that carries gradients)."""
        if self.kernel_impl != 'auto' or not ops.HAND_OVER_DELTA or not ops.REUSE_INDEX:
            return None
        d, n = self.dim_head, x.shape[1]
        if n < self.compress_block_sliding_stride or d % 8 or d > 256 or x.shape[0] == 0 or x.__class__ not in _PLAIN:
            return None
        native = self._native_parameters(x)
        if native is None:
            return None
        weights, eps = native
        cfg = (self.heads, self.kv_heads, d, self.sliding_window_size, self.compress_block_size,
               self.compress_block_sliding_stride, self.selection_block_size, self.num_selected_blocks,
               self.num_mem_compress_kv, int(self.causal), int(self.query_heads_share_selected_kv), int(self.use_diff_topk))
        inv_freq = inverse_frequencies(d, self.rotary_emb.theta, x.device)
        if torch.is_grad_enabled() and (x.requires_grad or any([p.requires_grad for p in weights if p is not None])):
            if return_cache or (weights[0] is not None and x.shape[2] * x.element_size() > 16 * MAX_PIECES):
                return None
            return L.host().layer_apply(x, weights, eps, inv_freq, cfg, ops._status_word(x.device))
        out, *cache = L.host().layer_forward(x, weights, eps, inv_freq, cfg, ops._status_word(x.device), False, return_cache)
        if not return_cache:
            return out
        keys, vals, ck, cv, run_k, run_v = cache
        return out, ((keys, vals), ((ck, cv), (run_k, run_v)))

    def _split_heads(self, t):
        b, n, _ = t.shape
        return t.view(b, n, -1, self.dim_head).transpose(1, 2)   # a view: the kernels take the strides

    def _default_network(self, name):
        """The parameters (two linear layers) of a compress network that is the default one, as built, else None."""
        net = self._modules[name]
        m = list(net._modules.values()) if _untouched(net, nn.Sequential) else ()
        if len(m) != 4 or not (_untouched(m[0], nn.Flatten) and (m[0].start_dim, m[0].end_dim) == (-2, -1) and
                               _untouched(m[1], nn.Linear) and _untouched(m[2], nn.ReLU) and _untouched(m[3], nn.Linear)):
            return None
        w = (m[1]._parameters.get('weight'), m[1]._parameters.get('bias'), m[3]._parameters.get('weight'), m[3]._parameters.get('bias'))
        return w if _plain(*w) else None

    def _compress_filled(self, ck, cv, run_k, run_v, native=False):
        """The window that was being filled is complete: compress it and keep its overlap with the next one (the step
        before attended the blocks that existed before this token, as upstream's does)."""
        grown = None
        pk, pv = self.k_intrablock_positions, self.v_intrablock_positions
        if native:
            k_net, v_net = self._default_network('k_compress'), self._default_network('v_compress')
            if k_net is not None and v_net is not None and _plain(pk, pv):
                grown = L.host().compress_filled(run_k, run_v, pk, pv, *k_net, *v_net, ck, cv)
        if grown is not None:
            ck, cv = grown
        else:
            ck = torch.cat((ck, self.k_compress((run_k + pk)[:, :, None])), dim=-2)
            cv = torch.cat((cv, self.v_compress((run_v + pv)[:, :, None])), dim=-2)
        first = run_k.shape[-2] - (self.compress_block_size - self.compress_block_sliding_stride)
        return ck, cv, run_k[..., first:, :], run_v[..., first:, :]

    def _native_step(self, x, past_k, past_v, ck, cv, run_k, run_v):
        """The step as three launches (norm with qkv and gate projections, attention with rotary and the append to the
        caches, output projection) where nothing on it needs a gradient; None where it has to run module by module.  The returned caches are views of
        buffers with some room behind them (csrc/host/rooms.h)."""
        if torch.is_grad_enabled() and (x.requires_grad or past_k.requires_grad or past_v.requires_grad or
                                        any(p.requires_grad for p in self.parameters())):
            return None
        d = self.dim_head
        if d % 8 or d > 128 or self.num_selected_blocks > 32 or self.num_grouped_queries > 16:
            return None
        native = self._native_weights(x)
        if native is None:
            return None
        for t in (past_k, past_v, ck, cv, run_k, run_v):
            if t.__class__ is not torch.Tensor:
                return None
        return L.host().layer_step(
            x, native[0], native[1], inverse_frequencies(d, self.rotary_emb.theta, x.device), past_k, past_v, ck, cv, run_k, run_v,
            (self.heads, self.compress_block_sliding_stride, self.selection_block_size, self.compress_block_size, self.num_selected_blocks,
             self.sliding_window_size))

    def forward_inference(self, inp, cache, return_cache=True):
        """One decoding step (upstream NSA:338-547): `inp` is the newest token [B, 1, dim], `cache` what the previous
        call returned: ((rotated keys, values), ((compressed keys, compressed values), (keys, values of the window
        that is being filled for the next compressed block, un-rotated))).  The attention part -- compressed branch,
        block selection, selected blocks plus the own block, sliding window, gated combine -- is one kernel launch
        (`ops.decode_step`, all (batch, KV head) units in its grid), and without gradients the whole step is three
        launches (`_native_step`) and the returned caches share memory with the ones they continue, where those are the
        newest of their buffer and of the same stream (csrc/host/rooms.h): editing one in place changes the rows the
        others have in common with it; clone a cache that is to be edited.  It keeps upstream's behaviour,
        including that the memory slots are attended only once a compressed block exists."""
        assert self.causal, 'inference only relevant for autoregressive'
        if not self.query_heads_share_selected_kv:
            raise NotImplementedError('decoding with per-query-head selection is not built (upstream gathers K/V with '
                                      'indices of the wrong head count in that case)')
        (past_k, past_v), ((ck, cv), (run_k, run_v)) = cache
        b = inp.shape[0]
        h, d = self.heads, self.dim_head
        st, cbs, sel = self.compress_block_sliding_stride, self.compress_block_size, self.selection_block_size
        native = self._native_step(inp, past_k, past_v, ck, cv, run_k, run_v)
        if native is not None:
            out, keys, vals, run_k, run_v = native
            if not return_cache:
                return out
            if run_k.shape[-2] % cbs == 0:
                ck, cv, run_k, run_v = self._compress_filled(ck, cv, run_k, run_v, native=True)
            return out, ((keys, vals), ((ck, cv), (run_k, run_v)))
        pos = past_k.shape[-2]                       # position of the new token
        x = self.norm(inp)
        q, k, v = (self._split_heads(t).contiguous() for t in self.to_qkv(x).split(self.qkv_split, dim=-1))
        run_k, run_v = torch.cat((run_k, k), dim=-2), torch.cat((run_v, v), dim=-2)   # compression sees un-rotated k, v
        qr = self.rotary_emb.rotate_queries_or_keys(q, offset=pos)
        keys = torch.cat((past_k, self.rotary_emb.rotate_queries_or_keys(k, offset=pos)), dim=-2)
        vals = torch.cat((past_v, v), dim=-2)

        gates = self.to_strategy_combine(x).view(b, h, 3)
        merged = ops.decode_step(q.view(b, h, d), qr.view(b, h, d), keys, vals, ck, cv, self.compress_mem_kv[0],
                                 self.compress_mem_kv[1], gates, stride=st, block=sel,
                                 num_selected=self.num_selected_blocks, window=self.sliding_window_size)

        if run_k.shape[-2] % cbs == 0:
            ck, cv, run_k, run_v = self._compress_filled(ck, cv, run_k, run_v)

        out = self.combine_heads(merged.view(b, 1, h * d))
        if not return_cache:
            return out
        return out, ((keys, vals), ((ck, cv), (run_k, run_v)))

    def forward(
        self,
        inp,
        cache=None,
        disable_triton_kernel=False,
        sliding_window_flex_mask=None,
        fine_selection_flex_mask=None,
        return_cache=False,
        return_intermediates=False,
        forced_selection=None,
    ):
        """Upstream's signature (NSA:549-557) plus two keyword arguments of this package: ``return_intermediates``
        also returns the tensors at the boundaries of the hot path, and ``forced_selection`` = (block indices,
        mask), both [B, Hs, N, k], replaces the layer's own block selection (used to compare two precisions of the
        layer on identical blocks).  A tensor-core kernel of an earlier call that gave up on a bounded wait is
        reported here, one call late and without synchronising (`ops.poll_device_status`)."""
        if inp.is_cuda:
            ops.poll_device_status(inp.device)
        if cache is not None:
            if not inp.is_cuda:
                raise RuntimeError('SparseAttention (B200 kernels) needs CUDA tensors; there is no CPU path here')
            return self.forward_inference(inp, cache, return_cache=return_cache)
        if not self.use_triton_kernel or disable_triton_kernel:
            raise RuntimeError('this package implements only the fused-kernel path: construct SparseAttention with '
                               'use_triton_kernel=True and do not pass disable_triton_kernel')
        if sliding_window_flex_mask is not None or fine_selection_flex_mask is not None:
            raise RuntimeError('flex-attention masks select another backend upstream; this package has one backend')
        if not inp.is_cuda:
            raise RuntimeError('SparseAttention (B200 kernels) needs CUDA tensors; there is no CPU path here')
        assert not (not self.causal and return_cache)

        if not return_intermediates and forced_selection is None:
            native = self._native_layer(inp, return_cache)
            if native is not None:
                return native

        b, n, _ = inp.shape
        h, hkv, d = self.heads, self.kv_heads, self.dim_head
        st, sel = self.compress_block_sliding_stride, self.selection_block_size
        impl = self.kernel_impl
        ncb = n // st

        x = self.norm(inp)
        q, k, v = self.to_qkv(x).split(self.qkv_split, dim=-1)
        q, k, v = map(self._split_heads, (q, k, v))

        # compressed keys / values: plug-in networks on un-rotated k, v (NSA:589-614)
        if ncb > 0 and ops.compress_windows_supported(k):
            kw = ops.compress_windows(k, self.k_intrablock_positions, self.compress_block_size, st, ncb)
            vw = ops.compress_windows(v, self.v_intrablock_positions, self.compress_block_size, st, ncb)
        elif ncb > 0:
            kw = self.split_compress_window(k[..., : ncb * st, :]) + self.k_intrablock_positions[None, :, None]
            vw = self.split_compress_window(v[..., : ncb * st, :]) + self.v_intrablock_positions[None, :, None]
        else:
            kw = k.new_zeros(b, hkv, 0, self.compress_block_size, d)
            vw = v.new_zeros(b, hkv, 0, self.compress_block_size, d)
        ck, cv = self.k_compress(kw), self.v_compress(vw)

        if return_cache:
            overlap = self.compress_block_size - st
            run_k, run_v = k, v
            if overlap > 0:
                run_k, run_v = F.pad(run_k, (0, 0, overlap, 0)), F.pad(run_v, (0, 0, overlap, 0))
            cache_compressed = ((ck, cv), (run_k[..., ncb * st:, :], run_v[..., ncb * st:, :]))

        # branch 1: compressed attention, with the per-block importance as a by-product
        num_mem = self.num_mem_compress_kv
        mem_k, mem_v = self.compress_mem_kv[0].expand(b, -1, -1, -1), self.compress_mem_kv[1].expand(b, -1, -1, -1)
        ck_full, cv_full = torch.cat((mem_k, ck), dim=-2), torch.cat((mem_v, cv), dim=-2)
        sel_heads = hkv if self.query_heads_share_selected_kv else h
        num_selected = min(self.num_selected_blocks, ncb, ncb // (sel // st))
        # the kernel also averages the logits per selection block where it can, unless their gradient is wanted
        pool = sel // st if self.causal and not self.use_diff_topk and sel % st == 0 else 0
        o_cmp, importance = ops.compressed_attend(q, ck_full, cv_full, num_mem, st, self.causal, sel_heads=sel_heads,
                                                  want_importance=True, impl=impl, pool=pool) if num_selected > 0 else \
            (ops.compressed_attend(q, ck_full, cv_full, num_mem, st, self.causal, want_importance=False, impl=impl), None)

        qr, kr = self.rotary_emb.rotate_queries_with_cached_keys(q, k)
        if return_cache:
            cache_kv = (kr, v)

        # branch 2: block selection, then attention over the selected blocks
        idx = vals = fmask = None
        if num_selected > 0:
            vals, idx = ops.select_blocks(importance if self.use_diff_topk else importance.detach(), sel, st,
                                          num_selected, dtype=q.dtype)
            fmask = vals > 1e-10
            if forced_selection is not None:
                idx, fmask = forced_selection
            # differentiable top-k (NSA:715): the slots are scaled by 1 in the forward, the gradient of that scale
            # reaches the selected probabilities and through them the compressed logits
            slot_scale = vals + (1. - vals).detach() if self.use_diff_topk else None
            o_sel = ops.native_sparse_attend(qr, kr, v, sel, idx, fmask, sel_scale=slot_scale,
                                             include_block_causal=self.causal, impl=impl)
        else:
            o_sel = ops.block_diagonal_attend(qr, kr, v, sel, self.causal, impl=impl)

        # branch 3: sliding window; then the learned gates mix the three and merge heads
        o_swa = ops.sliding_window_attend(qr, kr, v, self.sliding_window_size, self.causal, impl=impl)
        gates = self.to_strategy_combine(x).view(b, n, h, 3).transpose(1, 2)
        merged = ops.gated_combine(o_cmp, o_sel, o_swa, gates)
        out = self.combine_heads(merged)

        if return_intermediates:
            return out, dict(q=q, k=k, v=v, ck=ck, cv=cv, qr=qr, kr=kr, importance=importance, vals=vals, idx=idx,
                             fmask=fmask, o_cmp=o_cmp, o_sel=o_sel, o_swa=o_swa, gates=gates, merged=merged)
        if not return_cache:
            return out
        return out, (cache_kv, cache_compressed)
