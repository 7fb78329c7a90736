"""The merges of the tensor-core family at slot counts around their rounds (six rows forward, nine backward), around the 32
slots of a word and above, with slots that a query does not have, against the oracle; bf16 at the operators' tolerance."""
import pytest
import torch

import recipe
from oracle import nsa_oracle as O
from util import assert_close_bf16

import native_sparse_attention_pytorch_b200 as nsa

pytestmark = pytest.mark.gpu


# slots = selected blocks and the own block
@pytest.mark.parametrize('d', [64, 128])
@pytest.mark.parametrize('nsel', [1, 5, 6, 8, 9, 11, 17, 18, 31, 32, 34])
def test_slot_counts(nsel, d):
    b, hq, hkv, n = 1, 4, 2, 260
    q = recipe.randn((b, hq, n, d), 1).bfloat16()
    k, v = (recipe.randn((b, hkv, n, d), s).bfloat16() for s in (2, 3))
    up = recipe.randn(q.shape, 4).bfloat16()
    idx = recipe.randint(0, 5, (b, hkv, n, nsel), 5)
    mask = (recipe.randint(0, 3, idx.shape, 6) > 0) & (idx < (torch.arange(n) // 64)[None, None, :, None])
    ref_in = [t.float().requires_grad_() for t in (q, k, v)]
    ref = O.selected_attend(*ref_in, 64, idx, mask, True)
    want = torch.autograd.grad(ref, ref_in, up.float())
    ins = [t.cuda().requires_grad_() for t in (q, k, v)]
    out = nsa.native_sparse_attend(*ins, 64, idx.cuda(), mask.cuda(), include_block_causal=True, impl='sm100')
    assert_close_bf16(out, ref, 'out')
    for g, w, name in zip(torch.autograd.grad(out, ins, up.cuda()), want, ('dq', 'dk', 'dv')):
        # a key collects from every later query and head: the tolerance grows with the sums, half a percent of the largest
        assert_close_bf16(g, w, name, rel_to_max=0.0 if name == 'dq' else 5e-3)
